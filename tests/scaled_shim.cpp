// Host build of the scaled numbers of csrc/scaled.h for test_scaled_numbers.py.
#include "scaled.h"

extern "C" void to_scaled_n(const float* s, int n, float* x, float* c) {
    for (int i = 0; i < n; i++) {
        const float2 v = to_scaled(s[i]);
        x[i] = v.x;
        c[i] = v.y;
    }
}

// negative log of the product of n numbers exp(-s), brought into range after every factor
extern "C" float product(const float* s, int n) {
    float2 v = make_float2(0.f, 0.f);
    for (int i = 0; i < n; i++) {
        const float2 q = to_scaled(s[i]);
        v = normalised(mul_scaled(v.x, q.x), v.y + q.y);
    }
    return from_scaled(v);
}

// negative log of the sum of n numbers exp(-s), one after another
extern "C" float sum(const float* s, int n) {
    float x = 0.f, c = FBW_INF;
    for (int i = 0; i < n; i++) {
        const float2 q = to_scaled(s[i]);
        add_scaled(x, c, q.x, q.y);
    }
    return from_scaled(normalised(x, c));
}
