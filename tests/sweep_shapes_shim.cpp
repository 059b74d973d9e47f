// Host build of the launch shapes of csrc/sweep_shapes.h for sweep_shapes.py.
#include "sweep_shapes.h"

static fbw_b200_summary summary(int64_t degree, int64_t notes) {
    fbw_b200_summary s;
    memset(&s, 0, sizeof(s));
    s.max_degree  = degree;
    s.reserved[0] = notes;
    return s;
}

// found, registers for edges, split, computing threads, all threads, ring (bytes from the start of shared memory), row
// length of the ring, shared memory
extern "C" void block_form(int64_t degree, int64_t notes, int64_t ms, int64_t md, int64_t* out) {
    const BlockShape c = block_shape(summary(degree, notes), ms, md);
    const int64_t v[8] = {c.found, c.kreg, c.split, c.d.compute, c.nt, (int64_t)block_smem(c.d).ring, c.d.dpmax, (int64_t)c.smem};
    memcpy(out, v, sizeof(v));
}

// found, pieces of the largest sequence, pieces a CTA can hold, CTAs a cluster, split, blocks of score rows kept, shared
// memory
extern "C" void wave_form(int64_t degree, int64_t notes, int64_t ms, int64_t me, int64_t md, int cs, int64_t* out) {
    const WaveShape c = wave_shape(summary(degree, notes), ms, me, md, cs);
    const int64_t v[7] = {c.found, c.pieces, c.d.pieces, c.d.cs, c.d.split, c.d.ring, (int64_t)c.smem};
    memcpy(out, v, sizeof(v));
}
// CTAs per cluster and whether that is faster than k_sweep_cluster, in a batch of so many sequences and so many frames
extern "C" int wave_fits(int64_t degree, int64_t notes, int64_t ms, int64_t me, int64_t md, int64_t sequences, int items,
                         int spare, int sms) {
    fbw_b200_summary s = summary(degree, notes);
    s.B = sequences;
    return wave_clusters(s, ms, me, md, items, spare, sms);
}
extern "C" int wave_is_faster(int64_t degree, int64_t notes, int64_t ms, int64_t me, int64_t md, int64_t sequences,
                              int64_t length, int cs, int sms) {
    fbw_b200_summary s = summary(degree, notes);
    s.B       = sequences;
    s.max_len = length;
    return wave_pays(s, ms, me, wave_shape(s, ms, me, md, cs), sms);
}
