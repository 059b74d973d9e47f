// sweep_shapes.h -- launch shapes of k_sweep_block (sweep_block_b200.inc) and k_sweep_wave (sweep_wave_b200.inc): for
// which automata they are chosen, threads of each kind, shared memory.  Plain arithmetic on the plan's summary, compiled
// into the library and, for the tests, by the host compiler alone.
#pragma once
#include "fbw_b200.h"
#include "scaled.h"

#include <stddef.h>
#include <stdlib.h>
#include <string.h>

// CTAs per cluster that FBW_B200_CLUSTER asks for (1, 2, 4 or 8); 0: none
static inline int forced_cluster_size() {
    static const int forced = [] {
        const char* e = getenv("FBW_B200_CLUSTER");
        const int   n = e ? atoi(e) : 0;
        return n == 1 || n == 2 || n == 4 || n == 8 ? n : 0;
    }();
    return forced;
}

// ---- k_sweep_block ----
constexpr int kBlockStates = 256;  // threads that compute
constexpr int kBlockFrames = 8;    // frames of a block
constexpr int kBlockDegree = 16;   // edges of a state
constexpr int kBlockRow    = 640;  // classes: the two blocks of score rows are then at most 82 KB

struct BlockDims {
    int dpmax;                  // row length of the score ring
    int compute, copy, record;  // threads of each kind (multiples of 32)
};
struct BlockSmem {
    size_t rows, lane, ring, total;
};
FBW_HD BlockSmem block_smem(const BlockDims& d) {
    BlockSmem m;
    size_t off = 0;
    m.rows  = off; off += (size_t)16 * kBlockFrames * kBlockStates;
    m.lane  = off; off += (size_t)4 * kBlockStates;
    m.ring  = off; off += (size_t)16 * kBlockFrames * d.dpmax;
    m.total = off;
    return m;
}

struct BlockShape {
    bool      found;
    int       kreg, nt;
    bool      split;
    size_t    smem;
    BlockDims d;
};
// the most groups of three that the edges of a sequence's states take, by target or by source state; 0: not known
static inline int64_t edge_groups(const fbw_b200_summary& s) { return s.reserved[0] & 0xffffffffll; }

// Launch shape for automata of at most ms states and md class slots
static inline BlockShape block_shape(const fbw_b200_summary& s, int64_t ms, int64_t md) {
    BlockShape c;
    memset(&c, 0, sizeof(c));
    const int64_t degree = s.max_degree;
    if (edge_groups(s) == 0 || degree > kBlockDegree || ms > kBlockStates || md > kBlockRow) return c;
    c.kreg  = degree <= 2 ? 2 : 3;
    c.split = degree > c.kreg;
    // a warp may leave as many threads unused as a state has parts less one
    const int64_t parts = (degree + c.kreg - 1) / c.kreg;
    const int64_t warps = c.split ? (edge_groups(s) + 32 - parts) / (33 - parts) : (ms + 31) / 32;
    if (32 * warps > kBlockStates) return c;
    BlockDims& d = c.d;
    d.compute = 32 * (int)warps;
    d.copy    = md > 256 ? 64 : 32;
    d.record  = d.compute <= 64 ? 32 : 64;
    // (a launch whose sequences have no edges has no score rows; the steps read a place of the ring all the same, which
    // has to be there)
    d.dpmax   = md > 0 ? (int)((md + 3) & ~(int64_t)3) : 4;
    c.nt    = d.compute + d.copy + d.record;
    c.smem  = block_smem(d).total;
    c.found = true;
    return c;
}

// ---- k_sweep_wave ----
constexpr int kWavePiece  = 512;   // threads that compute
constexpr int kWaveEdges  = 4;     // edges of a thread
constexpr int kWaveHalo   = 32;    // states before its first one that a piece reads
constexpr int kWaveBlock  = 4;     // frames of a block
constexpr int kWaveStates = 7168;  // states of a sequence (k_hops)
constexpr int kWaveDegree = 16;    // edges of a state (four parts)
constexpr int kWaveInbox  = 4;     // blocks kept for the next CTA
constexpr int kWaveRow    = kWavePiece + kWaveHalo;  // row length of a block's state vectors
constexpr int kWaveCopy   = 128;   // threads that copy score rows
constexpr int kWaveRecord = 64;    // threads that record

struct WaveDims {
    int dpmax;    // row length of the score ring
    int pieces;   // pieces a CTA can hold
    int cs;       // CTAs per cluster
    int split;    // some state has more than kWaveEdges edges
    int states;   // most states of a sequence
    int ring;     // blocks of score rows kept: 2, or 1 where two do not fit
};
struct WaveSmem {
    size_t rows, save, lane, inbox, ring, info, total;
};
FBW_HD WaveSmem wave_smem(const WaveDims& d) {
    WaveSmem m;
    size_t off = 0;
    m.rows  = off; off += (size_t)16 * kWaveBlock * kWaveRow;
    m.save  = off; off += (size_t)8 * d.pieces * kWavePiece;
    m.lane  = off; off += (size_t)4 * d.pieces * kWavePiece;
    m.inbox = off; off += d.cs > 1 ? (size_t)8 * kWaveInbox * kWaveBlock * kWaveHalo : 0;
    m.info  = off; off += ((size_t)4 * (4 * d.pieces + 8) + 15) & ~(size_t)15;
    m.ring  = off;  // (at set-up: row pointers and the first states of the warps)
    const size_t ring = (size_t)4 * d.ring * kWaveBlock * d.dpmax, setup = (size_t)4 * (d.states + 2) + (size_t)2 * (d.states + 2);
    off += ring > setup ? ring : setup;
    m.total = (off + 15) & ~(size_t)15;
    return m;
}

struct WaveShape {
    bool     found;
    int      pieces;  // of the largest sequence
    size_t   smem;
    WaveDims d;
};
// Launch shape for automata of at most ms states, me edges and md class slots on clusters of cs CTAs.  What the plan
// says of the edges: see note_edges.
static inline WaveShape wave_shape(const fbw_b200_summary& s, int64_t ms, int64_t me, int64_t md, int cs) {
    WaveShape c;
    memset(&c, 0, sizeof(c));
    const int64_t reach = (s.reserved[0] >> 32) & 0xffff, groups = (s.reserved[0] >> 48) & 0xffff;
    if (groups == 0 || md == 0 || reach > kWaveHalo || s.max_degree > kWaveDegree || ms > kWaveStates) return c;
    WaveDims& d = c.d;
    d.cs     = cs;
    d.split  = s.max_degree > kWaveEdges;
    d.states = (int)ms;
    d.dpmax  = (int)((md + 3) & ~(int64_t)3);
    // warps: a warp may leave as many threads unused as a state has parts less one
    const int64_t parts = (s.max_degree + kWaveEdges - 1) / kWaveEdges;
    const int64_t most  = ms + me / kWaveEdges;
    const int64_t lanes = d.split ? (groups < most ? groups : most) : ms;
    const int64_t warps = (lanes + 32 - parts) / (33 - parts);
    c.pieces  = (int)((warps + kWavePiece / 32 - 1) / (kWavePiece / 32));
    d.pieces  = (c.pieces + cs - 1) / cs;
    for (d.ring = 2; d.ring >= 1 && !c.found; d.ring--) {
        c.smem  = wave_smem(d).total;
        c.found = c.smem <= 227 * 1024 - 256;
        if (c.found) break;
    }
    return c;
}

// FBW_B200_WAVE=0|1: k_sweep_wave never, wherever it fits; -1: by wave_pays
static inline int forced_wave() {
    static const int forced = [] {
        const char* e = getenv("FBW_B200_WAVE");
        return e ? atoi(e) : -1;
    }();
    return forced;
}
// Whether automata that both fit are faster with k_sweep_wave, on clusters of c.d.cs CTAs, than with k_sweep_cluster, in a
// batch of s.B sequences.  (Where the other sweep would be the one in logarithms, k_sweep, this one is taken in any
// case: its sums are up to thirty times nearer to the true ones.)
// k_sweep_cluster meets once a frame, 0.9 to 1.3 us for up to a few hundred states a CTA; k_sweep_wave has a thread for
// every four edges of a state, 0.8 us a frame for 512 of them and two thirds of it for 512 more, and leaves out what lies
// on no path.  So it gains where a cluster holds all pieces side by side, where few states have many edges (a warp of the
// other takes as long as its state with most) and where few frames leave out much; it loses where a CTA holds two pieces
// of states that all have the same edges.  Measured, us a call with k_sweep_cluster / k_sweep_wave:
//   some states with far more edges (loops, successors, one or two more; 3.5 on average, the most 9): 24 sequences of 1100
//     states and 440 frames 928 / 753, 12 of 2500 and 1000: 2906 / 1676, 12 of 3600 and 4320: 13250 / 9485
//   edges from every state to those 0, 1, 8 and 32 on: 4 sequences of 1100 states and 1320 frames 1303 / 1064 (a piece a CTA),
//     24: 1771 / 2234, 24 of 1400 and 1680: 2466 / 2897; 12 of 2500 and 3000: 5318 / 4889
//   0, 1 and 2 on, 24 of 1400 and 700 (no more frames than the way takes): 1509 / 1072
//   0, 1, 2, 4 and 7 on (two threads a state): 8 of 1100 and 1320: 1823 / 1020 (a piece a CTA), 24: 2157 / 3574; 24 of 1400
//     and 560: 1103 / 1625; 4 of 2500 and 3000: 3301 / 4093
static inline bool wave_pays(const fbw_b200_summary& s, int64_t ms, int64_t me, const WaveShape& c, int sms) {
    const int64_t way = (s.reserved[0] >> 32) & 0xffff, groups = (s.reserved[0] >> 48) & 0xffff;
    if (4 * s.max_degree * ms >= 7 * me) return true;
    const bool    one_each = c.pieces <= c.d.cs;
    const int64_t most     = ms + me / kWaveEdges;
    if (c.d.split && 2 * (groups < most ? groups : most) > 3 * ms) {  // two threads and more for most states
        return one_each && 2 * s.B * c.d.cs <= sms;                   // (every CTA of the batch has an SM to itself)
    }
    // (the last: a state lies on a path in less than a quarter of the frames)
    return one_each || ms >= 2048 || 4 * ms >= 3 * way * s.max_len;
}

// CTAs per cluster for `items` (sequence, direction) pairs: as many as the pieces need to fit, and more, up to one a
// piece, while `spare` SMs would stay idle; or as many as FBW_B200_CLUSTER says.  0: they do not fit.
// Numbers of pieces between the powers of two get the next one where every CTA of the batch has an SM to itself, and the
// CTAs without a piece leave at once: a second piece costs its CTA two thirds of a frame more.
static inline int wave_clusters(const fbw_b200_summary& s, int64_t ms, int64_t me, int64_t md, int items, int spare, int sms) {
    const int forced = forced_cluster_size();
    if (forced > 0) return wave_shape(s, ms, me, md, forced).found ? forced : 0;
    int least = 1;
    while (least <= 8 && !wave_shape(s, ms, me, md, least).found) least *= 2;
    if (least > 8) return 0;
    const int pieces = wave_shape(s, ms, me, md, least).pieces;
    int cs = 8;
    auto more_than_needed = [&](int n) { return n > pieces && (n / 2 >= pieces || 2 * s.B * n > sms); };
    while (cs > least && (more_than_needed(cs) || (cs - 1) * items > spare)) cs >>= 1;
    return cs;
}
