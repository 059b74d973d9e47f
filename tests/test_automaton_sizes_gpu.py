"""The op and the alignment on automata at the edges of their kernels' ranges: one state, a warp more or less,
the most states of the sweep with one state per thread, of one CTA and of a cluster, of state vectors in
shared memory; states with more edges than registers hold; sequences of one frame and of other than whole
groups of eight frames; one class for all edges (the class sum is then shared by all warps); weights and
scores that are infinite or far outside the usual range.  Against the double-precision and the exact oracle."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

# states, largest number of edges a state gets, frames, classes
CASES = [(1, 2, 1, 1), (2, 2, 9, 1), (7, 3, 8, 2), (31, 2, 33, 5), (33, 3, 40, 7), (64, 7, 31, 2), (300, 4, 65, 1),
         (736, 3, 70, 40), (736, 7, 33, 3000), (737, 3, 41, 900), (992, 5, 40, 3), (1025, 6, 48, 700), (2049, 9, 50, 3000), (4100, 5, 24, 60),
         (8192, 2, 17, 9), (8193, 3, 16, 11)]


def automaton(rng, S, deg, T, F, far_weights):
    """Every state has a loop and edges forward; jumps are long enough for the end to be reached in T frames."""
    jump = max(1, -(-2 * S // T))
    steps = {0, 1} | ({jump} if deg > 2 or jump > 1 else set())
    if jump > 64:
        steps |= {4, 16, 64, 256} - set(range(jump, 257))
    fr, to = [], []
    for s in range(S):
        hops = steps | {int(h) for h in rng.integers(1, jump + 1, max(0, deg - 3))}
        for h in sorted(hops):
            if s + h < S:
                fr.append(s)
                to.append(s + h)
    E = len(fr)
    w = rng.uniform(0.0, 3.0, E).astype(np.float32)
    if far_weights and E > 8:
        pick = rng.permutation(E)[:4]
        w[pick] = [np.inf, 1.0e3, 120.0, -95.0]
    return np.array(fr), np.array(to), rng.integers(0, F, E), w


def batch(S, deg, T, F, far=False):
    rng = np.random.default_rng(S * 7 + T)
    states = [S, max(1, S // 3), min(S, 5), 3]
    lens = np.array([T, max(1, T - 3), min(T, 6), 0], np.int32)
    edges, weights, start_end, off = [], [], [], 0
    for b, n in enumerate(states):
        fr, to, em, w = automaton(rng, n, deg, int(max(lens[b], 1)), F, far)
        edges.append(np.stack([fr + off, to + off, em, np.full(len(fr), b)]))
        weights.append(w)
        start_end.append((off, off + n - 1))
        off += n
    return (np.ascontiguousarray(np.concatenate(edges, 1), np.int32), np.concatenate(weights),
            np.ascontiguousarray(np.array(start_end, np.int32).T), lens, off, rng)


def on_device(dev, *arrays):
    return [torch.from_numpy(a).to(dev) for a in arrays]


@pytest.mark.parametrize("S,deg,T,F", CASES)
@pytest.mark.parametrize("far", [False, True])
def test_posteriors(cuda, S, deg, T, F, far):
    from i6_native_ops_b200.fbw import core

    e, w, se, lens, n, rng = batch(S, deg, T, F, far)
    am = (rng.normal(4.0, 3.0, (T, 4, F))).astype(np.float32)
    if far and F > 2:
        am[T // 2, 0, F // 2] = np.inf
        am[T // 3, 0, F // 3] = 1.0e30
        am[T // 4, 1, 0] = 2.0e4
    want, want_sums = oracle.fbw_oracle(am, e, w, se, lens, n, "f64")
    d = on_device(cuda, am, e, w, se, lens)
    out, sums = core.fbw(*d, n, core.DebugOptions())
    out, sums = out.cpu().numpy().astype(np.float64), sums.cpu().numpy().astype(np.float64)
    assert np.array_equal(np.isinf(out), np.isinf(want))
    assert np.array_equal(sums == 0, want_sums == 0)
    # an edge score is a sum of four values of magnitude M, each rounded to 2^-24 M
    M = max(1.0, np.abs(want_sums).max())
    assert np.abs(sums - want_sums).max() <= 4 * M * 2.0 ** -23 + 1e-6
    assert np.abs(np.exp(-out) - np.exp(-want)).max() <= 8 * M * 2.0 ** -23 + 2e-6


@pytest.mark.parametrize("S,deg,T,F", CASES)
def test_alignment(cuda, S, deg, T, F):
    from i6_native_ops_b200.fast_viterbi import core

    e, w, se, lens, n, rng = batch(S, deg, T, F)
    am = -np.round(np.abs(rng.normal(4.0, 3.0, (T, 4, F)))).astype(np.float32)  # coarse: many ties
    w = np.round(w).astype(np.float32)
    want, want_scores = oracle.viterbi_oracle(am, e, -w, se, lens, n)
    d = on_device(cuda, am, e, -w, se, lens)
    got, scores = core.fast_viterbi(*d, n)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(scores.cpu().numpy(), want_scores)
