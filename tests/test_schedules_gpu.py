"""All entry points give the same bits: groups of sequences, time chunks, one launch after another, the result
written by host threads, and the library's own scratch.  Batches whose sequences lie on both sides of the limits
between the kinds of sweeps, so that a choice made per launch would differ from schedule to schedule."""
import ctypes

import numpy as np
import pytest
import torch

from test_automaton_sizes_gpu import automaton, on_device
from test_zz_no_alloc import LIB, _noalloc

pytestmark = pytest.mark.gpu


def run(core, am, fsa, sl):
    out, sums = core.fbw(am, fsa[1], fsa[2], fsa[3], sl, int(fsa[0]), core.DebugOptions())
    return out, sums


def same(a, b):
    return torch.equal(a.cpu().view(torch.int32), b.cpu().view(torch.int32))


def test_long_ctc_sequences(cuda):
    """202 to 802 states: the shorter half of the batch has a thread per state, the longest sequences have not."""
    import i6_native_ops_b200.fbw as m
    from i6_native_ops_b200 import topology

    B, T, F, L = 16, 830, 10025, 400
    g = torch.Generator(device=cuda)
    g.manual_seed(1)
    lens = torch.linspace(100, L, B, device=cuda).to(torch.int32)
    labels = torch.randint(1, F, (B, L), dtype=torch.int32, device=cuda, generator=g)
    fsa = topology.ctc_topology(labels, lens)
    sl = torch.full((B,), T, dtype=torch.int32, device=cuda)
    am = torch.randn((T, B, F), device=cuda, generator=g).mul_(2.0).log_softmax(-1).neg_()
    out, sums = run(m.core, am, fsa, sl)
    plan = m.core.fbw_prepare(fsa[1], fsa[2], fsa[3], sl, T, F, int(fsa[0]))
    (out1, sums1, _), _ = m.core.fbw_run_phases(plan, am)
    assert same(out1, out) and same(sums1, sums)
    del out1
    am_h = torch.empty(am.shape, pin_memory=True).copy_(am)
    out_h, sums_h, _ = m.fbw_host_scores(am_h, fsa, sl)
    assert same(out_h, out) and same(sums_h, sums)
    del out_h
    out_p = torch.empty(am.shape, pin_memory=True)
    for staged in (True, False):
        out_p.fill_(float("nan"))
        _, sums_p, _ = m.fbw_host_scores(am_h, fsa, sl, out=out_p, staged=staged)
        torch.cuda.synchronize()
        assert same(sums_p, sums) and same(out_p, out)


@pytest.mark.parametrize("B", [3, 12, 30])
def test_mixed_automata(cuda, B):
    """40 to 2500 states: threads, several states per thread and clusters in one batch."""
    import i6_native_ops_b200.fbw as m

    rng = np.random.default_rng(B)
    T, F = 130, 300
    parts, off, ends = [], 0, []
    for b, n in enumerate(np.geomspace(40, 2500, B).astype(int)):
        fr, to, em, w = automaton(rng, n, 4, T, F, False)
        parts.append((np.stack([fr + off, to + off, em, np.full(len(fr), b)]), w))
        ends.append((off, off + n - 1))
        off += n
    am, e, w, se, sl = on_device(
        cuda, rng.normal(4.0, 3.0, (T, B, F)).astype(np.float32),
        np.ascontiguousarray(np.concatenate([p[0] for p in parts], 1), np.int32), np.concatenate([p[1] for p in parts]),
        np.ascontiguousarray(np.array(ends, np.int32).T), rng.integers(T - 40, T + 1, B).astype(np.int32))
    fsa = (off, e, w, se)
    out, sums = run(m.core, am, fsa, sl)
    plan = m.core.fbw_prepare(e, w, se, sl, T, F, off)
    (out1, sums1, _), _ = m.core.fbw_run_phases(plan, am)
    assert same(out1, out) and same(sums1, sums)
    lib = ctypes.CDLL(LIB)
    lib.fbw_b200_fbw_noalloc.restype = ctypes.c_int
    rc, out2, sums2, _ = _noalloc(lib, am, fsa, sl)
    torch.cuda.synchronize()
    assert rc == 0 and same(out2, out) and same(sums2, sums)
