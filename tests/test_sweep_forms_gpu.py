"""The sweeps of the smallest and of large left-to-right automata (sweep_block_b200.inc, sweep_wave_b200.inc) in every form
and at their limits, on the batches of sweep_forms.py (which form each takes: test_sweep_forms.py); with infinities; over
several time chunks; the second one on one CTA and on clusters of more CTAs than there are pieces (FBW_B200_WAVE=1: also
where another sweep is faster).  Against the
double-precision oracle.  And all entry points give the same bits on batches that take these sweeps."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import sweep_forms as sf
from sweep_shapes import wave_fits, wave_is_faster
from test_automaton_sizes_gpu import on_device
from test_cluster_sweeps_gpu import check
from test_schedules_gpu import run, same
from test_zz_no_alloc import LIB, _noalloc

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("infinities", [False, True])
@pytest.mark.parametrize("name", list(sf.BLOCK))
def test_blocks(cuda, name, infinities):
    from i6_native_ops_b200.fbw import core

    check(core, cuda, *sf.block_case(name, infinities=infinities))


CHILD = r"""
import torch
import sweep_forms as sf
from test_cluster_sweeps_gpu import check
from i6_native_ops_b200.fbw import core
for name, infinities in [(n, i) for n in NAMES for i in (False, True)]:
    check(core, torch.device("cuda:0"), *(sf.block_case if name in sf.BLOCK else sf.wave_case)(name, infinities=infinities))
print("done")
"""


def child(names, **env):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]), **env)
    r = subprocess.run([sys.executable, "-c", CHILD.replace("NAMES", repr(names))], env=env, capture_output=True, text=True,
                       timeout=600, cwd=ROOT)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("clusters", ["", "1", "2", "8"])
def test_waves(cuda, clusters):
    # (the batch that does not fit goes in logarithms on one CTA, which is further off than this test allows)
    child([n for n in sf.WAVE if sf.WAVE[n][1][0] or clusters != "1"], FBW_B200_WAVE="1", FBW_B200_CLUSTER=clusters)


def test_without_waves(cuda):
    child(["a_state_more", "one_block_of_rows"], FBW_B200_WAVE="0")


@pytest.mark.parametrize("chunks", ["2", "3"])
def test_time_chunks(cuda, chunks):
    # (at least two tiles a chunk: the longer ones are cut)
    child(["two_whole_pieces", "a_state_more", "few_states_many_frames"] + [n for n in sf.BLOCK if sf.BLOCK[n][1][0]],
          FBW_B200_WAVE="1", FBW_B200_NUM_CHUNKS=chunks, FBW_B200_NUM_GROUPS="1")


def test_some_groups_in_waves(cuda):
    """Four groups of one sequence, the larger two in waves: the states that a launch leaves out are left out where the groups
    are launched by themselves and not where one launch serves the batch."""
    import i6_native_ops_b200.fbw as m

    am, e, w, se, lens, n = sf.batch([1500, 1400, 300, 40], (0, 1, 5, 8), 300, [230, 215, 190, 60], 300)
    d = sf.describe(e, n)
    for k in (1500, 1400):  # (and no group below 737 states)
        args = (d["degree"], d["reach"], d["fours"], k, 4 * k, 300)
        cs = wave_fits(*args, 4, items=2, spare=200)
        assert d["general"] and cs > 0 and wave_is_faster(*args, 4, 230, cs)
    check(m.core, cuda, am, e, w, se, lens, n)
    am, e, w, se, sl = on_device(cuda, am, e, w, se, lens)
    fsa = (n, e, w, se)
    out, sums = run(m.core, am, fsa, sl)
    plan = m.core.fbw_prepare(e, w, se, sl, am.shape[0], am.shape[2], n)
    (out1, sums1, _), _ = m.core.fbw_run_phases(plan, am)
    assert same(out1, out) and same(sums1, sums)
    lib = ctypes.CDLL(LIB)
    lib.fbw_b200_fbw_noalloc.restype = ctypes.c_int
    rc, out2, sums2, _ = _noalloc(lib, am, fsa, sl)
    torch.cuda.synchronize()
    assert rc == 0 and same(out2, out) and same(sums2, sums)
    am_h = torch.empty(am.shape, pin_memory=True).copy_(am)
    out_h, sums_h, _ = m.fbw_host_scores(am_h, fsa, sl)
    assert same(out_h, out) and same(sums_h, sums)


def test_short_ctc_sequences(cuda):
    """Up to 221 states, so all groups go by blocks of frames, with the background beside them where it is written so."""
    import i6_native_ops_b200.fbw as m
    from i6_native_ops_b200 import topology

    B, T, F, L = 16, 830, 10025, 110
    g = torch.Generator(device=cuda)
    g.manual_seed(2)
    lens = torch.linspace(20, L, B, device=cuda).to(torch.int32)
    labels = torch.randint(1, F, (B, L), dtype=torch.int32, device=cuda, generator=g)
    fsa = topology.ctc_topology(labels, lens)
    d = sf.describe(fsa[1].cpu().numpy(), int(fsa[0]))
    assert sf.block_form(d["degree"], d["threes"], d["states"], d["slots"])["found"] and not d["general"]
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
