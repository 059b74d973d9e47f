"""The forms of the cluster sweep that depend on what fits into shared memory and on how many SMs are idle: few
score rows in flight, four or no recorded frames, edges read from global memory; clusters of two beside clusters
of four; and automata that go through clusters over several time chunks.  Against the double-precision oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import oracle
from test_automaton_sizes_gpu import automaton, batch, on_device

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def check(core, dev, am, e, w, se, lens, n):
    want, want_sums = oracle.fbw_oracle(am, e, w, se, lens, n, "f64")
    d = on_device(dev, am, e, w, se, lens)
    out, sums = core.fbw(*d, n, core.DebugOptions())
    out, sums = out.cpu().numpy().astype(np.float64), sums.cpu().numpy().astype(np.float64)
    assert np.array_equal(np.isinf(out), np.isinf(want))
    assert np.array_equal(sums == 0, want_sums == 0)
    # as in test_automaton_sizes_gpu: an edge score is a sum of four values of magnitude M
    M = max(1.0, np.abs(want_sums).max())
    assert np.abs(sums - want_sums).max() <= 4 * M * 2.0 ** -23 + 1e-6
    assert np.abs(np.exp(-out) - np.exp(-want)).max() <= 8 * M * 2.0 ** -23 + 2e-6


# states, edges a state, frames, classes; in shared memory then (score rows, recorded frames, edges):
@pytest.mark.parametrize("S,deg,T,F", [(1100, 9, 30, 9000),     # 4 rows, 8 frames, edges
                                       (1100, 24, 33, 8000),    # 2, 8, edges
                                       (1100, 24, 33, 17000),   # 2, 4, edges
                                       (1100, 24, 33, 18500),   # 2, none, edges
                                       (1100, 24, 33, 20000),   # 2, 8, no edges
                                       (3000, 9, 100, 20000),   # 2, 4, edges, clusters of eight
                                       (3000, 9, 100, 59000)])  # 2, none, no edges
def test_what_fits(cuda, S, deg, T, F):
    from i6_native_ops_b200.fbw import core

    e, w, se, lens, n, rng = batch(S, deg, T, F)
    check(core, cuda, rng.normal(4.0, 3.0, (T, 4, F)).astype(np.float32), e, w, se, lens, n)


def test_few_idle_sms(cuda):
    """72 sequences of 1100 to 1700 states: eight groups, clusters of four, then of two, then one CTA each."""
    from i6_native_ops_b200.fbw import core

    B, T, F = 72, 50, 200
    rng = np.random.default_rng(5)
    parts, ends, off = [], [], 0
    for b, n in enumerate(rng.integers(1100, 1700, B)):
        fr, to, em, w = automaton(rng, int(n), 3, T, F, False)
        parts.append((np.stack([fr + off, to + off, em, np.full(len(fr), b)]), w))
        ends.append((off, off + n - 1))
        off += int(n)
    e = np.ascontiguousarray(np.concatenate([p[0] for p in parts], 1), np.int32)
    am = rng.normal(4.0, 3.0, (T, B, F)).astype(np.float32)
    check(core, cuda, am, e, np.concatenate([p[1] for p in parts]), np.ascontiguousarray(np.array(ends, np.int32).T),
          rng.integers(T - 8, T + 1, B).astype(np.int32), off)


CHILD = r"""
import numpy as np, torch
from test_automaton_sizes_gpu import batch
from test_cluster_sweeps_gpu import check
from i6_native_ops_b200.fbw import core
for S, deg, T, F in [(1100, 4, 230, 700), (2300, 5, 257, 900), (1100, 24, 200, 8000), (300, 3, 201, 90)]:
    e, w, se, lens, n, rng = batch(S, deg, T, F)
    pick = e[3] < 3  # three sequences: one launch for the batch, cut in time
    check(core, torch.device("cuda:0"), rng.normal(4.0, 3.0, (T, 3, F)).astype(np.float32),
          np.ascontiguousarray(e[:, pick]), w[pick], np.ascontiguousarray(se[:, :3]), lens[:3], n)
print("done")
"""


@pytest.mark.parametrize("chunks", [2, 3])
def test_time_chunks(cuda, chunks):
    env = dict(os.environ, FBW_B200_NUM_CHUNKS=str(chunks), FBW_B200_NUM_GROUPS="1",
               PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
