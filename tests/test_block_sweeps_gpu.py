"""The sweep of the smallest automata (sweep_block_b200.inc) at the edges of its range: a warp and eight warps of
states and one more or less; edges that fill a state's registers, need several threads or are one too many; the most
classes and one more; edges that lead back, edges in any order; first and last blocks of fewer than eight frames; several
time chunks.  Against the double-precision oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_cluster_sweeps_gpu import check

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def automaton(rng, S, deg, F, back):
    """Loops, edges to the next state and to others up to 40 on; about `deg` edges a state, either way."""
    fr, to, into = [], [], np.zeros(S, int)
    for s in range(S):
        hops = [0, 1] + [int(h) for h in rng.integers(2, 41, max(0, deg - 2))]
        for h in dict.fromkeys(hops):
            if s + h < S and (into[s + h] < deg or h < 2):
                fr.append(s)
                to.append(s + h)
                into[s + h] += 1
        if back and s > 2 and s % 5 == 0:
            fr.append(s)
            to.append(int(rng.integers(0, s)))
    return np.array(fr), np.array(to), rng.integers(0, F, len(fr)), rng.uniform(0.0, 3.0, len(fr)).astype(np.float32)


def batch(S, deg, T, F, back=False, shuffle=False):
    rng = np.random.default_rng(S * 31 + deg * 7 + T)
    edges, weights, ends, off = [], [], [], 0
    lens = np.array([T, max(1, T - 5), min(T, 7), 0], np.int32)
    for b, n in enumerate([S, max(2, S // 2), min(S, 6), 3]):
        fr, to, em, w = automaton(rng, n, deg, F, back)
        e = np.stack([fr + off, to + off, em, np.full(len(fr), b)])
        if shuffle:  # the order of a sequence's edges is the order of the sums, nothing else
            pick = rng.permutation(len(fr))
            e, w = e[:, pick], w[pick]
        edges.append(e)
        weights.append(w)
        ends.append((off, off + n - 1))
        off += n
    am = rng.normal(4.0, 3.0, (T, 4, F)).astype(np.float32)
    return (am, np.ascontiguousarray(np.concatenate(edges, 1), np.int32), np.concatenate(weights).astype(np.float32),
            np.ascontiguousarray(np.array(ends, np.int32).T), lens, off)


@pytest.mark.parametrize("S,deg,T,F", [(2, 2, 1, 3), (32, 2, 40, 9), (33, 3, 41, 9), (64, 4, 16, 5), (65, 2, 8, 2), (100, 3, 9, 90),
                                       (255, 3, 150, 40), (256, 3, 151, 40), (257, 3, 152, 40), (255, 2, 260, 257),
                                       (200, 5, 47, 300), (60, 16, 30, 640), (60, 17, 30, 640), (128, 9, 31, 641)])
def test_sizes(cuda, S, deg, T, F):
    from i6_native_ops_b200.fbw import core

    check(core, cuda, *batch(S, deg, T, F))


@pytest.mark.parametrize("back,shuffle", [(True, False), (True, True)])
@pytest.mark.parametrize("deg", [2, 3, 6])
def test_order_of_the_edges(cuda, deg, back, shuffle):
    from i6_native_ops_b200.fbw import core

    check(core, cuda, *batch(120, deg, 90, 50, back, shuffle))


def test_infinite_scores_and_weights(cuda):
    from i6_native_ops_b200.fbw import core

    am, e, w, se, lens, n = batch(150, 5, 70, 30)
    am[20, 0, 3:7] = np.inf
    am[40, 1, :] = np.inf  # no path
    am[33, 0, 9] = 1.0e30
    w[5::50] = np.inf
    check(core, cuda, am, e, w, se, lens, n)


CHILD = r"""
import torch
from test_cluster_sweeps_gpu import check
from test_block_sweeps_gpu import batch
from i6_native_ops_b200.fbw import core
for S, deg, T, F in [(100, 5, 230, 30), (256, 3, 257, 40), (40, 12, 201, 90)]:
    check(core, torch.device("cuda:0"), *batch(S, deg, T, F))
print("done")
"""


@pytest.mark.parametrize("chunks", [2, 3])
def test_time_chunks(cuda, chunks):
    env = dict(os.environ, FBW_B200_NUM_CHUNKS=str(chunks), FBW_B200_NUM_GROUPS="1",
               PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]


CHILD_NO_EDGES = r"""
import numpy as np, torch
import oracle
from test_automaton_sizes_gpu import on_device
from test_cluster_sweeps_gpu import check
from test_block_sweeps_gpu import batch
from i6_native_ops_b200.fbw import core
dev = torch.device("cuda:0")
for deg in (2, 3, 6):
    am, e, w, se, lens, n = batch(60, deg, 45, 2000)
    keep = e[3] < 3  # the last sequence: a start, an end, no edge
    e, w = np.ascontiguousarray(e[:, keep]), w[keep]
    lens[3] = 40
    check(core, dev, am, e, w, se, lens, n)
    want, want_sums = oracle.fbw_oracle(am, e, w, se, lens, n, "f64")
    lp = np.ascontiguousarray(-am.transpose(1, 0, 2))
    grad, sums = core.fbw_fused(*on_device(dev, lp, e, w, se, lens), n)
    assert np.array_equal(sums.cpu().numpy() == 0, want_sums == 0)
    M = max(1.0, np.abs(want_sums).max())
    assert np.abs(grad.cpu().numpy().astype(np.float64) + np.exp(-want).transpose(1, 0, 2)).max() <= 8 * M * 2.0 ** -23 + 2e-6
print("done")
"""


@pytest.mark.parametrize("output", ["expand", "patch"])
def test_a_launch_without_edges(cuda, output):
    """Groups of one sequence each, of which the cheapest has no edge; with the background beside the sweeps and without."""
    env = dict(os.environ, FBW_B200_NUM_GROUPS="4", FBW_B200_OUTPUT=output,
               PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHILD_NO_EDGES], env=env, capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
