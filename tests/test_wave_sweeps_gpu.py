"""The sweep of large left-to-right automata (sweep_wave_b200.inc) at the edges of its range: a piece and several more or
less by a state, edges past a thread's four, edges that lead as far as a piece can see, one further and back (other
sweeps then), blocks of fewer than four frames, sequences as short as their automata allow (whole tiles of pieces are
left out), several time chunks.  Against the double-precision oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_cluster_sweeps_gpu import check

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def batch(S, reach, deg, T, F, back=False):
    """Four sequences of S states and fewer; enough edges that the plan takes its general path."""
    rng = np.random.default_rng(S + 17 * deg + T)
    edges, weights, ends, off = [], [], [], 0
    for b, n in enumerate([S, max(2, S - 1), S // 2 + 1, S]):
        fr, to, into = [], [], np.zeros(n, int)
        for s in range(n):
            for h in dict.fromkeys([0, 1, reach] + [int(x) for x in rng.integers(1, reach + 1, deg - 3)]):
                if s + h < n and (into[s + h] < deg or h < 2):
                    fr.append(s)
                    to.append(s + h)
                    into[s + h] += 1
        if back:
            fr.append(n - 1)
            to.append(n - 2)
        edges.append(np.stack([np.array(fr) + off, np.array(to) + off, rng.integers(0, F, len(fr)), np.full(len(fr), b)]))
        weights.append(rng.uniform(0.0, 3.0, len(fr)))
        ends.append((off, off + n - 1))
        off += n
    am = rng.normal(4.0, 3.0, (T, 4, F)).astype(np.float32)
    lens = np.array([T, max(1, T - 3), max(1, T - 6), -(-S // reach) + 1], np.int32).clip(max=T)
    return (am, np.ascontiguousarray(np.concatenate(edges, 1), np.int32), np.concatenate(weights).astype(np.float32),
            np.ascontiguousarray(np.array(ends, np.int32).T), lens, off)


@pytest.mark.parametrize("S,reach,deg,T,F,back", [(1024, 8, 4, 170, 300, False), (1025, 8, 4, 171, 300, False),
                                                  (1537, 32, 4, 100, 2000, False), (1100, 32, 16, 66, 700, False),
                                                  (1100, 33, 5, 70, 700, False), (1100, 8, 5, 140, 700, True),
                                                  (3900, 8, 6, 520, 4800, False), (2500, 9, 17, 300, 90, False)])
def test_sizes(cuda, S, reach, deg, T, F, back):
    from i6_native_ops_b200.fbw import core

    check(core, cuda, *batch(S, reach, deg, T, F, back))


def test_infinite_scores(cuda):
    from i6_native_ops_b200.fbw import core

    am, e, w, se, lens, n = batch(1300, 16, 5, 120, 400)
    am[20, 0, 3:90] = np.inf
    am[40, 1, :] = np.inf  # no path
    am[33, 2, 9] = 1.0e30
    w[5::50] = np.inf
    check(core, cuda, am, e, w, se, lens, n)


CHILD = r"""
import torch
from test_cluster_sweeps_gpu import check
from test_wave_sweeps_gpu import batch
from i6_native_ops_b200.fbw import core
check(core, torch.device("cuda:0"), *batch(1100, 8, 5, 230, 700))
print("done")
"""


@pytest.mark.parametrize("chunks", [2, 3])
def test_time_chunks(cuda, chunks):
    env = dict(os.environ, FBW_B200_NUM_CHUNKS=str(chunks), FBW_B200_NUM_GROUPS="1",
               PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
