"""Launch shapes around the shared memory that a kernel may use without asking (48 KB less its static shared
memory): the largest automaton of a call grows state by state, so that the dynamic shared memory of the cluster
sweep passes every size around that limit, in a process in which no larger call has raised it before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import numpy as np, torch
import oracle
from test_automaton_sizes_gpu import batch, on_device
from i6_native_ops_b200.fbw import core
dev = torch.device("cuda:0")
for S in range(1140, 1330):
    e, w, se, lens, n, rng = batch(S, 3, 60, 100)
    am = rng.normal(4.0, 3.0, (60, 4, 100)).astype(np.float32)
    want = oracle.fbw_oracle(am, e, w, se, lens, n, "f64")[1]
    d = on_device(dev, am, e, w, se, lens)
    sums = core.fbw(*d, n, core.DebugOptions())[1].cpu().numpy()
    # a sum of at most 60 frames: as in test_automaton_sizes_gpu
    assert np.abs(sums - want).max() <= 4 * np.abs(want).max() * 2.0 ** -23 + 1e-6, S
print("done")
"""


def test_sizes_around_the_default_limit(cuda):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
