"""CPU tests of the launch shapes of the sweeps by blocks and by pieces (csrc/sweep_shapes.h)."""
import os
import subprocess
import sys

import pytest

from sweep_shapes import block_form


@pytest.mark.parametrize("degree", [1, 3, 9])
@pytest.mark.parametrize("states", [1, 2, 40])
@pytest.mark.parametrize("slots", [0, 1, 2, 3, 4, 640])
def test_score_rows_are_there(degree, states, slots):
    """Every step reads a class of one of 16 rows: class 0 where a state has no edge, also when no sequence of the launch
    has any (the cheapest group of a batch)."""
    f = block_form(degree, 100, states, slots)
    assert f["found"] and f["dpmax"] >= max(1, slots)
    assert f["ring"] % 16 == 0 and f["smem"] - f["ring"] >= 16 * 8 * f["dpmax"] >= 16 * 8


CHILD = """
from sweep_shapes import wave_cluster, wave_form
for args in [(4, 8, 4000, 4000, 16000, 5000), (4, 8, 1025, 1025, 4100, 700), (6, 8, 2000, 1400, 7000, 9000), (3, 8, 7000, 7000, 20000, 9000)]:
    fits = wave_form(*args, cs=FORCED)["found"]
    assert wave_cluster(*args, items=16, spare=200) == (FORCED if fits else 0, 200), args
    print(fits, end=" ")
"""


@pytest.mark.parametrize("forced", [1, 2, 4, 8])
def test_the_switch_fixes_the_clusters_of_waves(forced):
    """FBW_B200_CLUSTER holds for every sweep; one that does not fit so many CTAs goes another way."""
    env = dict(os.environ, FBW_B200_CLUSTER=str(forced), PYTHONPATH=os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD.replace("FORCED", str(forced))], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "1" in r.stdout and ("0" in r.stdout) == (forced == 1)
