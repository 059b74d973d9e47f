"""CPU tests of the launch shapes of the sweeps by blocks and by pieces (csrc/sweep_shapes.h)."""
import os
import subprocess
import sys

import pytest

from sweep_shapes import block_form, wave_fits, wave_is_faster


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
from sweep_shapes import wave_fits, wave_form
for args in [(4, 8, 4000, 4000, 16000, 5000), (4, 8, 1025, 1025, 4100, 700), (6, 8, 2000, 1400, 7000, 9000), (3, 8, 7000, 7000, 20000, 9000)]:
    fits = wave_form(*args, cs=FORCED)["found"]
    assert wave_fits(*args, 8, items=16, spare=200) == (FORCED if fits else 0), args
    print(fits, end=" ")
"""


@pytest.mark.parametrize("forced", [1, 2, 4, 8])
def test_the_switch_fixes_the_clusters_of_waves(forced):
    """FBW_B200_CLUSTER holds for every sweep; one that does not fit so many CTAs goes another way."""
    env = dict(os.environ, FBW_B200_CLUSTER=str(forced), PYTHONPATH=os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD.replace("FORCED", str(forced))], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "1" in r.stdout and ("0" in r.stdout) == (forced == 1)


# Measured, us a call with k_sweep_wave and with k_sweep_cluster (see wave_pays).  Edges a state: the most and the mean, how
# far they lead, threads a state; states, frames, sequences (in four groups).
SOME = (9, 3.5, 15, 1.18)
FAR = (4, 3.99, 32, 1.0)
FAR3 = (3, 2.99, 32, 1.0)
THREE = (3, 3.0, 2, 1.0)
FIVE = (5, 5.0, 7, 2.0)
SIX = (6, 5.99, 8, 2.0)
MEASURED = [
    (SOME, 1100, 440, 24, 753, 928), (SOME, 1900, 2280, 12, 3509, 4213), (SOME, 2500, 1000, 12, 1676, 2906),
    (SOME, 3600, 4320, 12, 9485, 13250), (FAR, 1100, 1320, 4, 1064, 1302), (FAR, 1100, 1320, 24, 2234, 1771),
    (FAR, 1400, 1680, 24, 2897, 2466), (FAR, 2500, 3000, 12, 4889, 5318), (FAR, 3600, 4320, 4, 3770, 4575),
    (FAR3, 1100, 1320, 24, 2066, 1671), (FAR3, 1900, 2280, 8, 1971, 2342), (FAR3, 2500, 3000, 12, 4532, 5169),
    (THREE, 1100, 550, 24, 856, 1227), (THREE, 1400, 700, 24, 1072, 1509), (THREE, 2500, 1250, 12, 1841, 2632),
    (FIVE, 1100, 1320, 8, 1020, 1823), (FIVE, 1100, 1320, 24, 3574, 2157), (FIVE, 1400, 560, 24, 1625, 1102),
    (FIVE, 1400, 1680, 8, 1281, 2588), (FIVE, 2500, 3000, 4, 4093, 3301), (FIVE, 3600, 4320, 12, 11693, 10477),
    (SIX, 1100, 550, 24, 2278, 1457), (SIX, 1100, 1320, 8, 1527, 2502), (SIX, 2500, 1250, 12, 5073, 3587),
]


@pytest.mark.parametrize("edges,states,frames,sequences,with_it,without", MEASURED)
def test_waves_where_they_are_faster(edges, states, frames, sequences, with_it, without):
    degree, mean, reach, threads = edges
    args = (degree, reach, int(threads * states), states, int(mean * states), 1000)
    cs = wave_fits(*args, sequences, items=2 * sequences // 4, spare=int(148 * 1.65) - 2 * sequences)
    assert cs > 0 and wave_is_faster(*args, sequences, frames, cs) == (with_it < without)
