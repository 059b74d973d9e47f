"""CPU tests of the launch shapes of the sweeps by blocks (csrc/sweep_shapes.h)."""
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
