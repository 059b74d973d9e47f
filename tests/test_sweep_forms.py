"""CPU test: the batches of sweep_forms.py have the numbers of edges, states and classes they are named for and take the
form of sweep they are meant for, at the limits of each and one past them."""
import pytest

import sweep_forms as sf


@pytest.mark.parametrize("name", list(sf.BLOCK))
def test_blocks(name):
    (sizes, deg, classes, _), want = sf.BLOCK[name]
    d, got = sf.block_taken(name)
    assert d["degree"] == deg and d["states"] == max(sizes) and d["slots"] == classes and not d["general"]
    assert got == want


@pytest.mark.parametrize("name", list(sf.WAVE))
def test_waves(name):
    (sizes, hops, classes, _, _), want = sf.WAVE[name]
    d, got = sf.wave_taken(name)
    assert d["degree"] == len(hops) and d["reach"] == max(hops) and d["states"] == max(sizes) and d["slots"] == classes
    assert d["general"]
    assert got == want


@pytest.mark.parametrize("name,pieces,ring", [("two_whole_pieces", 2, 2), ("a_state_more", 3, 2), ("one_block_of_rows", 6, 1)])
def test_waves_on_one_cta(name, pieces, ring):
    d, got = sf.wave_taken(name, 1)
    assert (got[0], got[2], got[3], got[4]) == (1, pieces, 1, ring)
