"""Scores of a model that is sure of its labels: along one path nearly all of the probability, everything else
far away.  Per-frame sums are then small numbers whose last places count, and a frame's classes lie thousands
apart.  Automata of at most 128 edges, with a thread per state, with several states per thread and on clusters
of CTAs, against the double-precision oracle."""
import numpy as np
import pytest
import torch

import oracle
from test_automaton_sizes_gpu import batch, on_device

pytestmark = pytest.mark.gpu

CASES = [(12, 3, 40, 30), (60, 3, 64, 40), (300, 4, 90, 200), (700, 3, 96, 400), (1100, 4, 160, 900), (2300, 6, 129, 900)]


@pytest.mark.parametrize("S,deg,T,F", CASES)
@pytest.mark.parametrize("sure", [9.0, 12.0, 18.0, 40.0])
def test_sums_and_posteriors(cuda, S, deg, T, F, sure):
    from i6_native_ops_b200.fbw import core

    e, w, se, lens, n, rng = batch(S, deg, T, F)
    w = np.zeros_like(w)
    logits = rng.normal(0.0, 1.0, (T, 4, F))
    best, _ = oracle.viterbi_oracle(logits.astype(np.float32), e, w, se, lens, n)
    np.put_along_axis(logits, best[..., None], sure, 2)
    logits[:, :, 0] -= 400.0 * (best != 0)  # the first class, thousands away over the whole sequence
    am = (np.log(np.exp(logits).sum(-1, keepdims=True)) - logits).astype(np.float32)
    want, want_sums = oracle.fbw_oracle(am, e, w, se, lens, n, "f64")
    d = on_device(cuda, am, e, w, se, lens)
    out, sums = core.fbw(*d, n, core.DebugOptions())
    out, sums = out.cpu().numpy().astype(np.float64), sums.cpu().numpy().astype(np.float64)
    assert np.array_equal(sums == 0, want_sums == 0)
    live = want_sums != 0
    # T steps, each rounded to 2^-24 of the sum so far, in both directions, and the sum of the edge scores
    steps = 2 * T + 8
    assert (np.abs(sums - want_sums)[live] / np.abs(want_sums[live])).max() <= steps * 2.0 ** -24
    # a posterior p of a class at -log p = x is off by p times the rounding of its score: x and the sum once
    # more, p * x <= 1/e; on average half the largest rounding of a step
    bound = 0.5 * steps * 2.0 ** -24 * (1.0 + np.abs(want_sums).max(0, keepdims=True)[..., None])
    assert (np.abs(np.exp(-out) - np.exp(-want)) <= bound).all()
