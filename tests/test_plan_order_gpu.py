"""The plan's grouping by sequence (k_order): state ids of the sequences interleaved, some used by none, edges of the
sequences in any order.  Each sequence keeps the order of its own states and edges, so results are those of the batch
written down sequence after sequence, bit for bit."""
import numpy as np
import pytest
import torch

from test_block_sweeps_gpu import batch

pytestmark = pytest.mark.gpu


def interleaved(rng, ids, n):
    """a random order of n items in which items of the same id keep theirs"""
    order = rng.permutation(n)
    out = np.empty(n, int)
    for k in np.unique(ids):
        out[np.sort(order[ids[order] == k])] = np.nonzero(ids == k)[0]
    return out


@pytest.mark.parametrize("states,edges", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("S", [5, 90, 700])
def test_interleaved_sequences(cuda, S, states, edges):
    from i6_native_ops_b200.fbw import core

    am, e, w, se, lens, n = batch(S, 3, 40, 30)
    rng = np.random.default_rng(S)
    want = core.fbw(*[torch.from_numpy(x).to(cuda) for x in (am, e, w, se, lens)], n, core.DebugOptions())
    total = n
    if states:
        owner = np.zeros(n, int)
        owner[e[0]] = owner[e[1]] = e[3]
        owner[se[0]] = owner[se[1]] = np.arange(4)
        new = np.empty(n, int)
        new[interleaved(rng, owner, n)] = np.sort(rng.permutation(n + 7)[:n])  # seven ids are left unused
        total = n + 7
        e = np.stack([new[e[0]], new[e[1]], e[2], e[3]])
        se = new[se]
    if edges:
        order = interleaved(rng, e[3], e.shape[1])
        e, w = e[:, order], w[order]
    d = [torch.from_numpy(np.ascontiguousarray(x)).to(cuda) for x in (am, e.astype(np.int32), w, se.astype(np.int32), lens)]
    got = core.fbw(*d, total, core.DebugOptions())
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("total", [65536, 65537, 400001])
def test_many_state_ids(cuda, total, spread):
    """Up to 65536 ids k_order looks itself whether they are in order, beyond a launch before it does.  The ids in use
    come first (in order) or are spread over all (not in order)."""
    from i6_native_ops_b200.fbw import core

    am, e, w, se, lens, n = batch(90, 3, 40, 30)
    want = core.fbw(*[torch.from_numpy(x).to(cuda) for x in (am, e, w, se, lens)], n, core.DebugOptions())
    if spread:
        new = np.sort(np.random.default_rng(total).permutation(total)[:n])
        new[-1] = total - 1
        e = np.stack([new[e[0]], new[e[1]], e[2], e[3]])
        se = new[se]
    d = [torch.from_numpy(np.ascontiguousarray(x)).to(cuda) for x in (am, e.astype(np.int32), w, se.astype(np.int32), lens)]
    got = core.fbw(*d, total, core.DebugOptions())
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
