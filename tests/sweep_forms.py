"""Batches whose automata have exact numbers of edges a state and of classes, and the form of k_sweep_block
(sweep_block_b200.inc) or k_sweep_wave (sweep_wave_b200.inc) that each of them takes: the limits of both are counted in
states, in edges of the state that has most, in groups of edges, in classes and in how far an edge leads."""
import numpy as np

from sweep_shapes import block_form, wave_fits, wave_form


def automaton(rng, n, hops, ring, classes):
    """An edge from every state to the one `h` on, for each of `hops`; past the last state round to the first (`ring`: then
    every state has exactly as many edges in and out) or left out.  Exactly `classes` classes, if there are so many edges."""
    s, h = np.repeat(np.arange(n), len(hops)), np.tile(np.array(hops), n)
    to = (s + h) % n if ring else s + h
    fr, to = s[to < n], to[to < n]
    return fr, to, rng.permutation(np.arange(len(fr)) % classes), rng.uniform(0.0, 3.0, len(fr)).astype(np.float32)


def batch(sizes, hops, classes, lens, F, ring=False, inner=False, infinities=False):
    """scores, edges, weights, start and end states, lengths, number of states.  `inner`: sequences start a quarter into
    their states and end a quarter before the last."""
    rng = np.random.default_rng(sizes[0] * 31 + len(hops) * 7 + lens[0])
    edges, weights, ends, off = [], [], [], 0
    for b, n in enumerate(sizes):
        fr, to, em, w = automaton(rng, n, hops, ring, classes)
        edges.append(np.stack([fr + off, to + off, em, np.full(len(fr), b)]))
        weights.append(w)
        ends.append((off + (n // 4 if inner else 0), off + n - 1 - (n // 4 if inner else 0)))
        off += n
    T = max(lens)
    am = rng.normal(4.0, 3.0, (T, len(sizes), F)).astype(np.float32)
    w = np.concatenate(weights)
    if infinities:
        am[T // 4, 0, 3:7] = np.inf
        am[min(T // 3, lens[1] - 1), 1, :] = np.inf  # no path
        am[T // 2, 0, 9] = 1.0e30
        w[5::50] = np.inf
    return (am, np.ascontiguousarray(np.concatenate(edges, 1), np.int32), w, np.ascontiguousarray(np.array(ends, np.int32).T),
            np.array(lens, np.int32), off)


def describe(e, n):
    """what a plan knows of the edges: maxima over the sequences, over in and out edges"""
    into, out = np.bincount(e[1], minlength=n), np.bincount(e[0], minlength=n)
    owner = np.zeros(n, int)
    owner[e[0]] = owner[e[1]] = e[3]
    groups = lambda per: int(max(np.bincount(owner, np.maximum(1, -(-d // per))).max() for d in (into, out)))
    return dict(degree=int(max(into.max(), out.max())), threes=groups(3), fours=groups(4),
                reach=int((e[1] - e[0]).max()) if (e[1] >= e[0]).all() else 65535, states=int(np.bincount(owner).max()),
                edges=int(np.bincount(e[3]).max()), slots=max(len(np.unique(e[2][e[3] == b])) for b in np.unique(e[3])),
                general=e.shape[1] // (int(e[3].max()) + 1) > 2048)


# k_sweep_block: sizes, edges a state, classes, lengths, and what is expected: found, registers for edges, split, warps
BLOCK = {
    "two_edges_eight_warps": (([256, 100, 3], 2, 30, [140, 65, 5]), (1, 2, 0, 8)),
    "three_edges_eight_warps": (([256, 255, 1], 3, 200, [70, 9, 64]), (1, 3, 0, 8)),
    "three_edges_a_state_less": (([255, 31, 32], 3, 60, [71, 40, 33]), (1, 3, 0, 8)),
    "three_edges_a_state_more": (([257, 31, 32], 3, 60, [71, 40, 33]), (0, 0, 0, 0)),
    "four_edges_two_parts": (([124, 62, 7], 4, 80, [64, 58, 40]), (1, 3, 1, 8)),
    "four_edges_a_warp_more": (([125, 62, 7], 4, 80, [64, 58, 40]), (0, 3, 1, 0)),
    "sixteen_edges_six_parts": (([36, 20, 17], 16, 500, [50, 48, 16]), (1, 3, 1, 8)),
    "sixteen_edges_a_warp_more": (([37, 20, 17], 16, 500, [50, 48, 16]), (0, 3, 1, 0)),
    "seventeen_edges": (([20, 18, 17], 17, 300, [50, 48, 16]), (0, 0, 0, 0)),
    "the_most_classes": (([256, 250, 9], 3, 640, [73, 66, 33]), (1, 3, 0, 8)),
    "the_most_classes_two_parts": (([110, 108, 9], 6, 640, [41, 40, 33]), (1, 3, 1, 8)),
    "a_class_more": (([256, 250, 9], 3, 641, [73, 66, 33]), (0, 0, 0, 0)),
}
# k_sweep_wave: sizes, hops, classes, lengths, inner, and what is expected of the launch by default: found, split, pieces
# of the largest sequence, CTAs a cluster, blocks of score rows kept
WAVE = {
    "two_whole_pieces": (([1024, 1023, 512], (0, 1, 5, 8), 300, [170, 131, 66], False), (1, 0, 2, 2, 2)),
    "a_state_more": (([1025, 513, 1024], (0, 1, 5, 8), 300, [171, 70, 130], False), (1, 0, 3, 4, 2)),
    "a_quarter_off_either_end": (([1300, 1100, 900], (0, 1, 5, 8), 300, [120, 110, 60], True), (1, 0, 3, 4, 2)),
    "sixteen_edges_four_parts": (([1100, 900, 40], tuple(range(15)) + (32,), 700, [66, 61, 34], False), (1, 1, 10, 8, 2)),
    "seventeen_edges_and_large": (([1100, 900, 40], tuple(range(16)) + (32,), 700, [66, 61, 34], False), (0, 0, 0, 0, 0)),
    "one_block_of_rows": (([1500, 1400], (0, 1, 4, 20, 32), 6500, [90, 75], False), (1, 1, 6, 8, 1)),
    "hardly_any_frames": (([1100, 900, 800], (0, 1, 3, 32), 90, [41, 1, 0], False), (1, 0, 3, 4, 2)),
    "few_states_many_frames": (([1500, 2, 900], (0, 1, 3, 32), 90, [230, 200, 60], False), (1, 0, 3, 4, 2)),
}


def block_case(name, **kw):
    (sizes, deg, classes, lens), _ = BLOCK[name]
    return batch(sizes, tuple(range(deg)), classes, lens, max(classes, 10), ring=True, inner=True, **kw)


def block_taken(name):
    d = describe(block_case(name)[1], block_case(name)[5])
    f = block_form(d["degree"], d["threes"], d["states"], d["slots"])
    return d, (f["found"], f["kreg"], f["split"], f["compute"] // 32)


def wave_case(name, **kw):
    (sizes, hops, classes, lens, inner), _ = WAVE[name]
    return batch(sizes, hops, classes, lens, max(classes, 10), inner=inner, **kw)


def wave_taken(name, cs=None):
    """by default one launch for the batch (fewer than four sequences, few scores), as FBW_B200_WAVE=1 has it"""
    b = wave_case(name)
    d = describe(b[1], b[5])
    args = (d["degree"], d["reach"], d["fours"], d["states"], d["edges"], d["slots"])
    B = len(b[4])
    if cs is None:
        cs = wave_fits(*args, B, items=2 * B, spare=148 - 2 * B)
    f = wave_form(*args, cs=cs) if cs else wave_form(*args, cs=1)
    return d, (f["found"], f["split"], f["pieces"], f["cs"], f["ring"] if f["found"] else 0)
