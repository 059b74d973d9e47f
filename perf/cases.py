"""The calls whose speed counts: what a training or alignment program asks of this package.

Inputs, automata included, are synthetic and drawn from a seed: scores are ``log_softmax`` of normal
logits, automata have the topologies of ``i6_native_ops_b200.workloads`` (CTC, left-to-right HMM, HMM
with skips, irregular lattice).  A case is a dict of

  entry   the public entry point: ``loss`` (``fbw_loss`` and its backward pass), ``fused``
          (``fbw_loss_fused`` and its backward pass), ``cached`` (``fbw_loss_cached`` on a plan cache
          that has seen the automata, and its backward pass), ``op`` (``core.fbw``, the operation
          itself on negative log scores in (T,B,F)), ``align`` (``align_viterbi``)
  topo    the topology, ``T B F`` frames, sequences and classes
  lo hi   range of the label count of a sequence (CTC: symbols, HMM: phones or allophones of three
          states each, lattice: states)
  tlo     shortest sequence length drawn

``listed`` gives the sizes this repository is used at, ``draw`` others from the same ranges.
"""
import math

import numpy as np
import torch

from i6_native_ops_b200 import topology
from i6_native_ops_b200.fast_viterbi import align_viterbi
from i6_native_ops_b200.fbw import PlanCache, core, fbw_loss, fbw_loss_cached, fbw_loss_fused

#: standard deviation of the logits and bias of the blank's logit
LOGITS = {"ctc": (1.0, 0.0), "bpe": (2.0, 3.0), "mono": (2.0, 0.0), "tri": (3.0, 0.0), "lattice": (2.0, 0.0)}
ZIPF = 1.1  # exponent of the unit frequencies of a large CTC vocabulary


def case(name, entry, topo, T, B, F, lo, hi, tlo):
    return {"name": name, "entry": entry, "topo": topo, "T": T, "B": B, "F": F, "lo": lo, "hi": hi, "tlo": tlo}


def listed():
    return [
        # a handful of short utterances with a character vocabulary: the smallest calls, where launches,
        # allocations and the host's own time are everything
        case("ctc_tiny_loss", "loss", "ctc", 50, 4, 41, 5, 12, 40),
        # forced alignment of the same: recipes align small shards with small models
        case("monophone_align", "align", "mono", 500, 32, 121, 20, 60, 350),
        # a monophone system's training step, the first stage of an HMM recipe
        case("monophone_loss", "loss", "mono", 500, 32, 121, 20, 60, 350),
        # the same automata epoch after epoch: their preparation comes from the plan cache
        case("monophone_cached", "cached", "mono", 500, 32, 121, 20, 60, 350),
        # a training step of a tied-state triphone system through the reference-compatible wrapper, at a
        # batch that leaves room for an encoder beside it; sizes that divide nothing
        case("triphone_loss", "loss", "tri", 1499, 17, 12001, 50, 150, 1200),
        # the operation itself at the full batch of that system: the repository's headline workload
        case("triphone_op", "op", "tri", 1500, 64, 12001, 50, 150, 1200),
        # large-vocabulary CTC, the whole batch of the sharded configuration on one GPU, fused wrapper
        case("bpe_ctc_fused", "fused", "bpe", 400, 256, 10025, 20, 100, 41),
        # one GPU's share of that batch over eight GPUs, reference-compatible wrapper
        case("bpe_ctc_loss", "loss", "bpe", 400, 32, 10025, 20, 100, 41),
        # irregular lattices (sequence-discriminative training): few sequences, and one GPU's share of a
        # batch of 512 over four GPUs, the largest case
        case("lattice_loss", "loss", "lattice", 2000, 8, 5000, 200, 4000, 100),
        case("lattice_op", "op", "lattice", 2000, 128, 5000, 200, 4000, 100),
        # realignment of a corpus with the triphone system and with lattices
        case("triphone_align", "align", "tri", 1500, 64, 12001, 50, 150, 1200),
        case("lattice_align", "align", "lattice", 1777, 24, 5000, 200, 4000, 100),
    ]


def draw(rng):
    """A case of the listed ranges: any entry point and topology, sizes spread over their logarithm."""

    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    entry = rng.choice(["loss", "fused", "cached", "op", "align"])
    topo = rng.choice(["ctc", "mono", "tri", "bpe", "lattice"])
    lim = {"ctc": (30, 200, 2, 64, 30, 120), "mono": (100, 900, 4, 64, 121, 400), "tri": (300, 1500, 2, 64, 1000, 12001),
           "bpe": (100, 500, 4, 256, 1000, 10025), "lattice": (300, 2000, 2, 96, 500, 5000)}[topo]
    T, B, F = spread(*lim[0:2]), spread(*lim[2:4]), spread(*lim[4:6])
    if topo == "ctc":
        hi = rng.randint(5, max(6, T // 4))
        lo, tlo = max(1, hi // 2), (4 * T) // 5
    elif topo == "bpe":
        hi = rng.randint(5, max(6, T // 4))
        lo, tlo = max(1, hi // 5), min(T, 2 * hi + 1)
    elif topo == "mono":
        hi = rng.randint(5, max(6, T // 8))
        lo, tlo = max(1, hi // 3), (7 * T) // 10
    elif topo == "tri":
        hi = rng.randint(5, max(6, T // 10))
        lo, tlo = max(1, hi // 3), (4 * T) // 5
    else:
        hi = rng.randint(100, min(4000, 2 * T))
        lo, tlo = max(20, hi // 20), max(30, T // 20)
    return {"entry": entry, "topo": topo, "T": T, "B": B, "F": F, "lo": lo, "hi": hi, "tlo": tlo}


def zipf(F):
    p = np.arange(1, F) ** -ZIPF
    return p / p.sum()


def lattice_fsa(rng, S, F):
    """Lattices of S[b] states: every state has a loop, an edge to its successor and up to three more
    to states within the next eight; emissions and weights at random."""
    fr, to, sq, start, end, off = [], [], [], [], [], 0
    for b, n in enumerate(int(s) for s in S):
        j = np.arange(n)
        extra = np.minimum(rng.integers(0, 4, n), np.maximum(n - 2 - j, 0).clip(max=7))
        pick = np.zeros((n, 9), bool)  # column k: an edge to state j + k
        rank = np.where(j[:, None] + np.arange(2, 9) < n, rng.random((n, 7)), 2.0).argsort(1).argsort(1)
        pick[:, 2:] = rank < extra[:, None]
        pick[:, 0] = True
        pick[:-1, 1] = True
        f, k = np.nonzero(pick)
        fr.append(off + f)
        to.append(off + f + k)
        sq.append(np.full(len(f), b))
        start.append(off)
        end.append(off + n - 1)
        off += n
    fr = np.concatenate(fr)
    edges = np.stack([fr, np.concatenate(to), rng.integers(0, F, len(fr)), np.concatenate(sq)]).astype(np.int32)
    weights = (-np.log(rng.uniform(0.05, 1.0, len(fr)))).astype(np.float32)
    dev = torch.device("cuda")
    return (off, torch.from_numpy(edges).to(dev), torch.from_numpy(weights).to(dev),
            torch.tensor([start, end], dtype=torch.int32, device=dev))


def automata(c, rng):
    """The automata of a batch and its sequence lengths."""
    dev = torch.device("cuda")
    B, T, F, topo = c["B"], c["T"], c["F"], c["topo"]
    n = rng.integers(c["lo"], c["hi"] + 1, B)
    lens = rng.integers(c["tlo"], T + 1, B)
    if topo == "lattice":
        lens = np.clip(np.round(rng.lognormal(6.5, 0.6, B) * (T / 2000)), np.maximum(n // 4, c["tlo"]), T)
        fsa = lattice_fsa(rng, n, F)
    elif topo in ("ctc", "bpe"):
        labels = (rng.integers(1, F, (B, c["hi"])) if topo == "ctc"
                  else 1 + np.searchsorted(np.cumsum(zipf(F)), rng.random((B, c["hi"]))).clip(max=F - 2))
        lens = np.maximum(lens, np.minimum(2 * n + 1, T))
        fsa = topology.ctc_topology(torch.from_numpy(labels.astype(np.int32)).to(dev),
                                    torch.from_numpy(n.astype(np.int32)).to(dev))
    else:
        classes = np.zeros((B, 4 * c["hi"] + 2), np.int32)  # class 0: silence
        optional = np.zeros(classes.shape, np.uint8)
        count = np.zeros(B, np.int32)
        for b in range(B):
            if topo == "tri":  # every state tied to a class of its own
                row, opt = np.concatenate([[0], rng.integers(1, F, 3 * n[b]), [0]]), None
            else:  # 40 phones of three states, optional silence between words
                phone = rng.integers(0, 40, n[b])
                states = 1 + 3 * phone[:, None] + np.arange(3)
                sil = np.where(rng.random(n[b]) < 0.2, 0, -1)
                row = np.concatenate([[0], np.concatenate([states, sil[:, None]], 1).ravel()])
                row = row[row >= 0]
                opt = row == 0
                opt[0] = False
                if opt[-1]:
                    opt[-1] = False
                else:
                    row, opt = np.append(row, 0), np.append(opt, False)
                optional[b, :len(row)] = opt
            classes[b, :len(row)] = row
            count[b] = len(row)
        up = lambda x: torch.from_numpy(x).to(dev)  # noqa: E731
        fsa = (topology.hmm_topology(up(classes), up(count), 0.3, 0.7, skip_prob=0.05) if topo == "tri"
               else topology.hmm_topology(up(classes), up(count), 0.3, 0.7, optional=up(optional)))
    return fsa, torch.from_numpy(lens.astype(np.int32)).to(dev)


def prepare(c, seed):
    dev = torch.device("cuda")
    rng = np.random.default_rng(seed)
    fsa, seq_lens = automata(c, rng)
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    op = c["entry"] == "op"
    shape = (c["T"], c["B"], c["F"]) if op else (c["B"], c["T"], c["F"])
    sigma, bias = LOGITS[c["topo"]]
    scores = torch.empty(shape, device=dev)
    for part in scores.split(max(1, (1 << 28) // (shape[1] * shape[2]))):  # bounds the temporary memory
        part.normal_(0.0, sigma, generator=g)
        if bias:
            part[..., 0] += bias
        part.copy_(torch.log_softmax(part, -1))
    if op:
        scores.neg_()
    elif c["entry"] != "align":
        scores.requires_grad_(True)
    state = {"entry": c["entry"], "scores": scores, "fsa": fsa, "seq_lens": seq_lens}
    if c["entry"] == "cached":
        state["cache"] = PlanCache()
    return state


def run(s):
    entry, scores, fsa, seq_lens = s["entry"], s["scores"], s["fsa"], s["seq_lens"]
    if entry == "align":
        return align_viterbi(scores, fsa, seq_lens)
    if entry == "op":
        return core.fbw(scores, fsa[1], fsa[2], fsa[3], seq_lens, fsa[0], core.DebugOptions())
    if entry == "cached":
        loss = fbw_loss_cached(scores, fsa, seq_lens, s["cache"])
    else:
        loss = (fbw_loss if entry == "loss" else fbw_loss_fused)(scores, fsa, seq_lens)
    (grad,) = torch.autograd.grad(loss.sum(), scores)
    return loss, grad


def sizes(c):
    """Expected valid frames, states, edges and distinct classes of a sequence."""
    T, F, topo = c["T"], c["F"], c["topo"]
    n = (c["lo"] + c["hi"]) / 2
    frames = (c["tlo"] + T) / 2
    if topo == "lattice":
        frames = min(T, max(0.4 * T, n / 4))
        states, edges = n, 3.5 * n
        classes = F * (1 - (1 - 1 / F) ** edges)
    elif topo in ("ctc", "bpe"):
        states, edges = 2 * n + 2, 5 * n + 4
        classes = 1 + ((F - 1) * (1 - (1 - 1 / (F - 1)) ** n) if topo == "ctc" else float((1 - (1 - zipf(F)) ** n).sum()))
    elif topo == "tri":
        states, edges = 3 * n + 3, 9 * n + 3
        classes = 1 + (F - 1) * (1 - (1 - 1 / (F - 1)) ** (3 * n))
    else:
        states, edges = 3.2 * n + 3, 6.6 * n + 5
        classes = 1 + 120 * (1 - (1 - 1 / 40) ** n)
    return frames, states, edges, classes


def work(c):
    """Bytes: the 32-byte sectors of the scores that the automata refer to, read once; the dense result
    (posteriors or gradient) and the sums, or the alignment, written once.  Operations per valid frame
    and edge: two additions in each direction and a log-sum (counted as ten) in each direction and for
    the posterior; two additions and a comparison for the alignment."""
    frames, _, edges, classes = sizes(c)
    T, B, F = c["T"], c["B"], c["F"]
    read = B * frames * min(32 * classes, 4 * F) + 16 * B * edges
    if c["entry"] == "align":
        return {"bytes": read + 4 * T * B, "flops": 3 * B * frames * edges}
    return {"bytes": read + 4 * T * B * F + 4 * T * B, "flops": 34 * B * frames * edges}


def tolerance(c):
    if c["entry"] == "align":
        return "exact"  # sums of two operands in a fixed order and comparisons
    # Scores are accumulated over the frames as 32-bit negative logs: at a magnitude M the rounding of
    # one sum is M * 2^-24, and posteriors, differences of such sums, inherit it as a relative error.
    # Measured against the 64-bit oracle (relative 2-norm error in units of M * 2^-23): gradients 0.43
    # (triphone) to 1.1 (lattice), single values up to 18 times that; negative log posteriors 0.016 to
    # 0.03, single values 6 times that; sums 2.6e-6 at most.  Stated: about four times these.
    magnitude = c["T"] * {"ctc": 3.0, "bpe": 8.0, "mono": 6.1, "tri": 13.4, "lattice": 8.5}[c["topo"]]
    rel = max(1e-5, magnitude * 2.0 ** -23 * (0.125 if c["entry"] == "op" else 4.0))
    return {"rel": rel, "max": 20 * rel}
