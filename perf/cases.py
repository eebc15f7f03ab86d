"""What a program has this library do, as cases that can be timed: each a plain dict of sizes and options,
its inputs drawn from a seed, and one pass through the package's public calls.

Sequences are uniform over their alphabet; a query is a mutated copy of letters of its reference, each
letter taking an edit at the pair's rate (a substitution to another letter, a deletion, an insertion after
it). Letters lie in host memory, as every call takes them.
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dinara-align_b200"))

import dinara_align as da  # noqa: E402
from dinara_align import learned, serving  # noqa: E402

DNA = "ACGT"
PROTEIN = "ACDEFGHIKLMNPQRSTVWY"
THIRDS = (1 / 3, 1 / 3)  # the shares of substitutions and deletions; the rest are insertions
HALF_QUARTERS = (0.5, 0.25)
CHUNK = 1 << 25  # letters generated at once


def listed():
    return [
        # A handful of reads measured from a script, as lists of strings: latency and launches.
        dict(name="few_distances", path="few", what="distances", pairs=32, low=150, high=150, rate=0.02),
        # Reads against the molecules they came from: 250 bp at 2% errors.
        dict(name="read_distances", path="distances", policy="plain", pairs=10_000, low=250, high=250, rate_low=0.02,
             rate_high=0.02, thirds=True, pinned=False),
        # Clustering reads of all lengths and error rates: the learned band over an uneven batch.
        dict(name="uneven_distances", path="distances", policy="learned", pairs=70_000, low=100, high=20_000,
             rate_low=0.005, rate_high=0.15, thirds=False, pinned=True),
        # Short reads' scores and CIGARs against the windows a mapper gave them, a large batch.
        dict(name="read_alignments", path="alignments", mode="global", letters=4, match=0, mismatch=-4, opening=-6,
             extension=-2, pairs=200_000, low=100, high=300, rate=0.05, pinned=True),
        # Reads searched for in longer targets: local scores.
        dict(name="local_scores", path="scores", mode="local", letters=4, match=2, mismatch=-4, opening=-4,
             extension=-2, pairs=20_000, low=150, high=1000, target_low=1000, target_high=5000, rate=0.08, pinned=True),
        # The same with each hit's CIGAR and span.
        dict(name="local_alignments", path="alignments", mode="local", letters=4, match=2, mismatch=-4, opening=-4,
             extension=-2, pairs=5_000, low=150, high=1000, target_low=1000, target_high=5000, rate=0.08, pinned=False),
        # Reads placed in their candidate windows: the query whole, the window's ends free.
        dict(name="infix_alignments", path="alignments", mode="infix", letters=4, match=2, mismatch=-4, opening=-4,
             extension=-2, pairs=20_000, low=100, high=300, flank_low=20, flank_high=400, rate=0.05, pinned=False),
        # Seeds extended to the right until the score drops off; a third of the queries part from their
        # reference half way.
        dict(name="extensions", path="alignments", mode="extension", letters=4, match=2, mismatch=-4, opening=-4,
             extension=-2, pairs=10_000, low=100, high=1000, flank_low=0, flank_high=100, rate=0.05, anchor=0,
             zdrop=100, end_bonus=10, pinned=False),
        # Least-cost alignments under gap-affine costs, ties to the left.
        dict(name="cost_alignments", path="costs", mismatch=4, opening=6, extension=2, pairs=20_000, low=100,
             high=1000, rate_low=0.01, rate_high=0.10, ties="left", trace=True, pinned=False),
        # A service's mixed load: requests of a few to many pairs, reads of 100 bp to 50 kbp.
        dict(name="served_scores", path="serving", requests=8, most_pairs=128, low=100, high=50_000, rate_low=0.01,
             rate_high=0.10),
        # Proteins scored against each other under a 20-letter table.
        dict(name="protein_scores", path="scores", mode="local", letters=20, match=5, mismatch=-2, opening=-10,
             extension=-1, pairs=10_000, low=60, high=600, target_low=100, target_high=1000, rate=0.3, pinned=False),
        # One training batch of the band predictor, forward and backward.
        dict(name="predictor_gradients", path="gradients", batch=4096),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    path = rng.choice(["few", "distances", "distances", "alignments", "alignments", "alignments", "scores", "scores",
                       "costs", "costs", "serving", "gradients"])
    if path == "few":
        low = _log_int(rng, 20, 1000)
        return dict(path=path, what=rng.choice(["distances", "alignments"]), pairs=_log_int(rng, 1, 60), low=low,
                    high=low + rng.randint(0, 100), rate=rng.uniform(0.0, 0.1))
    if path == "distances":
        low = _log_int(rng, 30, 2000)
        high = min(20_000, _log_int(rng, low, 20 * low))
        pairs = min(70_000, max(1, _log_int(rng, 100, 70_000)))
        pairs = max(1, min(pairs, 250_000_000 // max(1, (low + high) // 2)))
        rate_low = rng.uniform(0.0, 0.05)
        return dict(path=path, policy=rng.choice(["plain", "learned"]), pairs=pairs, low=low, high=high,
                    rate_low=rate_low, rate_high=rate_low + rng.uniform(0.0, 0.1), thirds=rng.random() < 0.5,
                    pinned=rng.random() < 0.5)
    if path in ("alignments", "scores"):
        mode = rng.choice(["global", "local", "infix", "extension"])
        letters = rng.choice([4, 4, 4, 5, 20])
        table = rng.choice([(2, -4, -4, -2), (1, -3, -5, -2), (2, -4, -6, -1)]) if letters < 20 else (5, -2, -10, -1)
        if letters == 4 and mode == "global" and rng.random() < 0.5:
            table = (0, -4, -6, -2)
        low = _log_int(rng, 40, 600)
        high = low + _log_int(rng, 1, 600)
        case = dict(path=path, mode=mode, letters=letters, match=table[0], mismatch=table[1], opening=table[2],
                    extension=table[3], low=low, high=high, rate=rng.uniform(0.0, 0.15) * (2 if letters == 20 else 1),
                    pinned=rng.random() < 0.5)
        most = 30_000 if mode == "global" else 5_000
        if mode == "local":
            case.update(target_low=high, target_high=high + _log_int(rng, 10, 3000))
        if mode in ("infix", "extension"):
            flank = rng.randint(0, 60)
            case.update(flank_low=flank, flank_high=flank + _log_int(rng, 1, 500))
        if mode == "extension":
            case.update(anchor=rng.randint(0, 1), zdrop=rng.choice([-1, 20, 100, 400]),
                        end_bonus=rng.choice([-1, 5, 10]))
        # At most two thousand million cells, as the largest of the listed ones has.
        target = high + case.get("flank_high", 0) * 2
        cells = high * max(target, case.get("target_high", 0))
        case["pairs"] = _log_int(rng, 10, max(11, min(most, 2_000_000_000 // cells)))
        return case
    if path == "costs":
        unit = rng.random() < 0.4
        low = _log_int(rng, 50, 800)
        rate_low = rng.uniform(0.0, 0.05)
        return dict(path=path, mismatch=1 if unit else rng.choice([3, 4, 5]), opening=0 if unit else rng.randint(4, 9),
                    extension=1 if unit else rng.choice([1, 2]), pairs=_log_int(rng, 10, 10_000), low=low,
                    high=low + _log_int(rng, 1, 500), rate_low=rate_low, rate_high=rate_low + rng.uniform(0.0, 0.05),
                    ties=rng.choice(["left", "left", "right"]), trace=rng.random() < 0.8, pinned=rng.random() < 0.5)
    if path == "serving":
        return dict(path=path, requests=rng.randint(2, 8), most_pairs=_log_int(rng, 8, 100), low=100,
                    high=_log_int(rng, 1000, 40_000), rate_low=0.01, rate_high=rng.uniform(0.01, 0.1))
    return dict(path=path, batch=_log_int(rng, 200, 4096))


# ---- inputs -----------------------------------------------------------------------------------------

_DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


class _Source:
    """Random tensors of one seed."""

    def __init__(self, seed):
        self.generator = torch.Generator(device=_DEVICE).manual_seed(0x5EED + int(seed))

    def uniform(self, count):
        return torch.rand(count, generator=self.generator, device=_DEVICE, dtype=torch.float64)

    def integers(self, low, high, count):
        """`count` integers of [low, high]."""
        return torch.randint(low, high + 1, (count,), generator=self.generator, device=_DEVICE)

    def letters(self, count, size):
        return torch.randint(0, size, (count,), generator=self.generator, device=_DEVICE, dtype=torch.uint8)


def _starts(lengths):
    out = torch.zeros(len(lengths) + 1, dtype=torch.int64, device=lengths.device)
    torch.cumsum(lengths, 0, out=out[1:])
    return out


def _places(lengths):
    """For segments of `lengths` end to end: each element's segment, its place within it, and their starts."""
    starts = _starts(lengths)
    owner = torch.repeat_interleave(torch.arange(len(lengths), device=lengths.device), lengths)
    return owner, torch.arange(len(owner), device=lengths.device) - starts[owner], starts


def _mutated(source, codes, owner, rates, pairs, split, size):
    """Mutated copies of segments end to end: their codes and lengths."""
    rate = rates[owner]
    roll = torch.rand(len(codes), generator=source.generator, device=_DEVICE, dtype=torch.float32).double()
    substituted = roll < rate * split[0]
    deleted = (roll >= rate * split[0]) & (roll < rate * (split[0] + split[1]))
    inserted = (roll >= rate * (split[0] + split[1])) & (roll < rate)
    shifted = (codes.long() + source.integers(1, size - 1, len(codes))) % size
    letters = torch.where(substituted, shifted.to(torch.uint8), codes)
    emitted = 1 - deleted.long() + inserted.long()
    place = _starts(emitted)
    out = torch.empty(int(place[-1]), dtype=torch.uint8, device=codes.device)
    kept = ~deleted
    out[place[:-1][kept]] = letters[kept]
    out[place[:-1][inserted] + 1] = source.letters(int(inserted.sum()), size)
    lengths = torch.zeros(pairs, dtype=torch.int64, device=codes.device).index_add_(0, owner, emitted)
    return out, lengths


def _chunk(source, size, references, offsets, sources, rates, split, parted):
    """Letters and interleaved lengths of pairs: references of `references` letters, each query mutated from
    the `sources` letters at `offsets` of its reference; a `parted` query's second half is letters of its own."""
    pairs = len(references)
    a = source.letters(int(references.sum()), size)
    a_starts = _starts(references)
    owner, within, _ = _places(sources)
    b, b_lengths = _mutated(source, a[a_starts[owner] + offsets[owner] + within], owner, rates, pairs, split, size)
    if parted is not None:
        owner, within, _ = _places(b_lengths)
        apart = parted[owner] & (2 * within >= b_lengths[owner])
        b = torch.where(apart, source.letters(len(b), size), b)
    lengths = torch.stack([references, b_lengths], 1).reshape(-1)
    starts = _starts(lengths)
    letters = torch.empty(int(starts[-1]), dtype=torch.uint8, device=a.device)
    owner, within, _ = _places(references)
    letters[starts[0:-1:2][owner] + within] = a
    owner, within, _ = _places(b_lengths)
    letters[starts[1::2][owner] + within] = b
    return letters, lengths


def _tape(case, seed, alphabet):
    """The case's pairs as a Tape in host memory, page-locked where the case says so."""
    source = _Source(seed)
    pairs, low, high = case["pairs"], case["low"], case["high"]
    if high > 3 * low:
        lengths = torch.exp(math.log(low) + source.uniform(pairs) * math.log(high / low)).round().long()
    else:
        lengths = source.integers(low, high, pairs)
    references, offsets = lengths, torch.zeros_like(lengths)
    parted = None
    if "target_low" in case:
        references = torch.maximum(lengths, source.integers(case["target_low"], case["target_high"], pairs))
        offsets = (source.uniform(pairs) * (references - lengths + 1)).long()
    elif case.get("mode") == "infix":
        offsets = source.integers(case["flank_low"], case["flank_high"], pairs)
        references = offsets + lengths + source.integers(case["flank_low"], case["flank_high"], pairs)
    elif case.get("mode") == "extension":
        references = lengths + source.integers(case["flank_low"], case["flank_high"], pairs)
        parted = source.uniform(pairs) < 1 / 3
    rates = torch.full((pairs,), float(case["rate"]), dtype=torch.float64, device=_DEVICE) if "rate" in case else (
        case["rate_low"] + source.uniform(pairs) * (case["rate_high"] - case["rate_low"]))
    split = THIRDS if case.get("thirds") else HALF_QUARTERS
    # A chunk of pairs at a time, each of at most CHUNK reference letters.
    ends = _starts(references).cpu().numpy()
    pieces, sizes, first = [], [], 0
    while first < pairs:
        last = max(first + 1, int(np.searchsorted(ends, ends[first] + CHUNK, side="right")) - 1)
        part = slice(first, min(last, pairs))
        letters, counts = _chunk(source, len(alphabet), references[part], offsets[part], lengths[part], rates[part],
                                 split, None if parted is None else parted[part])
        pieces.append(letters)
        sizes.append(counts)
        first = part.stop
    codes = torch.frombuffer(bytearray(alphabet.encode()), dtype=torch.uint8).to(_DEVICE)
    total = sum(len(piece) for piece in pieces)
    pinned = bool(case.get("pinned")) and _DEVICE == "cuda"
    letters = torch.empty(total, dtype=torch.uint8, pin_memory=pinned)
    at = 0
    for piece in pieces:
        letters[at:at + len(piece)].copy_(codes[piece.long()])
        at += len(piece)
    offsets = np.zeros(2 * pairs + 1, dtype=np.int64)
    np.cumsum(torch.cat(sizes).cpu().numpy(), out=offsets[1:])
    letters = letters.numpy()
    if case.get("mode") == "extension" and case["anchor"] == 1:
        letters = _turned(letters, offsets)
    return da.Tape(letters, offsets)


def _turned(letters, offsets):
    """Every sequence of a tape back to front."""
    out = np.empty_like(letters)
    for k in range(len(offsets) - 1):
        out[offsets[k]:offsets[k + 1]] = letters[offsets[k]:offsets[k + 1]][::-1]
    return out


def _alphabet(case):
    return {4: DNA, 5: DNA + "N", 20: PROTEIN}[case.get("letters", 4)]


def _scoring(case):
    alphabet = _alphabet(case)
    if len(alphabet) < 20:
        return da.Scoring.uniform(case["match"], case["mismatch"], case["opening"], case["extension"], alphabet)
    # A symmetric table in a substitution matrix's range: matches of 4 and up, the rest from -4 to 2.
    rng = np.random.default_rng(20)
    table = rng.integers(case["mismatch"] - 2, 3, size=(20, 20))
    table = np.triu(table, 1) + np.triu(table, 1).T + np.diag(rng.integers(case["match"] - 1, case["match"] + 4, 20))
    return da.Scoring.tabulated(alphabet, [int(v) for v in table.reshape(-1)], case["opening"], case["extension"])


def _mode(case):
    if case["mode"] == "extension":
        return da.Mode.extension(0, case["anchor"], zdrop=case["zdrop"], end_bonus=case["end_bonus"])
    return {"global": da.Mode.GLOBAL, "local": da.Mode.local(), "infix": da.Mode.INFIX}[case["mode"]]


_kept = {}


def _predictor():
    """The band predictor a program trains once and keeps."""
    if "predictor" not in _kept:
        predictor = learned.Predictor()
        predictor.train(pairs=400_000, epochs=4, batch=1024, seed=2024)
        _kept["predictor"] = predictor.parameters() + (predictor.margins(),)
    return _kept["predictor"]


def _server():
    """The service a program opens once."""
    if "server" not in _kept:
        _kept["server"] = serving.Server(slots=4)
    return _kept["server"]


def prepare(case, seed):
    path = case["path"]
    if path == "gradients":
        x, t, flat = _training_batch(case, seed)
        predictor = learned.Predictor()
        return dict(path=path, predictor=predictor, flat=flat, x=x, t=t)
    if path == "serving":
        counts = np.geomspace(1, case["most_pairs"], case["requests"]).round().astype(int)
        tapes = [_tape(dict(case, pairs=int(count)), 97 * seed + k, DNA) for k, count in enumerate(counts)]
        return dict(path=path, server=_server(), tapes=tapes, scoring=da.Scoring.uniform(0, -4, -6, -2))
    if path == "few":
        tape = _tape(case, seed, DNA)
        return dict(path=path, what=case["what"], scoring=da.Scoring.dna(), text=_text_room(case),
                    references=[tape.reference(k).decode() for k in range(tape.pairs)],
                    queries=[tape.query(k).decode() for k in range(tape.pairs)])
    tape = _tape(case, seed, _alphabet(case))
    if path == "distances":
        predictor = None
        if case["policy"] == "learned":
            parameters, margin, slack, margins = _predictor()
            predictor = learned.Predictor()
            predictor.install(parameters, margin, slack)
            predictor.margins(margins)
        return dict(path=path, tape=tape, predictor=predictor,
                    policy=da._native.BAND_LEARNED if predictor else da._native.BAND_PLAIN)
    if path == "costs":
        return dict(path=path, tape=tape, costs=da.Costs.affine(case["mismatch"], case["opening"], case["extension"]),
                    ties=case["ties"], trace=case["trace"], text=_text_room(case))
    return dict(path=path, tape=tape, scoring=_scoring(case), mode=_mode(case), text=_text_room(case))


def _text_room(case):
    """A program's own buffer for a batch's CIGARs, of one size whatever the seed: about eight characters an
    edit, and as much again by half."""
    length, _square = _mean(case["low"], case["high"])
    rate = case["rate"] if "rate" in case else (case["rate_low"] + case["rate_high"]) / 2
    return np.zeros(4096 + int(case.get("pairs", 1) * 1.5 * (12 + 8 * rate * length)), dtype=np.uint8)


def _kept_text(room, data):
    """A batch's CIGAR bytes moved into the program's buffer."""
    if len(data) > len(room):
        raise ValueError(f"{len(data)} CIGAR bytes for a buffer of {len(room)}")
    room[:len(data)] = data
    return room


def _training_batch(case, seed):
    """A batch of features and targets in the range training meets, and parameters at the scale of a start."""
    rng = np.random.default_rng(1000 + seed)
    flat = rng.normal(0, 0.1, size=learned.PARAMETERS).astype(np.float32)
    x = np.abs(rng.normal(0, 0.5, size=(case["batch"], learned.INPUTS))).astype(np.float32)
    t = rng.uniform(0, 0.2, size=case["batch"]).astype(np.float32)
    return x, t, flat


def run(state):
    path = state["path"]
    if path == "gradients":
        state["predictor"].install(state["flat"])
        return state["predictor"].gradients(state["x"], state["t"])
    if path == "serving":
        server = state["server"]
        tickets = [server.submit(tape, state["scoring"]) for tape in state["tapes"]]
        done = [server.wait(ticket) for ticket in tickets]
        return [(code, scores, statuses) for code, scores, statuses, _timing in done]
    if path == "few":
        if state["what"] == "distances":
            return np.asarray(da.distances(state["references"], state["queries"]))
        found = da.alignments(state["references"], state["queries"], state["scoring"])
        text = np.frombuffer(" ".join(a.cigar for a in found).encode(), dtype=np.uint8)
        return np.asarray([a.score for a in found]), _kept_text(state["text"], text)
    if path == "distances":
        return da.distances_tape(state["tape"], policy=state["policy"])
    if path == "costs":
        found, offsets, data = da.cost_alignments_tape(state["tape"], state["costs"], ties=state["ties"],
                                                       trace=state["trace"])
        return found, offsets, _kept_text(state["text"], data)
    if path == "scores":
        return da.scores_tape(state["tape"], state["scoring"], state["mode"])
    found, spans, offsets, data, statuses = da.alignments_tape(state["tape"], state["scoring"], state["mode"])
    return found, spans, offsets, _kept_text(state["text"], data), statuses


# ---- what a pass cannot do without, and how far another implementation may differ ---------------------

def _mean(low, high):
    """The mean of the lengths _tape draws from [low, high], and of their squares."""
    if high > 3 * low:
        span = math.log(high / low)
        return (high - low) / span, (high * high - low * low) / (2 * span)
    return (low + high) / 2, (low * low + low * high + high * high) / 3


def work(case):
    path = case["path"]
    if path == "gradients":
        # Forward, and backward to weights and activations, of 258 -> 64 -> 64 -> 1.
        weights = 258 * 64 + 64 * 64 + 64
        return {"bytes": 4 * (case["batch"] * 259 + 2 * learned.PARAMETERS),
                "flops": case["batch"] * (6 * weights - 2 * 258 * 64)}
    length, square = _mean(case["low"], case["high"])
    rate = case["rate"] if "rate" in case else (case["rate_low"] + case["rate_high"]) / 2
    if path == "serving":
        counts = np.geomspace(1, case["most_pairs"], case["requests"]).round().sum()
        # Seven operations a cell of the diagonals that an alignment at this rate needs, two a letter edited.
        return {"bytes": float(counts * (2 * length + 4)), "flops": float(counts * 7 * square * 2 * rate)}
    pairs = case["pairs"]
    if path == "distances" or (path == "few" and case["what"] == "distances"):
        # A word step (64 cells) takes about 20 64-bit operations; a column needs the band's words.
        words = square * 2 * rate / 64 + length
        return {"bytes": pairs * (2 * length + 8), "flops": pairs * 40 * words}
    if path == "costs":
        # Diagonal fronts: one value a diagonal a cost, three layers under gap-affine costs.
        edits = rate * length
        cost = edits * (case["mismatch"] + case["opening"] + case["extension"]) / 2
        layers = 1 if case["opening"] == 0 else 3
        return {"bytes": pairs * (2 * length + 8 + (4 * edits if case["trace"] else 0)),
                "flops": pairs * (layers * 4 * (cost + 1) ** 2 + 2 * length)}
    target = length
    if "target_low" in case:
        target = _mean(case["target_low"], case["target_high"])[0]
    elif "flank_low" in case:
        target = length + (case["flank_low"] + case["flank_high"]) / (1 if case["mode"] == "infix" else 2)
    # Global pairs need the diagonals their score proves, at least 32; the others their whole matrix.
    cells = (32 * length if case.get("mode", "global") == "global" else length * target)
    out = 16 if path == "scores" else 48 + 6 * rate * length
    return {"bytes": pairs * (length + target + out), "flops": pairs * 7 * cells}


def tolerance(case):
    # Integer arithmetic throughout, except the predictor's fp32 sums (up to 1e-6 off 64 bits, and from themselves).
    return {"rel": 4e-6} if case["path"] == "gradients" else "exact"


def exact(case, seed):
    if case["path"] != "gradients":
        return None
    x, t, flat = (value.astype(np.float64) for value in _training_batch(case, seed))
    at = np.cumsum([258 * 64, 64, 64 * 64, 64, 64])
    w1, b1, w2, b2, w3, b3 = np.split(flat, at)
    w1, w2 = w1.reshape(258, 64), w2.reshape(64, 64)
    h1 = np.maximum(x @ w1 + b1, 0)
    h2 = np.maximum(h1 @ w2 + b2, 0)
    error = h2 @ w3 + b3[0] - t
    dy = 2 * error / len(t)
    d2 = np.outer(dy, w3) * (h2 > 0)
    d1 = (d2 @ w2.T) * (h1 > 0)
    gradients = np.concatenate([(x.T @ d1).reshape(-1), d1.sum(0), (h1.T @ d2).reshape(-1), d2.sum(0), h2.T @ dy,
                                [dy.sum()]])
    return gradients, float(np.mean(error * error))
