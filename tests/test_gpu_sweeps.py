"""The sweeps' own edges against the oracle: strips and lane groups at their widths and a column either side, the
16-bit forms at their limits and a step past them, hits cut to their rows, kept fronts at their sizes, the
first round's list, and the gradients' slices. Every result is an exact integer or text, except the gradients."""

import ctypes
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BIG = 1 << 40
PROTEIN = "ACDEFGHIKLMNPQRSTVWY"
THIRTY_TWO = "ABCDEFGHIJKLMNOPQRSTUVWXYZ012345"


def _mutated(rng, source, rate, alphabet):
    out = []
    for letter in source:
        roll = rng.random()
        if roll < rate / 2:
            out.append(rng.choice(list(alphabet)))
        elif roll < 3 * rate / 4:
            continue
        elif roll < rate:
            out.append(letter + rng.choice(list(alphabet)))
        else:
            out.append(letter)
    return "".join(out)


def _text(rng, length, alphabet="ACGT"):
    return "".join(np.asarray(list(alphabet))[rng.integers(0, len(alphabet), size=length)])


def _table(scoring):
    return np.asarray(scoring.table, dtype=np.int8)


def _tabulated(da, rng, alphabet, opening=-10, extension=-1):
    size = len(alphabet)
    table = rng.integers(-4, 3, size=(size, size))
    table = np.triu(table, 1) + np.triu(table, 1).T + np.diag(rng.integers(3, 9, size))
    return da.Scoring.tabulated(alphabet, [int(v) for v in table.reshape(-1)], opening, extension)


# ---- long pairs in strips of 1,024 columns ------------------------------------------------------------

# The last three: steps (largest shifted entry plus opening) of 100, the strips' limit, and 101 and 180, past it.
@pytest.mark.parametrize("entries", [(0, -4, -6, -2), (2, -4, -4, -2), (1, -1, 0, -1), (40, -20, -40, -10),
                                     (41, -20, -40, -10), (60, -60, -100, -10)])
def test_long_pairs_in_strips(da, oracle, entries):
    """Pairs past 16-bit pair sweeps: one strip and a letter, whole strips and a letter either side, more than
    eight strips (a warp's second), bands proven, bands widened and bands given up for the whole matrix."""
    rng = np.random.default_rng(abs(sum(entries)) + 5)
    scoring = da.Scoring.uniform(*entries)
    refs, queries = [], []
    for rows, columns, rate in ((1025, 1025, 0.05), (2600, 2048, 0.4), (2049, 2600, 0.3), (3071, 3072, 0.02),
                                (4100, 4097, 0.1), (5000, 5000, 0.003), (5000, 1025, 0.0), (1025, 5000, 0.0),
                                (9300, 9300, 0.01), (9300, 9217, 0.25)):
        source = _text(rng, max(rows, columns))
        refs.append(source[:rows])
        queries.append(_mutated(rng, source, rate, "ACGT")[:columns] if rate else _text(rng, columns))
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text) for pair in zip(refs, queries) for text in pair])
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    expected = oracle.batch_scores(coded, tape.offsets, _table(scoring), 4, op, ex, oracle.GLOBAL, threads=8)
    np.testing.assert_array_equal(da.scores_tape(tape, scoring), expected)


@pytest.mark.parametrize("pairs", [75, 592])
def test_many_long_pairs_in_strips(da, oracle, pairs):
    """Enough long pairs for strips of 16 columns a lane: a cluster a pair, and a block a pair (10 pairs, above,
    take eight columns a lane)."""
    rng = np.random.default_rng(pairs)
    scoring = da.Scoring.uniform(30, -40, -20, -3)
    refs = [_text(rng, 1025 + int(rng.integers(0, 90))) for _ in range(pairs)]
    queries = [_text(rng, 1025 + int(rng.integers(0, 90))) for _ in range(pairs)]
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text) for pair in zip(refs, queries) for text in pair])
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    expected = oracle.batch_scores(coded, tape.offsets, _table(scoring), 4, op, ex, oracle.GLOBAL, threads=8)
    np.testing.assert_array_equal(da.scores_tape(tape, scoring), expected)


def _shifted(rng, length, size, first, second, rate=0.01):
    """A sequence, and its copy with `size` letters put in at the share `first` of it and as many taken out at
    `second`: between the two the alignment lies `size` diagonals off."""
    source = _text(rng, length)
    copy = _mutated(rng, source, rate, "ACGT")
    a, b = int(first * len(copy)), int(second * len(copy))
    return source, copy[:a] + _text(rng, size) + copy[a:b] + copy[b + size:]


# The last table's steps (180) are past the 16-bit strips: a first band of 2,048.
@pytest.mark.parametrize("entries", [(2, -4, -4, -2), (0, -4, -6, -2), (60, -60, -100, -10)])
def test_long_alignments_off_the_diagonals(da, oracle, entries):
    """Alignments whose paths leave the main diagonals: bands proven at once, at the width a low score asked for, at
    2,048 where that is too wide for its worth, and not at all; recorded over what their own scores need."""
    rng = np.random.default_rng(abs(sum(entries)) + 97)
    scoring = da.Scoring.uniform(*entries)
    shapes = [(4200, 40, 0.3, 0.6), (4300, 300, 0.1, 0.9), (5000, 300, 0.2, 0.8), (5200, 700, 0.3, 0.7),
              (7000, 120, 0.1, 0.95), (9000, 300, 0.3, 0.6), (9000, 900, 0.05, 0.9), (6000, 1500, 0.4, 0.5)]
    pairs = [_shifted(rng, *shape) for shape in shapes]
    pairs += [(b, a) for a, b in pairs[:4]]
    pairs += [(_text(rng, 4500), _text(rng, 4400)), (_shifted(rng, 6000, 300, 0.2, 0.8)[0],
                                                     _shifted(rng, 6000, 300, 0.2, 0.8)[1][:5200])]
    refs, queries = [a for a, _b in pairs], [b for _a, b in pairs]
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text) for pair in pairs for text in pair])
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    expected, cigars = oracle.batch_alignments(coded, tape.offsets, _table(scoring), 4, op, ex, oracle.GLOBAL, threads=8)
    found = da.alignments(refs, queries, scoring)
    assert [a.score for a in found] == list(expected)
    assert [a.cigar for a in found] == cigars


def test_long_alignments_record_what_their_scores_need(da):
    """20,000 letters with 300 put in and taken out: the score lies 3,600 below the best, so 600 gap letters or so
    outside a band cost more, and with a strip of 512 columns no more than 2,048 places a row are recorded. (The
    band that finds the score, from the low one that 256 diagonals give, takes some 6,000.)"""
    import bench

    rng = np.random.default_rng(20)
    source, copy = _shifted(rng, 20_000, 300, 1 / 3, 2 / 3)
    tape = da.Tape.of([source], [copy])
    native, lib = da._native, da._native.lib()
    handle = lib.dinara_gpu_new(0)
    scoring, _table_kept, _alphabet_kept = da.Scoring.uniform(2, -4, -4, -2)._struct()
    mode, timing = da.Mode.GLOBAL._struct(), bench.Timing()
    native.check(lib.dinara_gpu_resident_load(handle, 1, tape.letters.ctypes.data,
                                              native.pointer(tape.offsets, ctypes.c_int64), ctypes.byref(scoring)), handle)
    native.check(lib.dinara_gpu_resident_align(handle, ctypes.byref(mode), 1, 1, ctypes.byref(timing)), handle)
    lib.dinara_gpu_free(handle)
    assert 0 < timing.whole_cells < 20_000 * 2_048


# ---- local alignments recorded over their hits' rows ----------------------------------------------------

@pytest.mark.parametrize("alphabet", ["ACGT", "ACGTN", PROTEIN])
def test_hits_in_long_targets(da, oracle, alphabet):
    """Queries planted once, twice alike (the first hit wins, its letters placed at their last occurrence) and not
    at all, at shape widths and a column either side, in targets whose hits start at every letter of a packed
    word; repeats of one letter; gaps that cost nothing a letter, whose hits may span any rows."""
    rng = np.random.default_rng(len(alphabet))
    refs, queries = [], []
    for trial, width in enumerate((1, 7, 16, 17, 63, 64, 65, 128, 129, 256, 257, 320, 321, 511, 512, 513, 800)):
        query = _text(rng, width, alphabet)
        lead = 100 + trial
        for copies in (1, 2, 0):
            target = _text(rng, lead, alphabet)
            for _ in range(copies):
                target += query + _text(rng, 200, alphabet)
            target += _text(rng, 400, alphabet)
            refs.append(target)
            queries.append(_mutated(rng, query, 0.06, alphabet))
    refs += [alphabet[0] * 300, alphabet[0] * 300, alphabet[0] * 40, "", alphabet[1] * 30]
    queries += [alphabet[0] * 20, alphabet[1] * 9, alphabet[0] * 120, alphabet[0], ""]
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text, alphabet) for pair in zip(refs, queries) for text in pair if text])
    scorings = [_tabulated(da, rng, alphabet), da.Scoring.uniform(2, -4, -4, -2, alphabet),
                da.Scoring.uniform(2, -3, -5, 0, alphabet)]
    for scoring in scorings:
        op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
        expected, cigars = oracle.batch_alignments(coded, tape.offsets, _table(scoring), len(alphabet), op, ex,
                                                   oracle.LOCAL, threads=8)
        np.testing.assert_array_equal(da.scores_tape(tape, scoring, da.Mode.local()), expected)
        found = da.alignments(refs, queries, scoring, da.Mode.local())
        assert [a.score for a in found] == list(expected)
        assert [a.cigar for a in found] == cigars
        for a, ref, query in zip(found, refs, queries):
            rows = ref[a.reference_start:a.reference_end]
            columns = query[a.query_start:a.query_end]
            top, bottom = a.gapped(ref, query)
            assert (top.replace("-", ""), bottom.replace("-", "")) == (rows, columns)
            assert a.reference_start == (ref.rfind(rows) if rows else 0)
            assert a.query_start == (query.rfind(columns) if columns else 0)


@pytest.mark.parametrize("entries", [(1, -1, 0, -1), (1, -3, -5, -2)])
def test_long_pairs_beside_hits(da, oracle, entries):
    """Pairs at and past 4,096 x 2,048 letters, whose hits no 16-bit sweep finds, in a batch of pairs whose hits it
    does: their whole matrices are recorded."""
    rng = np.random.default_rng(abs(sum(entries)) + 41)
    scoring = da.Scoring.uniform(*entries)
    refs, queries = [], []
    for rows, columns in ((4095, 2048), (4096, 2047), (4096, 2048), (4200, 4150), (300, 200), (900, 600)):
        source = _text(rng, columns)
        refs.append((_text(rng, 100) + _mutated(rng, source, 0.05, "ACGT") + _text(rng, rows))[:rows])
        queries.append(source)
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text) for pair in zip(refs, queries) for text in pair])
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    expected, cigars = oracle.batch_alignments(coded, tape.offsets, _table(scoring), 4, op, ex, oracle.LOCAL, threads=8)
    found = da.alignments(refs, queries, scoring, da.Mode.local())
    assert [a.score for a in found] == list(expected)
    assert [a.cigar for a in found] == cigars


@pytest.mark.parametrize("entries", [(2, -4, -4, -2), (1, -3, -5, 0), (0, -4, -6, -2)])
def test_scores_past_320_columns(da, oracle, entries):
    """Enough two-bit pairs for the strips of 384 to 768 columns, at the widths where one gives way to the next, a
    column either side, and past one strip of each; short and a few tall, no band proving them."""
    rng = np.random.default_rng(abs(sum(entries)) + 11)
    scoring = da.Scoring.uniform(*entries)
    widths = [w + d for w in (320, 384, 448, 512, 640, 768, 896, 1024, 1152, 1280, 1536) for d in (-1, 0, 1)]
    refs, queries = [], []
    for k in range(9600):
        source = _text(rng, widths[k % len(widths)])
        refs.append(source[100:100 + 3 + k % 30] if k >= 66 else _text(rng, 60) + source[:700])
        queries.append(source)
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text) for pair in zip(refs, queries) for text in pair])
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    for mode, kind in ((da.Mode.GLOBAL, oracle.GLOBAL), (da.Mode.local(), oracle.LOCAL)):
        if kind == oracle.LOCAL and entries[0] <= 0:
            continue
        expected = oracle.batch_scores(coded, tape.offsets, _table(scoring), 4, op, ex, kind, threads=8)
        np.testing.assert_array_equal(da.scores_tape(tape, scoring, mode), expected)


@pytest.mark.parametrize("alphabet", ["ACGT", PROTEIN])
@pytest.mark.parametrize("local", [False, True])
def test_recorded_pairs_that_fill_the_gpu(da, oracle, alphabet, local):
    """5,000 pairs: enough for the 16-bit recording globally, for a band's leftovers, and for its strips of 256
    columns; widths a column either side of its lane groups', one strip and more, an odd pair out."""
    rng = np.random.default_rng(len(alphabet) + local)
    scoring = da.Scoring.uniform(2, -4, -4, -2, alphabet)
    widths = (1, 15, 16, 17, 31, 32, 33, 64, 65, 128, 129)
    refs, queries = [], []
    for k in range(5001):
        width = widths[k % len(widths)] if k >= 40 else (255, 256, 257, 512, 513, 600, 768, 769)[k % 8]
        source = _text(rng, width, alphabet)
        refs.append(_text(rng, 3 + k % 30, alphabet) + (source[:40 + width // 2] if k % 3 else ""))
        queries.append(_mutated(rng, source, 0.1, alphabet) or alphabet[0])
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text, alphabet) for pair in zip(refs, queries) for text in pair])
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    expected, cigars = oracle.batch_alignments(coded, tape.offsets, _table(scoring), len(alphabet), op, ex,
                                               oracle.LOCAL if local else oracle.GLOBAL, threads=8)
    found = da.alignments(refs, queries, scoring, da.Mode.local() if local else da.Mode.GLOBAL)
    assert [a.score for a in found] == list(expected)
    assert [a.cigar for a in found] == cigars


# ---- free ends and extensions in 16-bit halves ----------------------------------------------------------

WIDTHS = (1, 8, 9, 15, 16, 17, 63, 64, 65, 127, 128, 129, 255, 256, 257, 320, 321, 512, 513, 700)


def _placed_pairs(rng, alphabet):
    refs, queries = [], []
    for width in WIDTHS:
        source = _text(rng, width, alphabet)
        for flank in (0, 1, 15, 16, 90):
            refs.append(_text(rng, flank, alphabet) + source + _text(rng, 2 * flank, alphabet))
            queries.append(_mutated(rng, source, 0.08, alphabet))
    return refs, queries


def _span(a):
    return a.reference_start, a.reference_end, a.query_start, a.query_end


# The last two: gaps past the 16-bit forms' limit, and values past it on the longer pairs.
@pytest.mark.parametrize("alphabet,entries", [("ACGT", (2, -4, -4, -2)), ("ACGT", (1, -3, -5, 0)),
                                              ("ACGTN", (2, -4, -6, -1)), (THIRTY_TWO, (5, -2, -10, -1)),
                                              ("ACGT", (5, -4, -2000, -1)), ("ACGT", (40, -30, -40, -30))])
def test_free_ends_and_extensions_at_the_widths(da, oracle, alphabet, entries):
    rng = np.random.default_rng(len(alphabet) + abs(sum(entries)))
    scoring = da.Scoring.uniform(*entries, alphabet)
    refs, queries = _placed_pairs(rng, alphabet)
    # Queries that part from their references half way, for the Z-drop.
    for k in range(0, len(queries), 3):
        queries[k] = queries[k][:len(queries[k]) // 2] + _text(rng, len(queries[k]) // 2, alphabet)
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    coded = [(oracle.codes(r, alphabet), oracle.codes(q, alphabet)) for r, q in zip(refs, queries)]
    size, table = len(alphabet), _table(scoring)
    for counts in ((BIG, BIG, 0, 0), (0, BIG, 0, 0), (BIG, 0, 0, 0), (0, 0, BIG, BIG), (9, 20, 0, 4)):
        mode = da.Mode.ends_free(*counts)
        found = da.alignments(refs, queries, scoring, mode)
        expected = [oracle.free_ends_alignment(a, b, table, size, op, ex, *counts) for a, b in coded]
        assert [(a.score, a.cigar, _span(a)) for a in found] == expected
        assert da.scores(refs, queries, scoring, mode) == [score for score, _c, _s in expected]
    for anchor in (da.Anchor.START, da.Anchor.END):
        for zdrop, bonus in ((-1, -1), (25, 8), (0, -1)):
            found = da.alignments(refs, queries, scoring, da.Mode.extension(0, anchor, zdrop=zdrop, end_bonus=bonus))
            expected = [oracle.extension_alignment(a, b, table, size, op, ex, anchor == da.Anchor.END, bonus, zdrop=zdrop)
                        for a, b in coded]
            assert [(a.score, a.cigar, _span(a)) for a in found] == expected


def _tiled(da, refs, queries, times):
    """The pairs over and over as one tape."""
    once = da.Tape.of(refs, queries)
    letters = int(once.offsets[-1])
    starts = (np.arange(times)[:, None] * letters + once.offsets[None, :-1]).reshape(-1)
    return da.Tape(np.tile(once.letters[:letters], times), np.append(starts, times * letters))


def _assert_tiled(da, tape, scoring, mode, expected, times):
    scores, spans, offsets, data, statuses = da.alignments_tape(tape, scoring, mode)
    assert not statuses.any()
    np.testing.assert_array_equal(scores, np.tile([score for score, _c, _s in expected], times))
    np.testing.assert_array_equal(spans, np.tile([span for _s, _c, span in expected], (times, 1)))
    np.testing.assert_array_equal(np.diff(offsets), np.tile([len(cigar) for _s, cigar, _p in expected], times))
    assert data.tobytes() == "".join(cigar for _s, cigar, _p in expected).encode() * times


def test_placed_alignments_in_several_units(da, oracle):
    """140,000 pairs take four units on four lanes, which share the spans' tape, shapes and scores."""
    rng = np.random.default_rng(140)
    scoring = da.Scoring.uniform(2, -4, -4, -2)
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    refs, queries = [], []
    for k in range(1400):
        source = _text(rng, 1 + k % 40)
        refs.append(_text(rng, k % 17) + source + _text(rng, k % 13))
        queries.append(_mutated(rng, source, 0.1, "ACGT") if k % 50 else "")
    coded = [(oracle.codes(r), oracle.codes(q)) for r, q in zip(refs, queries)]
    tape = _tiled(da, refs, queries, 100)
    expected = [oracle.free_ends_alignment(a, b, _table(scoring), 4, op, ex, BIG, BIG, 0, 0) for a, b in coded]
    _assert_tiled(da, tape, scoring, da.Mode.INFIX, expected, 100)
    for from_end in (False, True):
        mode = da.Mode.extension(0, da.Anchor.END if from_end else da.Anchor.START, zdrop=12, end_bonus=4)
        expected = [oracle.extension_alignment(a, b, _table(scoring), 4, op, ex, from_end, 4, zdrop=12)
                    for a, b in coded]
        _assert_tiled(da, tape, scoring, mode, expected, 100)


# 5 letters and 20; 26 and 27, either side of the fewer columns; pairs of each up to those columns, at and past them.
@pytest.mark.parametrize("size", [5, 20, 26, 27])
def test_free_ends_through_profiles(da, oracle, size):
    """Larger alphabets' free ends in batches that fill the GPU, in 16 bits up to the columns that their profiles pay for,
    the same pairs in a batch that does not, in 32 bits."""
    alphabet = THIRTY_TWO[:size]
    rng = np.random.default_rng(size)
    scoring = _tabulated(da, rng, alphabet)
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    refs, queries = _placed_pairs(rng, alphabet)
    for width in (255, 256, 257, 393, 394, 512, 513):
        source = _text(rng, width, alphabet)
        refs.append(_text(rng, 30, alphabet) + source + _text(rng, 20, alphabet))
        queries.append(source)
    coded = [(oracle.codes(r, alphabet), oracle.codes(q, alphabet)) for r, q in zip(refs, queries)]
    tape = _tiled(da, refs, queries, 20)
    for counts in ((BIG, BIG, 0, 0), (0, 0, BIG, BIG), (9, 20, 0, 4)):
        mode = da.Mode.ends_free(*counts)
        expected = [oracle.free_ends_alignment(a, b, _table(scoring), size, op, ex, *counts) for a, b in coded]
        _assert_tiled(da, tape, scoring, mode, expected, 20)
        _assert_tiled(da, _tiled(da, refs, queries, 1), scoring, mode, expected, 1)


@pytest.mark.parametrize("mode_name", ["INFIX", "GLOBAL"])
def test_alignments_without_spans(da, mode_name):
    """A caller that wants no spans gives none: the scores and CIGARs are those with them."""
    rng = np.random.default_rng(8)
    refs = [_text(rng, 60) for _ in range(20)]
    queries = [_mutated(rng, ref[10:50], 0.1, "ACGT") for ref in refs]
    mode = getattr(da.Mode, mode_name)
    tape = da.Tape.of(refs, queries)
    native, lib = da._native, da._native.lib()
    scoring, _table_kept, _alphabet_kept = da.Scoring.dna()._struct()
    mode_struct = mode._struct()
    scores, offsets, statuses = np.empty(20, np.int32), np.empty(21, np.int64), np.empty(20, np.int64)
    buffer = ctypes.c_void_p()
    handle = native.context(0)
    native.check(lib.dinara_gpu_alignments_tape(
        handle, 20, tape.letters.ctypes.data, native.pointer(tape.offsets, ctypes.c_int64), ctypes.byref(scoring),
        ctypes.byref(mode_struct), 1, native.pointer(scores, ctypes.c_int32), None,
        native.pointer(offsets, ctypes.c_int64), ctypes.byref(buffer), native.pointer(statuses, ctypes.c_int64)), handle)
    data = ctypes.string_at(buffer.value, int(offsets[20]))
    lib.dinara_free(buffer.value)
    expected = da.alignments(refs, queries, da.Scoring.dna(), mode)
    assert list(scores) == [a.score for a in expected]
    assert [data[offsets[p]:offsets[p + 1]].decode() for p in range(20)] == [a.cigar for a in expected]


def _check_spans_past_their_pairs_band(da, oracle):
    """2,400 overlaps of 4,000 x 4,000 letters, which as global pairs would keep a band of 64 diagonals, and whose spans
    of 3,800 x 3,900 do not: their recorded decisions take 18.7 GB, in parts of 8 GiB. Prints the device memory that
    the call leaves taken."""
    import torch

    rng = np.random.default_rng(24)
    scoring = da.Scoring.uniform(2, -4, -4, -2)
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    refs, queries = [], []
    for _ in range(8):
        core = _text(rng, 3800)
        refs.append(_text(rng, 200) + core)
        queries.append((_mutated(rng, core[:1900], 0.02, "ACGT") + _text(rng, 100) +
                        _mutated(rng, core[1900:], 0.02, "ACGT") + _text(rng, 200))[:4000])
    mode = da.Mode.ends_free(reference_start=BIG, query_end=BIG)
    da.alignments(refs[:1], queries[:1], scoring, mode)
    before = torch.cuda.mem_get_info()[0]
    expected = [oracle.free_ends_alignment(oracle.codes(r), oracle.codes(q), _table(scoring), 4, op, ex, BIG, 0, 0, BIG)
                for r, q in zip(refs, queries)]
    assert all(abs((s[1] - s[0]) - (s[3] - s[2])) >= 64 for _s, _c, s in expected)
    _assert_tiled(da, _tiled(da, refs, queries, 300), scoring, mode, expected, 300)
    print("bytes", before - torch.cuda.mem_get_info()[0])


def test_spans_past_their_pairs_band(da):
    """In a process of its own, whose memory no earlier call has taken: 8 GiB of decisions and a quarter (what a buffer
    grows by), and 2 GB for the rest of the call."""
    run = subprocess.run([sys.executable, os.path.abspath(__file__), "spans"], capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0, run.stdout[-2000:] + run.stderr[-2000:]
    assert int(run.stdout.split("bytes")[1]) < 1.25 * 2 ** 33 + 2e9, run.stdout


# ---- larger alphabets through profiles --------------------------------------------------------------------

@pytest.mark.parametrize("alphabet", ["ACGTN", PROTEIN, THIRTY_TWO])
def test_profiles_score_globally_and_locally(da, oracle, alphabet):
    rng = np.random.default_rng(7 * len(alphabet))
    refs, queries = _placed_pairs(rng, alphabet)
    refs += ["", alphabet[:3]]
    queries += [alphabet[:2], ""]
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text, alphabet) for pair in zip(refs, queries) for text in pair if text])
    # The second table's entries do not fit a byte once shifted: the 32-bit form.
    for scoring in (_tabulated(da, rng, alphabet), _tabulated(da, rng, alphabet, -70, -66)):
        op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
        for mode, how in ((da.Mode.GLOBAL, oracle.GLOBAL), (da.Mode.local(), oracle.LOCAL)):
            expected = oracle.batch_scores(coded, tape.offsets, _table(scoring), len(alphabet), op, ex, how, threads=8)
            np.testing.assert_array_equal(da.scores_tape(tape, scoring, mode), expected)


def _check_alphabet(da, oracle, size):
    """Every profile sweep at `size` letters: scores, hits and recorded alignments, globally and locally, free ends
    and an extension, in every lane group, globally in a batch large enough for the 16-bit recording."""
    alphabet = THIRTY_TWO[:size]
    rng = np.random.default_rng(size)
    scoring = _tabulated(da, rng, alphabet)
    op, ex = oracle.kernel_gaps(scoring.opening, scoring.extension)
    refs, queries = [], []
    for k in range(4800):
        source = _text(rng, (60, 120, 250, 300, 500)[k] if k < 5 else 5 + k % 9, alphabet)
        refs.append(_text(rng, k % 4, alphabet) + source)
        queries.append(_mutated(rng, source, 0.1, alphabet) or alphabet[0])
    tape = da.Tape.of(refs, queries)
    coded = np.concatenate([oracle.codes(text, alphabet) for pair in zip(refs, queries) for text in pair])
    for mode, how in ((da.Mode.local(), oracle.LOCAL), (da.Mode.GLOBAL, oracle.GLOBAL)):
        expected, cigars = oracle.batch_alignments(coded, tape.offsets, _table(scoring), size, op, ex, how, threads=8)
        np.testing.assert_array_equal(da.scores_tape(tape, scoring, mode), expected)
        found = da.alignments(refs, queries, scoring, mode)
        assert [(a.score, a.cigar) for a in found] == list(zip(expected, cigars))
    coded = [(oracle.codes(r, alphabet), oracle.codes(q, alphabet)) for r, q in zip(refs, queries)]
    found = da.alignments(refs, queries, scoring, da.Mode.INFIX)
    assert [(a.score, a.cigar, _span(a)) for a in found] == [
        oracle.free_ends_alignment(a, b, _table(scoring), size, op, ex, BIG, BIG, 0, 0) for a, b in coded]
    found = da.alignments(refs[:40], queries[:40], scoring, da.Mode.extension(0, da.Anchor.START, zdrop=25))
    assert [(a.score, a.cigar, _span(a)) for a in found] == [
        oracle.extension_alignment(a, b, _table(scoring), size, op, ex, False, -1, zdrop=25) for a, b in coded[:40]]


def test_alphabets_in_rising_order():
    """A profile's bytes grow with the alphabet, past 48 KB from 24 letters on with the block's table. In a process of
    its own: a larger alphabet's launch leaves its allowance with the kernel."""
    run = subprocess.run([sys.executable, os.path.abspath(__file__), "23", "24", "25", "32"], capture_output=True,
                         text=True, timeout=300)
    assert run.returncode == 0, run.stdout[-2000:] + run.stderr[-2000:]


def test_two_contexts_with_alphabets_apart(da):
    """A kernel's shared-memory allowance is the process's: contexts on threads of their own, one at 25 letters and one
    at 32, launch side by side. (One launch in some thousands was refused when each asked for its own size.)"""
    lib, native = da._native.lib(), da._native
    failures = []

    def score(size):
        context = lib.dinara_gpu_new(0)
        rng = np.random.default_rng(size)
        alphabet = THIRTY_TWO[:size]
        tape = da.Tape.of([_text(rng, 200, alphabet)] * 8, [_text(rng, 200, alphabet)] * 8)
        scoring, _table_kept, _alphabet_kept = da.Scoring.uniform(5, -2, -10, -1, alphabet)._struct()
        mode = da.Mode.local()._struct()
        scores, statuses = np.empty(8, np.int32), np.empty(8, np.int64)
        for _ in range(15_000):
            code = lib.dinara_gpu_scores_tape(context, 8, tape.letters.ctypes.data,
                                              native.pointer(tape.offsets, ctypes.c_int64), ctypes.byref(scoring),
                                              ctypes.byref(mode), native.pointer(scores, ctypes.c_int32),
                                              native.pointer(statuses, ctypes.c_int64))
            if code:
                failures.append((size, code, lib.dinara_gpu_last_error(context)))
                break
        lib.dinara_gpu_free(context)

    threads = [threading.Thread(target=score, args=(size,)) for size in (25, 32)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not failures, failures


# ---- alignments under Costs: kept fronts in 16 bits, in 32 and in the shared blocks ---------------------------

@pytest.mark.parametrize("letters", [31_998, 32_002])
def test_fronts_either_side_of_16_bits(da, oracle, letters):
    """A pair whose two sides hold 32,000 letters at most keeps 16-bit fronts, a longer one 32-bit: few edits, runs of
    one letter at both ends (slides that meet the sequences' ends), both tie rules."""
    rng = np.random.default_rng(letters)
    half = letters // 2
    source = "A" * 40 + _text(rng, half - 80) + "C" * 40
    query = list(source)
    for place in (3, half // 3, half // 2, half - 4):
        query[place] = "G" if query[place] != "G" else "T"
    refs, queries = [source, "ACGT" * 3], ["".join(query), "ACGT" * 2]
    for costs, fields in ((da.Costs.affine(4, 6, 2), (4, 6, 2)), (da.Costs(), None)):
        for ties in ("left", "right"):
            found = da.alignments(refs, queries, costs, ties=ties)
            for a, r, q in zip(found, refs, queries):
                expected = (oracle.edit_cigar(r, q, right=ties == "right") if fields is None else
                            oracle.affine_cigar(r, q, *fields, right=ties == "right"))
                assert (a.cost, a.cigar) == expected


def test_fronts_in_shared_blocks(da, oracle):
    """Pairs whose fronts pass a warp's own arena, more of them than run at once without the shared blocks, among
    short ones."""
    rng = np.random.default_rng(41)
    refs, queries = [], []
    for trial in range(150):
        source = _text(rng, 1500 if trial % 3 == 0 else 60)
        refs.append(source)
        queries.append(_mutated(rng, source, 0.14, "ACGT"))
    found = da.alignments(refs, queries, da.Costs.affine(4, 6, 2))
    assert [(a.cost, a.cigar) for a in found] == [oracle.affine_cigar(r, q, 4, 6, 2) for r, q in zip(refs, queries)]


@pytest.mark.parametrize("pairs", [1, 32, 40])
def test_fronts_past_their_first_room(da, oracle, pairs):
    """A few dear pairs, which have the room that the longest could need at once, and more than a few, which run again in
    rooms of up to 8 MB and of 64 MB: unrelated pairs of 1,400 letters, some of 1,000 at 40% errors, a short one."""
    rng = np.random.default_rng(pairs)
    refs, queries = [], []
    for k in range(pairs):
        refs.append(_text(rng, 1400 if k % 4 == 0 else 1000 if k % 4 < 3 else 50))
        queries.append(_text(rng, 1380) if k % 4 == 0 else _mutated(rng, refs[-1], 0.4, "ACGT"))
    found = da.alignments(refs, queries, da.Costs.affine(4, 6, 2))
    assert [(a.cost, a.cigar) for a in found] == [oracle.affine_cigar(r, q, 4, 6, 2) for r, q in zip(refs, queries)]


# ---- unit-cost distances: the first round's list ---------------------------------------------------------------

@pytest.mark.parametrize("pairs", [1, 2, 33, 400])
def test_distances_beside_pairs_that_take_no_round(da, oracle, pairs):
    """Refused pairs, empty sides and letters other than DNA among pairs of up to three rounds: patterns at words
    and a letter either side."""
    rng = np.random.default_rng(pairs)
    refs, queries = [], []
    for k in range(pairs):
        length = int(rng.choice([1, 3, 63, 64, 65, 127, 128, 129, 700, 3000]))
        ref = _text(rng, length, "ACGT" if k % 4 else "ACGTNRY")
        refs.append(ref)
        queries.append(_text(rng, length) if k % 5 == 3 else _mutated(rng, ref, 0.1, "ACGT"))
    refs = [r.encode() for r in refs]
    queries = [q.encode() for q in queries]
    for k in range(0, pairs, 7):
        queries[k] = b"" if k % 2 else queries[k] + b"\xfe"
    tape = da.Tape.of(refs, queries)
    found, report = da.distances_tape(tape, report=True)
    np.testing.assert_array_equal(found, da.distances_tape(tape))
    for k in range(pairs):
        if queries[k].endswith(b"\xfe"):
            assert found[k] == da._native.UNSUPPORTED_SYMBOLS
        else:
            assert found[k] == oracle.edit_distance_dp(refs[k], queries[k])
    swept = sum(1 for r, q in zip(refs, queries) if r and q and not q.endswith(b"\xfe"))
    assert (report["round_pairs"][0] if report["round_pairs"] else 0) == swept


# ---- the predictor's gradients: the batch's slices -----------------------------------------------------------------

@pytest.mark.parametrize("batch", [1, 31, 128, 129, 4096, 4097])
def test_gradients_at_slice_edges(da, batch):
    """Against 64 bits: an fp32 sum of `batch` products in slices of 128 and then 32 is off by some sqrt(160) * 2^-24 of
    its terms' root of squares, 8e-7, where roundings are as likely up as down. Six seeds a batch: at most 3e-7 of the
    largest gradient from 31 samples on, 8e-7 at one, whose residual cancels."""
    import mlp_oracle
    from dinara_align import learned

    rng = np.random.default_rng(batch)
    flat = rng.normal(0, 0.1, size=learned.PARAMETERS).astype(np.float32)
    x = rng.normal(0, 0.5, size=(batch, learned.INPUTS)).astype(np.float32)
    t = rng.uniform(0, 0.2, size=batch).astype(np.float32)
    # A sample with a unit within fp32's rounding of its bend may pass on either side of it: drawn anew.
    while True:
        _y, (_x, first, _h1, second, _h2) = mlp_oracle.forward(mlp_oracle.unpack(flat), x.astype(np.float64))
        bent = np.minimum(np.abs(first).min(axis=1), np.abs(second).min(axis=1)) < 5e-6
        if not bent.any():
            break
        x[bent] = rng.normal(0, 0.5, size=(int(bent.sum()), learned.INPUTS))
    predictor = learned.Predictor()
    predictor.install(flat, 1.0, 0.0)
    got, loss = predictor.gradients(x, t)
    expected, expected_loss = mlp_oracle.gradients(*(v.astype(np.float64) for v in (flat, x, t)))
    np.testing.assert_allclose(got, expected, rtol=0, atol=(1e-6 if batch >= 31 else 4e-6) * np.abs(expected).max())
    assert abs(loss - expected_loss) <= 1e-5 * expected_loss


if __name__ == "__main__":
    # What needs a process of its own: the spans past their pairs' band, or alphabets in turn.
    import conftest  # noqa: F401
    import dinara_align
    import oracle as cpu

    if sys.argv[1] == "spans":
        _check_spans_past_their_pairs_band(dinara_align, cpu)
    else:
        for letters in sys.argv[1:]:
            _check_alphabet(dinara_align, cpu, int(letters))
