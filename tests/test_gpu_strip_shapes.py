"""The thread kernels at the strip shapes and key widths where their fills
branch (gotoh.cu): strips whose row windows slope on both sides, stand still
on one or both, or begin or end clamping inside the strip; reads of 8k - 1,
8k and 8k + 1 rows; bands narrower than a strip; row-maximum keys of one
column, and of blocks of columns (long reads on the paired kernel); best
columns that tie inside such a block; traceback walks whose matches run off
the left edge of a clamped band; gap costs of 0.  Pairs with a partner of
their geometry, without one, and with N in the window share every batch, so
that the paired kernel's ways of filling a pair run side by side.
Every record, touch and CIGAR equals the oracle's."""
import random

import numpy as np
import pytest

import oracle as O
from esperanto_gb300 import batch as B
from esperanto_gb300.extend import ExtendBuffer, ExtendParams

pytestmark = pytest.mark.gpu


def _seq(rng, n, letters=b"ACGT"):
    return bytes(rng.choice(letters) for _ in range(n))


def _read_of(rng, win, at, m):
    """m bases of the window from `at` on (random past its ends), 4 % changed."""
    out = bytearray()
    for k in range(m):
        b = win[at + k] if 0 <= at + k < len(win) else rng.choice(b"ACGT")
        out.append(rng.choice(b"ACGT") if rng.random() < .04 else b)
    return bytes(out)


def _bands(m, n):
    """Band offsets and halves that slope, stand still and change shape."""
    yield None
    for half in (0, 3, 7, 8, 16):
        flank = (n - m) // 2
        yield (flank, half)             # sloped all along when half <= flank
        yield (0, half)                 # left edge stands still, then slopes
        yield (n - m + half + 3, half)  # right edge slopes, then stands still
        yield (-m // 2, half)           # clamped at column 1 for half the rows
        yield (n, half)                 # clamped at column n throughout


def _batch(rng, shapes):
    cases = []
    for m, n, band in shapes:
        win = _seq(rng, n, rng.choice([b"ACGT", b"ACGT", b"AC", b"A"]))
        cases.append((_read_of(rng, win, (n - m) // 2, m), win, band))
        twin = bytes(rng.choice(b"ACGT") if rng.random() < .03 else b for b in win)
        cases.append((_read_of(rng, twin, band[0] if band else 3, m), twin, band))
        if rng.random() < .3:  # a window with N, and a lone geometry
            w = bytearray(win)
            w[rng.randrange(n)] = ord("N")
            cases.append((cases[-1][0], bytes(w), band))
            cases.append((_read_of(rng, win, 0, m) + b"A", win, band))
    rng.shuffle(cases)
    return cases


def _check(cases, params, variant, copies=1, mode=B.MODE_BAND):
    """variant None: what the batch's size selects; copies: the batch holds the
    cases so often."""
    buf = ExtendBuffer()
    buf.set_warp_max(0)
    if variant is not None:
        buf.set_kernel_variant(variant)
    arena, pairs, iv = B.pack_ascii_pairs([c[0] for c in cases], [c[1] for c in cases],
                                          [c[2][0] if c[2] else 0 for c in cases],
                                          [c[2][1] if c[2] else -1 for c in cases])
    stride = max(2 * (len(c[0]) + len(c[1])) + 8 for c in cases)
    n = len(cases)
    out, cig = B.extend_batch_host(np.tile(pairs, copies), arena, iv, params, mode, stride, buf=buf)
    op = O.Params(params.match_score, params.mismatch, params.gap_open, params.gap_ext,
                  edit_dir=int(params.edit_dir))
    for k, (read, win, band) in enumerate(cases):
        if mode == B.MODE_HINT:
            e, t = O.extend_hint(read, win, op, offset=band[0] if band else 0), None
        else:
            e, t = O.run_dispatch(read, win, op, band=band)
        o = out[k]
        got = (int(o["score"]), int(o["read_start"]), int(o["read_end"]), int(o["ref_start"]),
               tuple(B.cigar_of(cig[k], int(o["n_ops"]))))
        touch = O.Touch(bool(o["touched"]), int(o["touch_row"]), bool(o["touch_left"]),
                        bool(o["touch_clamped"]))
        assert int(o["status"]) == 0 and got == e.key(), (len(read), len(win), band)
        assert t is None or touch == t, (len(read), len(win), band)
        ops = int(o["n_ops"])
        for c in range(1, copies):
            assert out[k + c * n] == o and (cig[k + c * n][:ops] == cig[k][:ops]).all(), (k, c)


@pytest.mark.parametrize("variant", [0, 1, 2, 3, None])
@pytest.mark.parametrize("rows", [(1, 7, 8, 9), (15, 16, 17), (63, 64, 65)])
def test_strip_shapes(rows, variant):
    rng = random.Random(rows[0] * 10 + (variant or 0))
    shapes = [(m, m + 2 * f, b) for m in rows for f in (1, 8, 16) for b in _bands(m, m + 2 * f)]
    _check(_batch(rng, shapes), ExtendParams(edit_dir=(variant or 1) % 3), variant)


@pytest.mark.parametrize("params", [ExtendParams(2, -4, 0, 0), ExtendParams(1, 1, 2, 1),
                                    ExtendParams(5, -3, 400, 400), ExtendParams(0, -1, 1, 1),
                                    ExtendParams(2, 3, 4, 2), ExtendParams(31, -32, 1600, 400)])
def test_score_ranges(params):
    rng = random.Random(7)
    shapes = [(m, m + 24, b) for m in (9, 24, 40) for b in _bands(m, m + 24)]
    for variant in (1, 3, None):
        _check(_batch(rng, shapes), params, variant)


@pytest.mark.parametrize("m,band", [(300, (128, 128)), (1200, (40, 40)), (2500, (16, 16)),
                                    (4095, (8, 8)), (700, None)])
def test_row_maximum_blocks(m, band):
    """Reads whose row-maximum keys cover blocks of columns (two-letter
    sequences make equal row maxima common)."""
    rng = random.Random(m)
    flank = band[0] if band else 30
    cases = []
    for letters in (b"ACGT", b"AC"):
        win = _seq(rng, m + 2 * flank, letters)
        for _ in range(3):
            cases.append((_read_of(rng, win, flank, m), win, band))
    for variant in (3, None):
        _check(cases * 6, ExtendParams(), variant)


@pytest.mark.parametrize("mode", [B.MODE_BAND, B.MODE_HINT])
@pytest.mark.parametrize("copies", [12, 50, 130, 330, 800, 2200])
def test_groups_by_batch_size(copies, mode):
    """The mixed kernel's groups of 32, 16, 8 and 4 lanes, a batch whose costly
    pairs alone go to groups, and one that the paired kernel takes."""
    rng = random.Random(copies)
    shapes = [(m, m + 2 * f, b) for m in (9, 41) for f in (4, 10) for b in _bands(m, m + 2 * f)]
    shapes = rng.sample(shapes, 40) + [(150, 182, (16, 16)), (96, 352, (128, 128)), (70, 130, None)]
    _check(_batch(rng, shapes), ExtendParams(), None, copies, mode)
