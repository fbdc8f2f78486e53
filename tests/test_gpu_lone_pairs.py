"""The warp-per-pair kernel (gotoh.cu, warp_fill) where its wavefront changes:
reads of one strip, of 32 strips and one row to either side (a second pass of
the lanes begins), and of several passes; passes that the next one follows 32
steps behind, those just too wide for it, and full matrices, whose rows cross
passes through the row buffer; windows of one column and of odd widths (two
columns a step); bands that clamp at either end; N in read and window; touches
and extend_hint's second attempt.  Every record and CIGAR equals the oracle's."""
import random

import pytest

import oracle as O
from esperanto_gb300 import batch as B
from esperanto_gb300.extend import ExtendBuffer, ExtendParams

pytestmark = pytest.mark.gpu


def _cases(rng, m, widths, bands):
    for n in widths:
        win = bytearray(rng.choice(b"ACGT") for _ in range(n))
        for band in bands(m, n):
            at = (n - m) // 2 if rng.random() < .5 else rng.randrange(-20, 20)
            read = bytearray(win[at + k] if 0 <= at + k < n and rng.random() > .04
                             else rng.choice(b"ACGT") for k in range(m))
            if rng.random() < .2:
                win[rng.randrange(n)] = read[rng.randrange(m)] = ord("N")
            yield bytes(read), bytes(win), band


def _check(cases, params, mode):
    buf = ExtendBuffer()
    buf.set_warp_max(1 << 20)
    arena, pairs, iv = B.pack_ascii_pairs([c[0] for c in cases], [c[1] for c in cases],
                                          [c[2][0] if c[2] else 0 for c in cases],
                                          [c[2][1] if c[2] else -1 for c in cases])
    stride = max(2 * (len(c[0]) + len(c[1])) + 8 for c in cases)
    out, cig = B.extend_batch_host(pairs, arena, iv, params, mode, stride, buf=buf)
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


def _bands(m, n):
    yield None
    for half in (0, 7, 31, 151, 156, 157, 158, 159, 160, 200):
        yield (n - m) // 2, half
        yield 0, half
        yield -m // 2, half


@pytest.mark.parametrize("m", [1, 8, 9, 255, 256, 257, 264, 511, 513, 777])
def test_passes_of_the_wavefront(m):
    rng = random.Random(m)
    _check(list(_cases(rng, m, (1, 2, 63, 66, m + 64, m + 401), _bands)),
           ExtendParams(edit_dir=m % 3), B.MODE_BAND)


@pytest.mark.parametrize("m", [40, 150, 257, 600])
def test_hint_second_attempts(m):
    rng = random.Random(m)
    _check(list(_cases(rng, m, (29, m + 61, m + 64, m + 300),
                       lambda m, n: [(o, -1) for o in (0, 30, (n - m) // 2, -50, 100)])),
           ExtendParams(), B.MODE_HINT)
