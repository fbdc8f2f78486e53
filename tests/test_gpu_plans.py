"""The plans of a batch below 2^18 pairs (bins.cu): groups of few and many
lanes, two pairs per thread and one, by size and shape -- short reads, narrow and
wide bands, whole windows, reads that differ in length -- on both sides of each
line.  Every record, touch and CIGAR equals that of the same pairs by the one-pair
kernel, and a sample of them the oracle's."""
import random

import numpy as np
import pytest

import oracle as O
from esperanto_gb300 import batch as B
from esperanto_gb300.extend import ExtendBuffer, ExtendParams

pytestmark = pytest.mark.gpu


def _pairs(rng, n, lo, hi, half):
    """n pairs over 60 distinct ones of reads cut from their windows."""
    reads, wins, offs, halves = [], [], [], []
    for _ in range(60):
        m = rng.randint(lo, hi)
        flank = half if half >= 0 else 20
        win = bytes(rng.choice(b"ACGT") for _ in range(m + 2 * flank))
        reads.append(bytes(rng.choice(b"ACGT") if rng.random() < .03 else b for b in win[flank:flank + m]))
        wins.append(win)
        offs.append(flank if half >= 0 else 0)
        halves.append(half)
    arena, pairs, iv = B.pack_ascii_pairs(reads, wins, offs, halves)
    return np.tile(pairs, n // 60 + 1)[:n], arena, list(zip(reads, wins, offs, halves))


def _run(pairs, arena, mode, variant):
    buf = ExtendBuffer()
    if variant is not None:
        buf.set_kernel_variant(variant)
    out, cig = B.extend_batch_host(pairs, arena, params=ExtendParams(), mode=mode, cigar_stride=48, buf=buf)
    used = np.arange(48) < np.where(out["status"] == 0, out["n_ops"], 0)[:, None]
    return out, np.where(used, cig, 0)


@pytest.mark.parametrize("mode", [B.MODE_BAND, B.MODE_HINT])
@pytest.mark.parametrize("lo,hi,half", [(16, 16, 10), (30, 32, 20), (50, 50, 16), (100, 130, 16),
                                        (128, 128, 32), (129, 150, 32), (100, 100, 64), (150, 150, 64),
                                        (64, 64, -1), (50, 150, 16)])
def test_plans(lo, hi, half, mode):
    rng = random.Random(lo * 1000 + hi)
    for n in (2049, 4900, 7000, 12000, 19457, 26000, 38912, 38913, 41000, 47000):
        pairs, arena, cases = _pairs(rng, n, lo, hi, half)
        got, want = _run(pairs, arena, mode, None), _run(pairs, arena, mode, 1)
        assert (got[0] == want[0]).all() and (got[1] == want[1]).all(), n
        for k in range(0, 60, 7):
            read, win, off, h = cases[k]
            if mode == B.MODE_HINT:
                key = O.extend_hint(read, win, O.Params(), offset=off).key()
            else:
                key = O.run_dispatch(read, win, O.Params(), band=(off, h) if h >= 0 else None)[0].key()
            o = got[0][k]
            assert key == (int(o["score"]), int(o["read_start"]), int(o["read_end"]), int(o["ref_start"]),
                           tuple(B.cigar_of(got[1][k], int(o["n_ops"])))), (n, k)
