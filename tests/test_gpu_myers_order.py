"""The Myers kernel where its launch and its loops branch (myers.cu): batches
in their own order and (from 256 pairs an SM on) ordered by limb count within a
block, the last block whole or short; reads of every limb count with one row to either side, empty reads
among them; texts of every length modulo 16, empty, shorter than 16, and with N
runs in partial and full chunks.  Every distance and position equals the
oracle's."""
import random

import numpy as np
import pytest

import oracle as O
from esperanto_gb300 import batch as B

pytestmark = pytest.mark.gpu


def _pairs(rng, count):
    reads, texts = [], []
    for k in range(count):
        m = rng.choice([1, 31, 32, 33, 64, 65, 95, 96, 97, 128, 129, 160, 161, 192, 193, 224, 225, 256])
        n = rng.choice([0, 3, 15, 16, 17, 48, m + k % 16, m + 50 + k % 16])
        text = bytearray(rng.choice(b"ACGT") for _ in range(n))
        at = rng.randrange(0, max(1, n - m))
        read = bytes(text[at + i] if at + i < n and rng.random() > .05 else rng.choice(b"ACGTN")
                     for i in range(m))
        if k % 4 == 0 and n:
            a = rng.randrange(n)
            for i in range(a, min(n, a + rng.choice([1, 2, 20]))):
                text[i] = ord("N")
        reads.append(read)
        texts.append(bytes(text))
    return reads, texts


@pytest.mark.parametrize("mode", [B.MYERS_BEST_END, B.MYERS_BEST_START, B.MYERS_GLOBAL])
@pytest.mark.parametrize("count", [1, 31, 33, 600, 10007, 40001, 90001])
def test_ordered_blocks(count, mode):
    rng = random.Random(count)
    base = min(count, 601)
    reads, texts = _pairs(rng, base)
    arena, pairs, iv = B.pack_ascii_myers(reads, texts)
    order = np.random.default_rng(count).integers(0, base, count)
    order[:base] = np.arange(base)
    got = B.myers_batch_host(pairs[order], arena, iv, mode)
    assert (got["status"] == 0).all()
    want = np.zeros((base, 2), np.int64)
    for k, (r, t) in enumerate(zip(reads, texts)):
        want[k] = (O.myers_long_infix_best_end(r, t) if mode == B.MYERS_BEST_END else
                   O.myers_long_infix_best_start(r, t) if mode == B.MYERS_BEST_START else
                   (O.engine_global(r, t), 0))
    assert (got["dist"] == want[order, 0]).all() and (got["pos"] == want[order, 1]).all()
