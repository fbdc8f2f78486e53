"""Host batches of several chunks (esp_host.h, run_chunks): from page-locked
arrays, whose copies are all queued first, and from ordinary ones, whose chunks are
launched as they are sent.  Both equal the same pairs in a batch of one chunk, with
reads of no bases among the Myers pairs; and the DP batches on either side of the
size where two pairs share a thread."""
import random

import numpy as np
import pytest

import oracle as O
from esperanto_gb300 import batch as B
from esperanto_gb300.extend import ExtendBuffer, ExtendParams

pytestmark = pytest.mark.gpu

LARGE = 1 << 18  # pairs from which the paired kernel runs and host batches are chunked


def _locked(a):
    """A page-locked copy of the array and what keeps it alive."""
    import torch
    t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    t.numpy()[:] = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
    return t.numpy().view(a.dtype), t


def _seqs(rng, count, lens, flank):
    reads, wins = [], []
    for _ in range(count):
        m = rng.choice(lens)
        win = bytes(rng.choice(b"ACGT") for _ in range(m + 2 * flank))
        reads.append(bytes(rng.choice(b"ACGT") if rng.random() < .03 else b for b in win[flank:flank + m]))
        wins.append(win)
    return reads, wins


@pytest.mark.parametrize("mode", [B.MYERS_BEST_END, B.MYERS_BEST_START, B.MYERS_GLOBAL])
@pytest.mark.parametrize("count", [LARGE - 1, LARGE, LARGE + 70001])
def test_myers(count, mode):
    rng = random.Random(mode)
    empty = [] if mode == B.MYERS_GLOBAL else [0, 0]  # the oracle refuses those
    reads, texts = _seqs(rng, 301, empty + [1, 31, 32, 33, 64, 100, 150, 255, 256], 9)
    arena, pairs, iv = B.pack_ascii_myers(reads, texts)
    search = {B.MYERS_BEST_END: O.myers_long_infix_best_end, B.MYERS_BEST_START: O.myers_long_infix_best_start,
              B.MYERS_GLOBAL: lambda r, t: (O.engine_global(r, t), 0)}[mode]
    want = np.array([search(r, t) for r, t in zip(reads, texts)], np.int64)
    order = np.random.default_rng(count).integers(0, len(reads), count)
    batch, keep = _locked(pairs[order])
    bases, keep2 = _locked(arena)
    for p, a in ((batch, bases), (pairs[order], arena)):
        got = B.myers_batch_host(p, a, iv, mode)
        assert (got["status"] == 0).all()
        assert (got["dist"] == want[order, 0]).all() and (got["pos"] == want[order, 1]).all()


@pytest.mark.parametrize("mode", [B.MODE_BAND, B.MODE_HINT])
@pytest.mark.parametrize("count", [LARGE - 1, LARGE, LARGE + 70001])
def test_extend(count, mode):
    rng = random.Random(mode)
    reads, wins = _seqs(rng, 211, list(range(10, 48)), 8)
    arena, pairs, iv = B.pack_ascii_pairs(reads, wins, [8] * len(reads), [8] * len(reads))
    order = np.random.default_rng(count).integers(0, len(reads), count)

    def run(p, a):
        out, cig = B.extend_batch_host(p, a, iv, params=ExtendParams(), mode=mode, cigar_stride=24,
                                       buf=ExtendBuffer())
        return out, np.where(np.arange(24) < np.where(out["status"] == 0, out["n_ops"], 0)[:, None], cig, 0)

    one, one_cig = run(pairs, arena)
    for k in range(0, len(reads), 3):
        key = (O.extend_hint(reads[k], wins[k], O.Params(), offset=8) if mode == B.MODE_HINT
               else O.run_dispatch(reads[k], wins[k], O.Params(), band=(8, 8))[0]).key()
        o = one[k]
        assert o["status"] == 0
        assert key == (int(o["score"]), int(o["read_start"]), int(o["read_end"]), int(o["ref_start"]),
                       tuple(B.cigar_of(one_cig[k], int(o["n_ops"]))))
    batch, keep = _locked(pairs[order])
    bases, keep2 = _locked(arena)
    for p, a in ((batch, bases), (pairs[order], arena)):
        out, cig = run(p, a)
        assert (out == one[order]).all() and (cig == one_cig[order]).all()
