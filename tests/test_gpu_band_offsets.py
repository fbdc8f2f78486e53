"""Band offsets of a batch: every 32-bit value is a band (one far outside the
window keeps each row's centre on column 1 or n), in every DP kernel.  Results
and touches equal the oracle's, which computes in 64 bits."""
import random

import numpy as np
import pytest

from gpu_helpers import _compare
from esperanto_gb300 import batch as B
from esperanto_gb300.extend import ExtendBuffer, ExtendParams
import workloads as W

pytestmark = pytest.mark.gpu

FAR = [-2**31, -2**31 + 1, -2**31 + 40, -2**31 + 5000, 2**31 - 1, 2**31 - 40, 2**31 - 33000,
       -70000, 70000, -32800, 32800]


@pytest.mark.parametrize("mode", [B.MODE_BAND, B.MODE_HINT])
@pytest.mark.parametrize("kernel", ["warp", "thread", "paired"])
def test_far_offsets(kernel, mode):
    rng = random.Random(4)
    cases = []
    for m, n, half in ((40, 72, 16), (70, 134, 32), (150, 214, 32), (9, 30, 3), (60, 61, 0)):
        for off in FAR:
            win = bytes(rng.choice(b"ACGT") for _ in range(n))
            read = bytes(rng.choice(b"ACGT") if rng.random() < .03 else b for b in win[-m:])
            cases += [(read, win, (off, half))] * 2
    _compare(cases, [1] * len(cases), mode, None, kernel)


def _by(pairs, arena, mode, variant):
    buf = ExtendBuffer()
    if variant is not None:
        buf.set_kernel_variant(variant)
    out, cig = B.extend_batch_host(pairs, arena, params=ExtendParams(), mode=mode, cigar_stride=32, buf=buf)
    used = np.arange(32) < np.where(out["status"] == 0, out["n_ops"], 0)[:, None]
    return out, np.where(used, cig, 0)


@pytest.mark.parametrize("mode", [B.MODE_BAND, B.MODE_HINT])
@pytest.mark.parametrize("n", [2500, 16384, 47000, 262144, 300001])
@pytest.mark.parametrize("shape", [0, 2])
def test_offsets_that_differ(shape, n, mode):
    """Pairs of one size at several offsets, which cannot share a thread: none,
    a few (below and above the share at which a batch runs one pair per
    thread), all; some without a band among them.  Every record and CIGAR
    equals that of the same pairs by the one-pair kernel."""
    arena, base = W.synth_gotoh(9, n, shape)
    rng = np.random.default_rng(n + shape)
    for share in (0.0005, 0.02, 1.0):
        pairs = base.copy()
        moved = rng.random(n) < share
        pairs["band_offset"][moved] += rng.integers(-12, 13, moved.sum()).astype(np.int32)
        pairs["band_half"][moved & (rng.random(n) < .01)] = -1
        got, want = _by(pairs, arena, mode, None), _by(pairs, arena, mode, 1)
        assert (got[0] == want[0]).all() and (got[1] == want[1]).all(), share
