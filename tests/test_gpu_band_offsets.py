"""Band offsets of a batch: every 32-bit value is a band (one far outside the
window keeps each row's centre on column 1 or n), in every DP kernel.  Results
and touches equal the oracle's, which computes in 64 bits."""
import random

import pytest

from gpu_helpers import _compare
from esperanto_gb300 import batch as B

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
