"""Plans of batches of unlike pairs (bins.cu, abi.cu) where the lanes that a read's
strips or its band keep busy differ from those its share of the batch asks for:
short reads in wide bands, reads of many lengths in narrow ones, and reads just under
and over 0.8 of the costliest.  Equal to the one-pair kernel's results and, for a
sample, the oracle's."""
import random

import pytest

import oracle as O
from esperanto_gb300 import batch as B
from test_gpu_plans import _pairs, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [B.MODE_BAND, B.MODE_HINT])
@pytest.mark.parametrize("n,lo,hi,half", [(5541, 86, 86, 128), (7441, 52, 253, 16), (2049, 52, 253, 16),
                                          (42555, 112, 155, -1), (30001, 120, 150, 32), (30001, 110, 150, 32)])
def test_unlike_shapes(n, lo, hi, half, mode):
    pairs, arena, cases = _pairs(random.Random(n + lo), n, lo, hi, half)
    got, want = _run(pairs, arena, mode, None), _run(pairs, arena, mode, 1)
    assert (got[0] == want[0]).all() and (got[1] == want[1]).all()
    for k in range(0, 60, 11):
        read, win, off, h = cases[k]
        key = (O.extend_hint(read, win, O.Params(), offset=off) if mode == B.MODE_HINT
               else O.run_dispatch(read, win, O.Params(), band=(off, h) if h >= 0 else None)[0]).key()
        o = got[0][k]
        assert key == (int(o["score"]), int(o["read_start"]), int(o["read_end"]), int(o["ref_start"]),
                       tuple(B.cigar_of(got[1][k], int(o["n_ops"]))))
