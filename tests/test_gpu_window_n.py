"""N in reads alone, in one window of a batch, and in neither: which fill a batch
takes depends on the windows.  Sizes of the mixed and the paired kernel, on a
default handle and one set to two pairs per thread.  Every record and CIGAR
equals that of the same pairs by the one-pair kernel, which tests each window."""
import numpy as np
import pytest

from esperanto_gb300 import batch as B
from esperanto_gb300.extend import ExtendBuffer, ExtendParams
import workloads as W

pytestmark = pytest.mark.gpu


def _run(pairs, arena, iv, mode, variant):
    buf = ExtendBuffer()
    if variant is not None:
        buf.set_kernel_variant(variant)
    out, cig = B.extend_batch_host(pairs, arena, iv, ExtendParams(), mode, 32, buf=buf)
    used = np.arange(32) < np.where(out["status"] == 0, out["n_ops"], 0)[:, None]
    return out, np.where(used, cig, 0)


@pytest.mark.parametrize("mode", [B.MODE_BAND, B.MODE_HINT])
@pytest.mark.parametrize("where", ["read", "window", "both"])
@pytest.mark.parametrize("n,variant", [(3000, None), (50000, None), (262144, None), (5000, 3)])
def test_where_n_lies(n, variant, where, mode):
    arena, pairs = W.synth_gotoh(6, n, 2)
    rng = np.random.default_rng(n)
    iv = []
    for k in rng.choice(n, 5 if where == "read" else 1, replace=False):
        pairs["n_first"][k] = len(iv)
        if where != "window":
            a = int(rng.integers(0, pairs["read_len"][k] - 3))
            iv.append((a, a + 3))
            pairs["n_read"][k] = 1
        if where != "read":
            a = int(pairs["win_len"][k]) // 2
            iv.append((a, a + 2))
            pairs["n_win"][k] = 1
    iv = np.array(iv, B.NIV_DTYPE)
    got, want = _run(pairs, arena, iv, mode, variant), _run(pairs, arena, iv, mode, 1)
    assert (got[0] == want[0]).all() and (got[1] == want[1]).all()
