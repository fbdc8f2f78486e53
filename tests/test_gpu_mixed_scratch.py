"""The mixed kernel's scratch: a warp's own for groups, and slots for pairs per
thread that warps take as they come.  Batches that use both, under budgets
that leave one block, a few warps and slots, or all; every record and
CIGAR equals that of the same pairs by the one-pair kernel."""
import numpy as np
import pytest
import torch

from esperanto_gb300 import batch as B
from esperanto_gb300.extend import ExtendBuffer, ExtendParams
import workloads as W

pytestmark = pytest.mark.gpu


def _run(pairs, arena, mode, buf):
    out, cig = B.extend_batch_host(pairs, arena, params=ExtendParams(), mode=mode, cigar_stride=32, buf=buf)
    used = np.arange(32) < np.where(out["status"] == 0, out["n_ops"], 0)[:, None]
    return out, np.where(used, cig, 0)


@pytest.mark.parametrize("mode", [B.MODE_BAND, B.MODE_HINT])
@pytest.mark.parametrize("budget", [1 << 20, 40 << 20, 300 << 20, 8 << 30])
def test_budgets(budget, mode, monkeypatch):
    arena, pairs = W.synth_gotoh(2, 60000, 2)  # mixed lengths: costly pairs in groups
    one = ExtendBuffer()
    one.set_kernel_variant(1)
    want = _run(pairs, arena, mode, one)
    monkeypatch.setenv("ESP_SCRATCH_BUDGET", str(budget))
    got = _run(pairs, arena, mode, ExtendBuffer())
    assert (got[0] == want[0]).all() and (got[1] == want[1]).all()


def test_scratch_of_a_middling_batch():
    """65,536 extend_hint pairs of 150 x 214: 1.04 MB a warp with two pairs a
    lane (19 strips x 214 columns x 64 words), 0.28 MB with groups of 4.  1,152
    slots of the first kind (32 items a warp, an eighth more for lone pairs)
    and groups in all 2,432 resident warps: 1.9 GB; 2.5 GB if every warp had the
    first."""
    arena, pairs = W.synth_gotoh(1, 65536, 0)
    buf = ExtendBuffer()
    free = torch.cuda.mem_get_info()[0]
    _run(pairs, arena, B.MODE_HINT, buf)
    assert free - torch.cuda.mem_get_info()[0] < 2 << 30
