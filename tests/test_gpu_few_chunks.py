"""Batches with fewer chunks of work than a launch has warps: the blocks that
come after a chunk for every warp before them leave.  Sizes with as many chunks
as one, two or three blocks an SM have warps, one pair more and one fewer; pairs
that all keep extend_hint's first attempt (its second finds no work).  Every
record and CIGAR equals that of the same pairs by the one-pair kernel."""
import numpy as np
import pytest
import torch

from esperanto_gb300 import batch as B
from esperanto_gb300.extend import ExtendBuffer, ExtendParams
import workloads as W

pytestmark = pytest.mark.gpu

PER_BLOCK = 64 * 4  # pairs: two a lane, four warps


def _run(pairs, arena, mode, variant):
    buf = ExtendBuffer()
    buf.set_warp_max(0)
    if variant is not None:
        buf.set_kernel_variant(variant)
    out, cig = B.extend_batch_host(pairs, arena, params=ExtendParams(), mode=mode, cigar_stride=32, buf=buf)
    used = np.arange(32) < np.where(out["status"] == 0, out["n_ops"], 0)[:, None]
    return out, np.where(used, cig, 0)


@pytest.mark.parametrize("variant", [None, 3])
@pytest.mark.parametrize("kind", ["band", "hint", "hint_first"])
@pytest.mark.parametrize("blocks", [0, 1, 2, 3])
def test_leaving_blocks(blocks, kind, variant):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mode = B.MODE_BAND if kind == "band" else B.MODE_HINT
    for more in (-1, 0, 1):
        n = max(40, blocks * sms * PER_BLOCK + more)
        arena, pairs = W.synth_gotoh(7, n, 0)
        if kind == "hint_first":  # windows no wider than the first band: its result stands
            pairs["read_pos"], pairs["read_len"] = pairs["win_pos"] + 3, 24
            pairs["win_len"] = 30
        got, want = _run(pairs, arena, mode, variant), _run(pairs, arena, mode, 1)
        if kind == "hint_first":
            assert not got[0]["escalated"].any()
        assert (got[0] == want[0]).all() and (got[1] == want[1]).all(), n
