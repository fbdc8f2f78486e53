"""The mixed kernel's scratch: warps that run pairs per thread own more of it
than those that run groups only.  Batches that use both kinds, under budgets
that leave one block, a few warps, or all of either kind; every record and
CIGAR equals that of the same pairs by the one-pair kernel."""
import numpy as np
import pytest

from esperanto_gb300 import batch as B
from esperanto_gb300 import serve as SV
from esperanto_gb300.extend import ExtendBuffer, ExtendParams
from esperanto_gb300.split import Genome
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


def test_serving_launch_takes_half_the_pool():
    """65,536 reads of at most 300 bases in windows of 428: 4.2 MB a warp with
    two pairs a lane (38 strips x 428 columns x 64 words), 10.1 GB if all 2,432
    resident warps had that.  The 1,152 that have such work (32 items each, an
    eighth more for lone pairs) are two of the four on every scheduler."""
    garena, contigs = W.synth_genome(5, 2_000_000, 2)
    g = Genome(garena, contigs)
    arena, reads = W.synth_request(5, 3, garena, contigs, 65536)
    reads = reads.copy()
    reads["read_len"][0] = 300
    reads["win_len"][0] = 428
    srv = SV.Server(g, n_streams=1, max_reads=65536, mem_budget=16 << 30)
    t = srv.submit(arena, reads)
    assert srv.wait(t)[0] == 0
    st = srv.stats()
    srv.destroy()
    assert st["launches"] == 1 and st["pool_peak_bytes"] < 8 << 30, st
