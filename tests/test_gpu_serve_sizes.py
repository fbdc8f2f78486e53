"""A server whose launches may hold more reads than the mixed kernel takes
(2^18): requests of sizes that choose each kernel, submitted by several threads
at once, while launches run.  Every result equals the same request served
alone by a server of small launches."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from esperanto_gb300 import serve as SV  # noqa: E402
from esperanto_gb300.split import Genome  # noqa: E402
import workloads as W  # noqa: E402


def _same(a, b):
    assert (a.out == b.out).all()
    used = np.arange(a.stride) < a.out["n_ops"][:, None]
    shape = (len(a.reads), a.stride)
    assert (a.cigar.reshape(shape)[used] == b.cigar.reshape(shape)[used]).all()


def test_large_launches_from_several_threads():
    garena, contigs = W.synth_genome(5, 2_000_000, 2)
    g = Genome(garena, contigs)
    sizes = [300, 1500, 2500, 6000, 15000, 40000, 70000, 263000]
    reqs = [W.synth_request(5, 40 + k, garena, contigs, n) for k, n in enumerate(sizes)]
    one = SV.Server(g, n_streams=1, max_reads=2048, mem_budget=1 << 30)
    want = [one.submit(*r) for r in reqs]
    for t in want:
        assert one.wait(t)[0] == 0
    one.destroy()
    srv = SV.Server(g, n_streams=3, max_reads=270000, mem_budget=12 << 30)
    got, errors = [None] * len(reqs), []

    def client(k):
        try:
            for _ in range(3):
                got[k] = srv.submit(*reqs[k])
                assert srv.wait(got[k])[0] == 0
        except Exception as e:  # noqa: BLE001
            errors.append((k, e))

    threads = [threading.Thread(target=client, args=(k,)) for k in range(len(reqs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    srv.destroy()
    assert not errors, errors
    for a, b in zip(got, want):
        _same(a, b)
