"""A lightly loaded server cuts its waves' items into pieces for idle blocks; a
bound on the items in flight turns that off.  Results, probes' errors included,
are the same to the last bit."""
import numpy as np
import pytest

from test_gpu_serve import req

pytestmark = pytest.mark.gpu

MIX = [req(2.0, 20.0, 101, 0.02, base=1 << 32), req(10.0, 1.0, 101, 0.03, base=2 << 32),
       req(0.05, 300.0, 33, 0.2, cap=1 << 13, base=3 << 32), req(1.0, 300.0, 501, 0.05, base=4 << 32),
       req(0.2, 900.0, 1, 0.3, cap=1 << 12, base=5 << 32)]


@pytest.mark.parametrize("stream", [0, 1])
@pytest.mark.parametrize("some", [1, 2, 5])
def test_pieces_change_nothing(tmc_mod, some, stream):
    from tiny_mc_gb300.serve import Server
    got = []
    for bound in (0, 100000):
        s = Server(slots=8, stream=stream, inflight_items=bound)
        ids = {s.submit(r): int(r["shells"]) for r in MIX[-some:]}
        out = s.run(ids)
        s.close()
        got.append([out[i] for i in ids])
    for (t0, r0), (t1, r1) in zip(*got):
        assert np.array_equal(t0, t1)
        for f in ("photons", "photon_steps", "batches", "batch_photons", "reached_target", "rse"):
            assert r0[f] == r1[f], f
