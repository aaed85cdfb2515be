"""The room that a persistent server launch leaves for small kernels, for every
block size: the colour map and the FP64 report run beside it.  (A launch that
keeps them waiting gives up after 120 s, and the server ends with an error.)"""
import time

import numpy as np
import pytest

from test_gpu_serve import req

pytestmark = pytest.mark.gpu

LONG = (req(0.2, 90.0, 101, 1e-4, cap=1 << 16, base=1 << 32), req(2.0, 20.0, 501, 1e-4, cap=1 << 20, base=2 << 32))


def small_calls(tmc_mod, tally, p):
    from tiny_mc_gb300 import view
    heats = np.linspace(0.0, 1.0, 101, dtype=np.float32)
    return view.colormap(heats, 64, 64), tmc_mod.report_fp64(tally, p, 2000)


def same(a, b):
    return (all(np.array_equal(x, y) for x, y in zip(a[0], b[0])) and
            all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a[1][:2], b[1][:2])))


@pytest.mark.parametrize("max_shells", [501, 2000])
@pytest.mark.parametrize("math", [0, 1])
@pytest.mark.parametrize("stream", [0, 1])
@pytest.mark.parametrize("block", [128, 256, 512])
def test_small_calls_beside_any_block_size(tmc_mod, block, stream, math, max_shells):
    from tiny_mc_gb300.serve import Server
    p = tmc_mod.params(seed=1)
    tally, _ = tmc_mod.photon_batch_fx(2000, p)
    before = small_calls(tmc_mod, tally, p)              # loads the kernels
    s = Server(slots=8, persistent=1, block=block, stream=stream, math=math, max_shells=max_shells)
    ids = {s.submit(r): int(r["shells"]) for r in LONG}
    s.progress()
    t0 = time.monotonic()
    beside = small_calls(tmc_mod, tally, p)
    took = time.monotonic() - t0
    out = s.run(ids)
    s.close()
    assert took < 20.0
    assert same(before, beside)
    assert all(r["photons"] for _, r in out.values())


@pytest.mark.parametrize("stream", [0, 1])
@pytest.mark.parametrize("block", [128, 512])
def test_small_calls_beside_a_relaunch(tmc_mod, block, stream):
    """Requests that arrive right after the server has run dry (its blocks wait 20
    ms before they end): the next launch does not share the SMs with the last one."""
    from tiny_mc_gb300.serve import Server
    p = tmc_mod.params(seed=1)
    tally, _ = tmc_mod.photon_batch_fx(2000, p)
    before = small_calls(tmc_mod, tally, p)
    s = Server(slots=8, persistent=1, block=block, stream=stream)
    for k in range(3):
        short = req(2.0, 20.0, 101, 0.05, cap=1 << 18, base=(9 + k) << 32)
        rid = s.submit(short)
        assert s.run({rid: 101})[rid][1]["photons"]
        s.progress()                                     # nothing active: drain
        ids = {s.submit(r): int(r["shells"]) for r in LONG}
        launches = s.stats()[2] + 1
        t0 = time.monotonic()
        while s.stats()[2] < launches and time.monotonic() - t0 < 5.0:
            in_flight, _ = s.progress()
        assert in_flight == 1                            # the last launch has ended
        beside = small_calls(tmc_mod, tally, p)
        took = time.monotonic() - t0
        out = s.run(ids)
        assert took < 20.0
        assert same(before, beside)
        assert all(r["photons"] for _, r in out.values())
        assert s.stats()[2] == launches
    s.close()
