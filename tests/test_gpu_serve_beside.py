"""While a persistent server launch holds the SMs (128-thread blocks), calls that
need few of them still run beside it: the colour map and the FP64 report."""
import time

import numpy as np
import pytest

from test_gpu_serve import req

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("math", ["exact", "fast"])
@pytest.mark.parametrize("stream", [0, 1])
def test_small_calls_beside_persistent_launch(tmc_mod, stream, math):
    from tiny_mc_gb300 import view
    from tiny_mc_gb300.serve import Server
    p = tmc_mod.params(seed=1)
    tally, _ = tmc_mod.photon_batch_fx(2000, p)
    heats = np.linspace(0.0, 1.0, 101, dtype=np.float32)
    image = view.colormap(heats, 64, 64)               # loads the kernels
    table = tmc_mod.report_fp64(tally, p, 2000)
    s = Server(slots=8, persistent=1, stream=stream, math=1 if math == "fast" else 0)
    ids = {s.submit(r): int(r["shells"]) for r in (req(0.2, 90.0, 101, 1e-4, cap=1 << 16, base=1 << 32),
                                                   req(2.0, 20.0, 501, 1e-4, cap=1 << 20, base=2 << 32))}
    s.progress()
    t0 = time.monotonic()
    again, table2 = view.colormap(heats, 64, 64), tmc_mod.report_fp64(tally, p, 2000)
    beside = time.monotonic() - t0
    out = s.run(ids)
    s.close()
    assert beside < 60.0        # a launch that kept them waiting gives up after 120 s
    assert all(np.array_equal(a, b) for a, b in zip(image, again))
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(table[:2], table2[:2]))
    assert all(r["photons"] for _, r in out.values())
