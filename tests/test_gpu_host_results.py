"""Host-array calls: results come through pinned memory that is allocated with
the context, in pieces, whatever their size and whatever runs beside the call."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PIECE = (1 << 22) - 64                     # bytes of one piece; two halves beyond
TALLIES, DOUBLES = PIECE // 32, PIECE // 8


@pytest.mark.parametrize("shells", [TALLIES, TALLIES + 1, TALLIES // 2 * 3, TALLIES // 2 * 4 + 1, DOUBLES // 2, DOUBLES // 2 + 1,
                                    DOUBLES // 4 * 3 + 1, DOUBLES // 2 * 2 + 5])
def test_results_in_pieces(tmc_mod, shells):
    torch = pytest.importorskip("torch")
    p = tmc_mod.params(shells=shells, microns_per_shell=6000.0 / shells, mu_a=2.0, mu_s=20.0, seed=6, math="fast")
    d = torch.zeros((shells, 4), dtype=torch.int64, device="cuda")
    steps = torch.zeros(1, dtype=torch.int64, device="cuda")
    tmc_mod.photon_batch_device(d.data_ptr(), 3000, p, steps.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    ref = d.cpu().numpy().view(np.uint64)
    tally, n = tmc_mod.photon_batch_fx(3000, p)
    got = np.stack([tally[f] for f in ("w_lo", "w_hi", "w2_lo", "w2_hi")], axis=1)
    assert n == int(steps.item()) and np.array_equal(got, ref) and ref[shells // 3 * 2:].any()
    heat, heat2 = np.full(shells, 0.5, np.float32), np.full(shells, 0.25, np.float32)
    tmc_mod.photon_batch(heat, heat2, 3000, p)
    h, h2 = tmc_mod.tally_to_heat(tally, p)
    assert np.array_equal(heat, (0.5 + h).astype(np.float32))
    assert np.array_equal(heat2, (0.25 + h2).astype(np.float32))


# A fresh process, whose first calls have few shells; then calls with more beside a
# persistent server launch that waits for this process.  No photons: a walk's shared
# memory need not fit beside the launch.
_CHILD = r"""
import json, sys, time
import numpy as np
sys.path.insert(0, ROOT); sys.path.insert(0, ROOT + "/tests")
import tiny_mc_gb300 as tmc
from tiny_mc_gb300.serve import Server
from test_gpu_serve import req
def calls(shells):
    par = tmc.params(shells=shells, seed=1)
    h, h2 = np.full(shells, 0.5, np.float32), np.full(shells, 0.25, np.float32)
    tmc.photon_batch(h, h2, 0, par)
    t, steps = tmc.photon_batch_fx(0, par)
    return bool((h == 0.5).all() and (h2 == 0.25).all() and not t["w_lo"].any() and steps == 0)
assert calls(101)
s = Server(slots=4, persistent=1, max_shells=101)
ids = {s.submit(r): int(r["shells"]) for r in (req(0.2, 90.0, 101, 1e-4, cap=1 << 16, base=1 << 32),)}
s.progress()
t0 = time.monotonic()
right = calls(2000) and calls(70000) and calls(300000)
took = time.monotonic() - t0
s.run(ids)
s.close()
print(json.dumps({"took": took, "right": right}))
"""


def test_larger_results_beside_a_persistent_launch():
    """(A call that waits for the launch, which waits for the host, ends after 120 s
    with an error.)"""
    out = subprocess.run([sys.executable, "-c", _CHILD.replace("ROOT", repr(ROOT))], capture_output=True, text=True,
                         timeout=300, env={**os.environ, "PYTHONPATH": ROOT})
    assert out.returncode == 0, out.stderr
    r = json.loads(out.stdout.strip().splitlines()[-1])
    assert r["took"] < 20.0 and r["right"], r
