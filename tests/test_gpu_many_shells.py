"""Small launches over more shells than eight blocks' histograms hold: which
block size they take does not change the tallies, and short walks take the one
whose histograms cost less to set up and add."""
import numpy as np
import pytest

from test_gpu_parity import gpu_fx, oracle_fx

pytestmark = pytest.mark.gpu


# shells on both sides of what eight 128-thread blocks (1057), two 512-thread
# blocks (4513) and one (11809) have room for; walks of 3 steps and of 31
@pytest.mark.parametrize("mu_a,mu_s", [(10.0, 1.0), (4.0, 16.0)])
@pytest.mark.parametrize("shells", [1057, 1058, 4513, 4514, 11809, 11810])
@pytest.mark.parametrize("mps", [0.15, 0.4, 3.0])
def test_forms_equal_oracle(tmc_mod, oracle_mod, shells, mps, mu_a, mu_s):
    optics = dict(shells=shells, microns_per_shell=mps, mu_a=mu_a, mu_s=mu_s)
    tmc_mod.set_plain_launch(0, 0, 0)
    got, steps = gpu_fx(tmc_mod, 20011, seed=8, **optics)
    ref, _, ref_steps = oracle_fx(oracle_mod, 20011, seed=8, **optics)
    assert steps == ref_steps and np.array_equal(got, ref)


def test_short_walks_take_the_cheaper_block(tmc_mod):
    """75000 photons of 3 steps, 12000 shells of 0.3 um: 83 us in 128-thread blocks,
    29 in 512-thread ones."""
    torch = pytest.importorskip("torch")
    p = tmc_mod.params(shells=12000, microns_per_shell=0.3, mu_a=10.0, mu_s=1.0, seed=3, math="fast")
    d = torch.zeros((12000, 4), dtype=torch.int64, device="cuda")
    ws = torch.zeros(tmc_mod.workspace_bytes() // 8, dtype=torch.int64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    n = torch.cuda.get_device_properties(0).multi_processor_count * 490
    ms = {}
    for block in (0, 512):
        tmc_mod.set_plain_launch(block, 0, 0)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            tmc_mod.photon_batch_device(d.data_ptr(), n, p, 0, ws.data_ptr(), s)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        ms[block] = min(times)
    tmc_mod.set_plain_launch(0, 0, 0)
    assert ms[0] < 1.6 * ms[512], ms
