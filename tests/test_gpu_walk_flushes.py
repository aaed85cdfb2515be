"""What a walk of many photons does to its shared tallies while it walks: one
block takes enough photons that its warps empty them in the middle of the walk."""
import numpy as np
import pytest

from test_gpu_parity import PARAMS_H, gpu_fx, oracle_fx

pytestmark = pytest.mark.gpu


# Shells of which the histogram holds the nearest (128 threads: 1056, 256: 2208,
# 512: 4512) and the last.  Photons end about sqrt(73) mean free paths of 455 um
# out: in some rows between the two, in some beyond all; one row has a single
# shell between; in the last ones the histogram holds the last shell alone.
@pytest.mark.parametrize("block,shells,mps,n", [(128, 2800, 2.3, 150000), (256, 2600, 1.2, 170000),
                                                (512, 20000, 5.0, 200000), (512, 20000, 0.6, 200000),
                                                (512, 5000, 0.6, 200000), (512, 4514, 0.6, 200000),
                                                (128, 20000, 0.1, 150000), (512, 20000, 0.1, 200000)])
def test_split_histogram_emptied_mid_walk(tmc_mod, oracle_mod, block, shells, mps, n):
    """A block's warps empty the histogram every 2^23 / threads iterations; n
    photons of about 76 steps on one block's lanes are more than that."""
    optics = dict(shells=shells, microns_per_shell=mps, mu_a=2.0, mu_s=20.0)
    tmc_mod.set_plain_launch(block, 1, 1)
    try:
        got, steps = gpu_fx(tmc_mod, n, seed=15, base=3 << 33, **optics)
    finally:
        tmc_mod.set_plain_launch(0, 0, 0)
    assert steps > 2 ** 23 * 1.2                     # iterations of a lane: steps / block and more
    ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=15, base=3 << 33, **optics)
    assert steps == ref_steps and np.array_equal(got, ref)


@pytest.mark.parametrize("thin", [0.62, 1e-4])
def test_last_shell_is_shared_in_every_form(tmc_mod, thin):
    """Photons that leave the shells all deposit into the last one.  4480 shells
    fit a block's histogram whole and more do not; as global atomics on one
    address 4600 took 97 times as long (19.4 against 0.20 ms), 2^20 shells that
    nearly all leave at once 100 times."""
    torch = pytest.importorskip("torch")
    ms = {}
    other = 4600 if thin == 0.62 else 1 << 20
    for shells in (4480, other):
        # the shells end at `thin` sqrt(1 + 73) mean free paths
        p = tmc_mod.params(shells=shells, microns_per_shell=3910.0 * thin / shells, mu_a=2.0, mu_s=20.0, seed=3, math="fast")
        d = torch.zeros((shells, 4), dtype=torch.int64, device="cuda")
        ws = torch.zeros(tmc_mod.workspace_bytes() // 8, dtype=torch.int64, device="cuda")
        s = torch.cuda.current_stream().cuda_stream
        times = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            tmc_mod.photon_batch_device(d.data_ptr(), 300000, p, 0, ws.data_ptr(), s)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        ms[shells] = min(times)
    assert ms[other] < 4 * ms[4480], ms


LOW_ALBEDO = dict(shells=101, microns_per_shell=50.0, mu_a=10.0, mu_s=1.0)


def sms():
    return pytest.importorskip("torch").cuda.get_device_properties(0).multi_processor_count


# The photons per SM from which a launch counts steps instead of summing weights.
@pytest.mark.parametrize("more", [-1, 0, 1])
@pytest.mark.parametrize("optics,line", [(PARAMS_H, 900), (LOW_ALBEDO, 256)])
def test_counts_line_equals_oracle(tmc_mod, oracle_mod, optics, line, more):
    n = sms() * line + more
    tmc_mod.set_plain_launch(0, 0, 0)
    got, steps = gpu_fx(tmc_mod, n, seed=12, base=1 << 35, **optics)
    ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=12, base=1 << 35, **optics)
    assert steps == ref_steps and np.array_equal(got, ref)


@pytest.mark.parametrize("math", ["exact", "fast"])
@pytest.mark.parametrize("optics,n", [(PARAMS_H, 1 << 25), (LOW_ALBEDO, 800_000_000)])
def test_counts_emptied_mid_walk(tmc_mod, optics, n, math):
    """A warp empties its block's counts every 2^22 iterations.  One block of 512
    threads walks enough photons for that; spread over the device, the same photons
    end long before it."""
    tmc_mod.set_plain_launch(0, 1, 1)
    try:
        got, steps = gpu_fx(tmc_mod, n, seed=13, base=1 << 36, math=math, **optics)
    finally:
        tmc_mod.set_plain_launch(0, 0, 0)
    assert steps / 512 > 1.1 * (1 << 22)             # iterations of a lane, and more
    ref, ref_steps = gpu_fx(tmc_mod, n, seed=13, base=1 << 36, math=math, **optics)
    assert steps == ref_steps and np.array_equal(got, ref)
