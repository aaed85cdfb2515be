"""What a walk of many photons does to its shared tallies while it walks: one
block takes enough photons that its warps empty them in the middle of the walk."""
import numpy as np
import pytest

from test_gpu_parity import gpu_fx, oracle_fx

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
