"""Batches whose longest photons would set the end of the launch: fewer blocks
per SM and problems walked one photon to a warp give the plain kernel's tallies
for any block size and through a graph."""
import numpy as np
import pytest

from test_gpu_batch import plain_tally
from test_gpu_parity import as_array

pytestmark = pytest.mark.gpu


def long_and_short():
    """Photon counts around the smallest items (a photon per warp of 128 .. 512
    threads) of long problems beside many photons of short ones."""
    from tiny_mc_gb300.sweep import PROBLEM_DTYPE
    pr = np.zeros(12, PROBLEM_DTYPE)
    pr["shells"] = [101, 501, 1, 101, 501, 7, 101, 33, 501, 101, 2, 101]
    pr["microns_per_shell"] = 50.0
    pr["mu_a"] = [0.02, 0.05, 0.1, 0.1, 0.05, 5.0, 2.0, 1.0, 0.5, 10.0, 2.0, 0.03]
    pr["mu_s"] = [200.0, 300.0, 400.0, 100.0, 50.0, 1.0, 20.0, 0.0, 50.0, 1.0, 20.0, 90.0]
    pr["n_photons"] = [1, 3, 4, 5, 16, 4000, 3000, 33, 100, 5000, 0, 17]
    pr["photon_id_base"] = np.concatenate([[0], np.cumsum(pr["n_photons"][:-1])])
    return pr


@pytest.mark.parametrize("math", ["exact", "fast"])
@pytest.mark.parametrize("block,ipb,graph", [(128, 4, False), (256, 8, True), (512, 16, False), (128, 1, True)])
def test_long_problems_one_photon_per_warp(tmc_mod, math, block, ipb, graph):
    pr = long_and_short()
    b = tmc_mod.Batch(pr, seed=21, math=math)
    b.set_config(block, ipb, graph, False)
    for _ in range(2):
        b.run()
        t, s = b.read()
        for i in range(len(pr)):
            if pr["n_photons"][i] == 0:
                assert s[i] == 0 and not as_array(b.tally_of(t, i)).any()
                continue
            ref, ref_steps = plain_tally(tmc_mod, pr[i], 21, math)
            assert int(s[i]) == ref_steps, i
            assert np.array_equal(as_array(b.tally_of(t, i)), ref), i
    # another kernel and back: the problems' claims follow the plan
    b.set_config(block, ipb, graph, True)
    b.run()
    t2, s2 = b.read()
    b.set_config(block, ipb, graph, False)
    b.run()
    t3, s3 = b.read()
    b.close()
    assert np.array_equal(t2, t) and np.array_equal(s2, s)
    assert np.array_equal(t3, t) and np.array_equal(s3, s)
