"""The plain walk's launch rules: claim sizes and block sizes chosen by photon
count give the oracle's tallies bit for bit on both sides of every line."""
import numpy as np
import pytest

from test_gpu_parity import HIGH_ALBEDO, PARAMS_H, gpu_fx, oracle_fx

pytestmark = pytest.mark.gpu

SMALL = 152 * 512      # below: blocks of 128 on a 152-SM device


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 4865, SMALL - 1, SMALL, SMALL + 1])
def test_block_rule_params_h(tmc_mod, oracle_mod, n):
    tmc_mod.set_plain_launch(0, 0, 0)
    got, steps = gpu_fx(tmc_mod, n, seed=n, base=1 << 33, **PARAMS_H)
    ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=n, base=1 << 33, **PARAMS_H)
    assert steps == ref_steps
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("n", [1, 33, 517])
def test_block_rule_high_albedo(tmc_mod, oracle_mod, n):
    tmc_mod.set_plain_launch(0, 0, 0)
    got, steps = gpu_fx(tmc_mod, n, seed=n, **HIGH_ALBEDO)
    ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=n, **HIGH_ALBEDO)
    assert steps == ref_steps
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("math", ["exact", "fast"])
@pytest.mark.parametrize("n", [SMALL - 1, (1 << 20) + 3, 7296 * 32 * 4 * 2 + 5, 7296 * 256 * 4 + 1])
def test_claim_sizes_agree(tmc_mod, n, math):
    """Claims of 32 .. 256 photons: the default launch equals one 128-thread
    launch of few blocks, whose claims are as long as they get."""
    tmc_mod.set_plain_launch(0, 0, 0)
    got = gpu_fx(tmc_mod, n, math=math, **PARAMS_H)
    tmc_mod.set_plain_launch(128, 1, 0)
    try:
        ref = gpu_fx(tmc_mod, n, math=math, **PARAMS_H)
    finally:
        tmc_mod.set_plain_launch(0, 0, 0)
    assert got[1] == ref[1]
    assert np.array_equal(got[0], ref[0])
