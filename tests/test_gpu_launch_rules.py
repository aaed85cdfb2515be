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


@pytest.mark.parametrize("math", ["exact", "fast"])
@pytest.mark.parametrize("optics", [PARAMS_H, HIGH_ALBEDO, dict(shells=20000, microns_per_shell=5.0, mu_a=2.0, mu_s=20.0),
                                    dict(shells=7, microns_per_shell=50.0, mu_a=10.0, mu_s=1.0),
                                    dict(shells=101, microns_per_shell=50.0, mu_a=0.5, mu_s=50.0)])
def test_whole_warp_walk_equals_lane_walk(tmc_mod, optics, math):
    """Photons walked one to a warp (small launches, and the last photons of
    every warp) against the same photons in the middle of a large launch, all
    of whose other photons are subtracted: the tallies are sums over photons."""
    tmc_mod.set_plain_launch(0, 0, 0)
    n = 257
    base = 5 << 20
    few, few_steps = gpu_fx(tmc_mod, n, seed=4, base=base, math=math, **optics)
    parts = [gpu_fx(tmc_mod, k, seed=4, base=b, math=math, **optics) for k, b in ((1, base), (n - 1, base + 1))]
    assert sum(s for _, s in parts) == few_steps

    def ints(t):
        return [(int(r[1]) << 64 | int(r[0]), int(r[3]) << 64 | int(r[2])) for r in t]
    summed = [tuple(x + y for x, y in zip(a, b)) for a, b in zip(ints(parts[0][0]), ints(parts[1][0]))]
    assert summed == ints(few)
    many = 40000 if optics is not HIGH_ALBEDO else 20000
    before = gpu_fx(tmc_mod, many, seed=4, base=base - many, math=math, **optics)
    both = gpu_fx(tmc_mod, many + n, seed=4, base=base - many, math=math, **optics)
    assert both[1] - before[1] == few_steps
    diff = [tuple(x - y for x, y in zip(a, b)) for a, b in zip(ints(both[0]), ints(before[0]))]
    assert diff == ints(few)


@pytest.mark.parametrize("shells", [1, 2, 31, 33, 130])
def test_last_shell_cells(tmc_mod, oracle_mod, shells):
    """An optically thin medium, nearly every deposit in the last shell: its
    per-lane cells add up to the oracle's tallies in the plain and batched forms
    (probe shell included: a served request's error is checked elsewhere)."""
    from test_gpu_parity import as_array
    from tiny_mc_gb300.sweep import PROBLEM_DTYPE
    optics = dict(shells=shells, microns_per_shell=10.0, mu_a=1.0, mu_s=4.0)
    n = 20011
    tmc_mod.set_plain_launch(0, 0, 0)
    ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=9, **optics)
    got, steps = gpu_fx(tmc_mod, n, seed=9, **optics)
    assert steps == ref_steps and np.array_equal(got, ref)
    pr = np.zeros(1, PROBLEM_DTYPE)
    for k, v in optics.items():
        pr[k] = v
    pr["n_photons"] = n
    for block, stream in ((128, False), (512, False), (128, True), (256, True)):
        b = tmc_mod.Batch(pr, seed=9, math="exact")
        b.set_config(block, 8, False, stream)
        b.run()
        t, s = b.read()
        b.close()
        assert int(s[0]) == ref_steps and np.array_equal(as_array(t), ref), (block, stream)


# Optics for the count table: rows up to the second, third or fourth roulette,
# the largest shell count and albedo that still take it, one shell, albedo 0,
# and walks of a few steps; then two the table is too large for.
COUNT_OPTICS = [PARAMS_H, dict(shells=1, microns_per_shell=50.0, mu_a=2.0, mu_s=20.0),
                dict(shells=101, microns_per_shell=50.0, mu_a=10.0, mu_s=1.0),
                dict(shells=101, microns_per_shell=50.0, mu_a=1.0, mu_s=0.0),
                dict(shells=501, microns_per_shell=20.0, mu_a=5.0, mu_s=5.0),
                dict(shells=130, microns_per_shell=50.0, mu_a=2.0, mu_s=16.0),
                dict(shells=101, microns_per_shell=50.0, mu_a=1.0, mu_s=12.0),
                dict(shells=1001, microns_per_shell=50.0, mu_a=1.0, mu_s=9.0)]


@pytest.mark.parametrize("math", ["exact", "fast"])
@pytest.mark.parametrize("optics", COUNT_OPTICS)
def test_counts_equal_sums(tmc_mod, optics, math):
    """The per-(step, shell) counts of default launches give the tallies and
    steps of the 64-bit sums (a given block size takes those), for enough
    photons that some outlive the table and lanes walk several each."""
    n = SMALL * 5 + 13
    tmc_mod.set_plain_launch(0, 0, 0)
    got = gpu_fx(tmc_mod, n, seed=6, base=1 << 34, math=math, **optics)
    tmc_mod.set_plain_launch(0, 1, 3)          # few blocks: hundreds of photons per lane
    few = gpu_fx(tmc_mod, n, seed=6, base=1 << 34, math=math, **optics)
    tmc_mod.set_plain_launch(512, 0, 0)
    ref = gpu_fx(tmc_mod, n, seed=6, base=1 << 34, math=math, **optics)
    tmc_mod.set_plain_launch(0, 0, 0)
    assert got[1] == ref[1] and few[1] == ref[1]
    assert np.array_equal(got[0], ref[0]) and np.array_equal(few[0], ref[0])


def test_counts_equal_oracle(tmc_mod, oracle_mod):
    tmc_mod.set_plain_launch(0, 0, 0)
    n = SMALL + 7
    got, steps = gpu_fx(tmc_mod, n, seed=12, **PARAMS_H)
    ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=12, **PARAMS_H)
    assert steps == ref_steps and np.array_equal(got, ref)


# Shell counts on both sides of the block histogram's limit (1057 / 1058 cells
# of a 128-thread block, 4513 / 4514 of a 512-thread one) and shell widths on
# both sides of the split form's reach; the last one deposits everywhere beyond.
@pytest.mark.parametrize("block", [0, 128, 512])
@pytest.mark.parametrize("shells,mps", [(1057, 50.0), (1058, 50.0), (1089, 5.0), (4513, 10.0), (4514, 10.0), (4544, 2.0),
                                        (4545, 0.5), (20000, 5.0), (20000, 0.05), (1 << 20, 0.001)])
def test_split_and_global_tallies(tmc_mod, oracle_mod, shells, mps, block):
    optics = dict(shells=shells, microns_per_shell=mps, mu_a=2.0, mu_s=20.0)
    n = 3001
    tmc_mod.set_plain_launch(block, 0, 0)
    got, steps = gpu_fx(tmc_mod, n, seed=3, **optics)
    tmc_mod.set_plain_launch(0, 0, 0)
    ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=3, **optics)
    assert steps == ref_steps and np.array_equal(got, ref)


@pytest.mark.parametrize("n", [152 * 256 - 1, 152 * 256, 152 * 256 + 1])
def test_block_rule_short_walks(tmc_mod, oracle_mod, n):
    optics = dict(shells=101, microns_per_shell=50.0, mu_a=10.0, mu_s=1.0)
    tmc_mod.set_plain_launch(0, 0, 0)
    got, steps = gpu_fx(tmc_mod, n, seed=5, **optics)
    ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=5, **optics)
    assert steps == ref_steps and np.array_equal(got, ref)
