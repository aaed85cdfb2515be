"""Batches and served requests of short walks (a few steps a photon): they take
a kernel and a plan of their own, with the plain kernel's tallies."""
import numpy as np
import pytest

from test_gpu_batch import plain_tally
from test_gpu_parity import as_array
from test_gpu_serve import req

pytestmark = pytest.mark.gpu


def problems(k, n, mu_a, mu_s, shells=101):
    from tiny_mc_gb300.sweep import PROBLEM_DTYPE
    pr = np.zeros(k, PROBLEM_DTYPE)
    pr["shells"], pr["microns_per_shell"], pr["mu_a"], pr["mu_s"], pr["n_photons"] = shells, 50.0, mu_a, mu_s, n
    pr["photon_id_base"] = np.arange(k, dtype=np.uint64) * np.uint64(n)
    return pr


def ms(tmc_mod, pr, math, block, stream):
    torch = pytest.importorskip("torch")
    b = tmc_mod.Batch(pr, seed=5, math=math)
    b.set_config(block, 8, False, stream)
    times = []
    for _ in range(6):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        b.run()
        t1.record()
        t1.synchronize()
        times.append(t0.elapsed_time(t1))
    b.close()
    return min(times)


@pytest.mark.parametrize("math", ["exact", "fast"])
@pytest.mark.parametrize("block", [128, 256, 512])
@pytest.mark.parametrize("rest", [0, 1])
def test_short_batches_equal_plain(tmc_mod, math, block, rest):
    """Albedos over the kernel's range (up to 0.87, exact arithmetic 0.94) and the
    photons a warp walks whole (one per 8 steps to the first roulette), and none;
    `rest`: one longer problem that leaves most steps with the short ones, or does not."""
    pr = problems(9, 1500, 10.0, [0.0, 0.1, 1.0, 10.0, 13.7, 13.8, 30.0, 66.0, 68.0], [1, 2, 33, 101, 501, 7, 101, 101, 64])
    pr["n_photons"] = [1500, 33, 3000, 1, 257, 800, 1023, 50, 31]
    if rest:
        pr[0]["mu_a"], pr[0]["mu_s"], pr[0]["n_photons"] = 0.1, 30.0, 700
    b = tmc_mod.Batch(pr, seed=31, math=math)
    for graph, stream in ((False, False), (True, False), (False, True)):
        b.set_config(block, 8, graph, stream)
        b.run()
        t, s = b.read()
        for i in range(len(pr)):
            ref, ref_steps = plain_tally(tmc_mod, pr[i], 31, math)
            assert int(s[i]) == ref_steps, (i, graph, stream)
            assert np.array_equal(as_array(b.tally_of(t, i)), ref), (i, graph, stream)
    b.close()


@pytest.mark.parametrize("mu_s", [[0.1, 1.0, 5.0], [0.1, 1.0, 400.0]])
def test_short_requests_equal_plain(tmc_mod, mu_s):
    from tiny_mc_gb300.serve import Server
    reqs = [req(10.0, m, 101, 1e-3, cap=1 << 14, base=(3 + i) << 32) for i, m in enumerate(mu_s)]
    s = Server(slots=4)
    ids = {s.submit(r): int(r["shells"]) for r in reqs}
    out = s.run(ids)
    s.close()
    for rid, r in zip(ids, reqs):
        tally, res = out[rid]
        p = tmc_mod.params(shells=101, microns_per_shell=50.0, mu_a=10.0, mu_s=float(r["mu_s"]), seed=1,
                           photon_id_base=int(r["photon_id_base"]), math="fast")
        ref, steps = tmc_mod.photon_batch_fx(int(res["photons"]), p)
        assert int(res["photon_steps"]) == steps and np.array_equal(as_array(tally), as_array(ref))


@pytest.mark.parametrize("math", ["exact", "fast"])
def test_walks_of_one_step_cost_less_than_of_ten(tmc_mod, math):
    """4000 problems of 200 photons: with the last eight photons of a warp walked
    one by one by the whole warp, walks of one step took 0.83 (0.9) of the time of
    walks of ten; a whole-warp round costs as much for either."""
    one, ten = (ms(tmc_mod, problems(4000, 200, 10.0, m), math, 512, False) for m in (0.1, 10.0))
    assert one < 0.65 * ten, (one, ten)


@pytest.mark.parametrize("math", ["exact", "fast"])
def test_small_batch_is_one_turn_of_lanes(tmc_mod, math):
    """100 problems of 300 photons of three steps: a plan that gave short photons
    to whole warps, and a launch fewer blocks than items, took walk_stream 52 us
    where walk_batch took 24 (both about 20 us in one turn)."""
    pr = problems(100, 300, 10.0, 1.0)
    assert ms(tmc_mod, pr, math, 256, True) < 1.6 * ms(tmc_mod, pr, math, 256, False)


@pytest.mark.parametrize("math", ["exact", "fast"])
def test_equal_problems_take_one_route(tmc_mod, math):
    """300 equal problems of long walks, one photon to a lane: the plan takes all or
    none of them one photon to a warp, and as many blocks as there are items (in two
    turns of 152 blocks 512 threads take 1.5 of the time of 256; exact arithmetic's
    time varies from process to process by more than half of that)."""
    pr = problems(300, 200, 0.1, 100.0)
    if math == "fast":
        assert ms(tmc_mod, pr, math, 512, False) < 1.25 * ms(tmc_mod, pr, math, 256, False)
    b = tmc_mod.Batch(pr, seed=31, math=math)
    b.set_config(512, 8, False, False)
    b.run()
    t, s = b.read()
    b.close()
    for i in (0, 1, 299):
        ref, ref_steps = plain_tally(tmc_mod, pr[i], 31, math)
        assert int(s[i]) == ref_steps and np.array_equal(as_array(b.tally_of(t, i)), ref)
