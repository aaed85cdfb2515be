"""Device-form calls without a workspace share the library's photon claim
counter: a call on one stream waits on the GPU for the call before it on another."""
import numpy as np
import pytest

from test_gpu_parity import PARAMS_H, oracle_fx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("math", ["exact"])
def test_calls_on_two_streams_are_ordered(tmc_mod, oracle_mod, math):
    """One block walks 65536 photons, which takes tens of milliseconds; two calls made
    meanwhile on other streams, with counters of their own they would finish first,
    must not have it hand out its photons anew."""
    torch = pytest.importorskip("torch")
    counts = (1 << 16, 4096, 513)
    streams = [torch.cuda.Stream() for _ in counts]
    tallies = [torch.zeros((101, 4), dtype=torch.int64, device="cuda") for _ in counts]
    steps = torch.zeros(len(counts), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    tmc_mod.set_plain_launch(512, 1, 1)
    try:
        base = 0
        for k, n in enumerate(counts):
            p = tmc_mod.params(seed=21, photon_id_base=base, math=math, **PARAMS_H)
            tmc_mod.photon_batch_device(tallies[k].data_ptr(), n, p, steps.data_ptr() + 8 * k, 0, streams[k].cuda_stream)
            base += n
    finally:
        tmc_mod.set_plain_launch(0, 0, 0)
    torch.cuda.synchronize()
    base = 0
    for k, n in enumerate(counts):
        ref, _, ref_steps = oracle_fx(oracle_mod, n, seed=21, base=base, **PARAMS_H)
        assert np.array_equal(tallies[k].cpu().numpy().view(np.uint64), ref) and int(steps[k].item()) == ref_steps, k
        base += n
