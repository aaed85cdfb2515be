"""The work that a user of this library has it do, as measurable cases.

Kinds of case (each runs one pass through the public entry points):

  host     photon_batch: the drop-in call, float32 heat/heat2 in host arrays
  fx       photon_batch_fx: exact integer tallies and the photon-step count
  device   photon_batch_device: tallies in device memory on the caller's stream
  frame    the viewer's frame: a few photons, then the colour map of the heat
  batch    Batch.run + Batch.read: many problems in one persistent launch
  serve    Server.submit + Server.run: requests that stop at their target RSE

Optics are the repository's own: params_h (the reference's defaults),
high_albedo, low_albedo, fine_shells and wide_shells (more shells than a
shared-memory histogram holds), and the sweep's parameter distribution.
"""
import math

import numpy as np
import torch

import tiny_mc_gb300 as tmc
from tiny_mc_gb300 import serve, sweep, view

OPTICS = {
    # shells, microns per shell, mu_a (1/cm), mu_s (1/cm)
    "params_h": (101, 50.0, 2.0, 20.0),
    "high_albedo": (1001, 10.0, 0.1, 100.0),
    "low_albedo": (101, 50.0, 10.0, 1.0),
    "fine_shells": (4001, 1.0, 2.0, 20.0),
    "wide_shells": (20000, 5.0, 2.0, 20.0),
}

# Floating-point operations of one photon step: logarithm 2, move 6, radius 7,
# square and decay of the weight 2, 1.27 rejection tries of 7, direction 7.
FLOPS_PER_STEP = 34

IMAGE = 800   # the viewer's window


def listed():
    return [
        # the viewer's loop: up to 20 photons a frame, then every pixel's colour
        {"name": "viewer_frame", "kind": "frame", "optics": "params_h", "photons": 20, "math": "exact"},
        # the reference's own run: 32768 photons, default arithmetic, host arrays
        {"name": "drop_in", "kind": "host", "optics": "params_h", "photons": 32768, "math": "exact"},
        # a usual accuracy run through the drop-in call, an odd count
        {"name": "host_1m", "kind": "host", "optics": "params_h", "photons": 1000003, "math": "fast"},
        # a device-resident tally advanced on the caller's stream
        {"name": "device_16m", "kind": "device", "optics": "params_h", "photons": 1 << 24, "math": "fast"},
        # the large run of the headline benchmark (an eighth of it)
        {"name": "host_128m", "kind": "host", "optics": "params_h", "photons": 1 << 27, "math": "fast"},
        # the bit-reproducible arithmetic at size, with its exact tallies
        {"name": "exact_32m", "kind": "fx", "optics": "params_h", "photons": 1 << 25, "math": "exact"},
        # a quick look at a high-albedo medium: few photons, thousands of steps each
        {"name": "albedo_4k", "kind": "fx", "optics": "high_albedo", "photons": 4099, "math": "exact"},
        # the high-albedo workload: long walks, 1001 shells
        {"name": "albedo_512k", "kind": "device", "optics": "high_albedo", "photons": 1 << 19, "math": "fast"},
        # more shells than shared memory holds: deposits go to the global tally
        {"name": "wide_2m", "kind": "fx", "optics": "wide_shells", "photons": 2000003, "math": "fast"},
        # a parameter study of ordinary size with the library's default launch
        {"name": "study_256", "kind": "batch", "problems": 256, "log2_photons": 14.0, "mu_a_min": 0.1,
         "math": "exact", "block": 256, "items": 8, "graph": False, "stream": False},
        # the 4096-problem sweep at a reduced photon scale, replayed through its graph
        {"name": "sweep_4096", "kind": "batch", "problems": 4096, "log2_photons": 12.0, "mu_a_min": 0.01,
         "math": "fast", "block": 128, "items": 16, "graph": True, "stream": False},
        # a burst of requests served to their target errors
        {"name": "serve_48", "kind": "serve", "requests": 48, "rse_min": 0.02, "mu_a_min": 0.1,
         "photons": 1 << 18, "math": "fast"},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame", "host", "host", "fx", "fx", "device", "device", "batch", "batch", "serve"])
    arith = rng.choice(["exact", "fast"])
    if kind == "frame":
        return {"kind": kind, "optics": "params_h", "photons": rng.randint(1, 20), "math": arith}
    if kind == "batch":
        return {"kind": kind, "problems": log_int(16, 2048), "log2_photons": round(rng.uniform(8.0, 14.0), 2),
                "mu_a_min": round(math.exp(rng.uniform(math.log(0.03), math.log(1.0))), 3), "math": arith,
                "block": rng.choice([128, 256, 512]), "items": rng.choice([4, 8, 16]),
                "graph": rng.random() < 0.5, "stream": rng.random() < 0.4}
    if kind == "serve":
        return {"kind": kind, "requests": log_int(4, 48), "rse_min": round(rng.uniform(0.02, 0.04), 4),
                "mu_a_min": round(rng.uniform(0.1, 1.0), 3), "photons": log_int(1 << 15, 1 << 18), "math": arith}
    name = rng.choice(["params_h", "params_h", "high_albedo", "low_albedo", "fine_shells", "wide_shells"])
    most = {"high_albedo": 1 << 19, "wide_shells": 1 << 21}.get(name, 1 << 26)
    least = 256 if name == "high_albedo" else 1024
    return {"kind": kind, "optics": name, "photons": log_int(least, most) | 1, "math": arith}


# ------------------------------------------------------------------ inputs

def _params(case, seed):
    shells, mps, mu_a, mu_s = OPTICS[case["optics"]]
    return tmc.params(shells, mps, mu_a, mu_s, seed=_key(seed), math=case["math"])


def _key(seed):
    """The Philox key of a seed: any two seeds below 2^63 differ."""
    return int(seed) & (2**63 - 1)


def _problems(case, seed):
    """The sweep's distribution over mu_a >= mu_a_min; photon counts
    log-uniform over a factor of 32 below 2^log2_photons.  The optics are the
    study's, so they do not change with the seed; the photons do."""
    top = case["log2_photons"]
    return sweep.make_sweep(case["problems"], seed=case["problems"], log2_photons=(top - 5.0, top),
                            mu_a_range=(case["mu_a_min"], 10.0))


def _requests(case, seed):
    req, _ = serve.make_trace(case["requests"], seed=case["requests"], rse=(case["rse_min"], 0.05),
                              max_photons=case["photons"], mu_a_range=(case["mu_a_min"], 10.0))
    return req


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = tmc.Batch(_problems(case, seed), seed=_key(seed), math=case["math"])
        b.set_config(case["block"], case["items"], case["graph"], case["stream"])
        return {"kind": kind, "batch": b}
    if kind == "serve":
        math_id = tmc.MATH_FAST if case["math"] == "fast" else tmc.MATH_EXACT
        s = serve.Server(slots=64, seed=_key(seed), math=math_id)
        return {"kind": kind, "server": s, "requests": _requests(case, seed)}
    state = {"kind": kind, "photons": case["photons"], "params": _params(case, seed)}
    if kind == "device":
        shells = state["params"].shells
        state["tally"] = torch.zeros((shells, 4), dtype=torch.int64, device="cuda")
        state["steps"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        state["workspace"] = torch.zeros(tmc.workspace_bytes(), dtype=torch.uint8, device="cuda")
    return state


# --------------------------------------------------------------------- run

def _words(tally):
    """Integer tallies as rows of four 64-bit words."""
    return tally.view("<i8").reshape(-1, 4)


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        b.run(torch.cuda.current_stream().cuda_stream)
        tallies, steps = b.read()
        return [_words(tallies), steps.view(np.int64)]
    if kind == "serve":
        s = state["server"]
        ids = {}
        for r in state["requests"]:
            ids[s.submit(r)] = int(r["shells"])
        out = s.run(ids)
        tallies = np.concatenate([_words(out[i][0]) for i in ids])
        res = [out[i][1] for i in ids]
        counts = np.array([[int(r[f]) for f in ("photons", "photon_steps", "batches", "reached_target")]
                           for r in res], np.int64)
        return [tallies, counts, np.array([float(r["rse"]) for r in res])]
    p, n = state["params"], state["photons"]
    if kind == "device":
        state["tally"].zero_()
        state["steps"].zero_()
        tmc.photon_batch_device(state["tally"].data_ptr(), n, p, state["steps"].data_ptr(),
                                state["workspace"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return [state["tally"], state["steps"]]
    if kind == "fx":
        tally, steps = tmc.photon_batch_fx(n, p)
        return [_words(tally), steps]
    heat = np.zeros(p.shells, np.float32)
    heat2 = np.zeros(p.shells, np.float32)
    tmc.photon_batch(heat, heat2, n, p)
    if kind == "host":
        return [heat, heat2]
    red, rgba = view.colormap(heat, IMAGE, IMAGE)
    return [heat, heat2, red, rgba]


# -------------------------------------------------------------------- work

def work(case):
    """Expected photon steps times the operations of one; the results written
    once and the parameters read once (the walk has no input arrays)."""
    kind = case["kind"]
    if kind == "batch":
        pr = _problems(case, 0)
        steps = sum(tmc.expected_steps(float(q["mu_a"]), float(q["mu_s"])) * float(q["n_photons"]) for q in pr)
        out = 32 * int(pr["shells"].sum()) + 8 * len(pr)
        return {"bytes": out + pr.nbytes, "flops": FLOPS_PER_STEP * steps}
    if kind == "serve":
        # a request walks 16 batches at least; how many more follows from its error
        cfg = serve.default_config()
        steps = 0.0
        out = 0
        for r in _requests(case, 0):
            batch, _, per = serve.plan(r, cfg)
            steps += per * min(float(r["max_photons"]), 16.0 * batch)
            out += 32 * int(r["shells"]) + 48
        return {"bytes": out, "flops": FLOPS_PER_STEP * steps}
    shells, _, mu_a, mu_s = OPTICS[case["optics"]]
    steps = tmc.expected_steps(mu_a, mu_s) * case["photons"]
    out = {"host": 8, "frame": 8, "fx": 32, "device": 32}[kind] * shells + 40
    flops = FLOPS_PER_STEP * steps
    if kind == "frame":
        out += 8 * IMAGE * IMAGE
        flops += 16 * IMAGE * IMAGE
    return {"bytes": out, "flops": flops}


# ------------------------------------------------------------------- exact

def _philox(key, blk, pid):
    """Philox-4x32-10 of counter {blk, 0, pid low, pid high}: four words, as
    int64 tensors."""
    mask = 0xffffffff
    c0, c1, c2, c3 = blk & mask, torch.zeros_like(blk), pid & mask, (pid >> 32) & mask
    k0, k1 = key & mask, (key >> 32) & mask
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & mask) ^ c1 ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c3 ^ k1, p0 & mask
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return torch.stack([c0, c1, c2, c3])


def _uniform(key, pid, pos):
    """The photon's draws rand()/RAND_MAX at stream positions pos."""
    w = _philox(key, pos >> 2, pid).gather(0, (pos & 3).unsqueeze(0))[0]
    return torch.clamp(w >> 1, min=1).double() / 2.0**31


def _walk(shells, mps, mu_a, mu_s, key, first, count, device):
    """photon.c's walk of photons first .. first + count - 1 in 64 bits."""
    albedo = mu_s / (mu_s + mu_a)
    spm = 1e4 / mps / (mu_a + mu_s)
    pid = torch.arange(first, first + count, device=device)
    pos = torch.zeros_like(pid)
    xyz = torch.zeros((3, count), dtype=torch.float64, device=device)
    uvw = torch.zeros_like(xyz)
    uvw[2] = 1.0
    weight = torch.ones(count, dtype=torch.float64, device=device)
    heat = torch.zeros(shells, dtype=torch.float64, device=device)
    heat2 = torch.zeros_like(heat)
    while pid.numel():
        t = -torch.log(_uniform(key, pid, pos))
        pos = pos + 1
        xyz = xyz + t * uvw
        shell = (xyz.pow(2).sum(0).sqrt() * spm).clamp(max=shells - 1).long()
        dep = (1.0 - albedo) * weight
        heat.index_add_(0, shell, dep)
        heat2.index_add_(0, shell, dep * dep)
        weight = weight * albedo
        todo = torch.arange(pid.numel(), device=device)
        while todo.numel():
            a = 2.0 * _uniform(key, pid[todo], pos[todo]) - 1.0
            b = 2.0 * _uniform(key, pid[todo], pos[todo] + 1) - 1.0
            pos[todo] += 2
            s = a * a + b * b
            ok = s <= 1.0
            i, a, b, s = todo[ok], a[ok], b[ok], s[ok]
            u = 2.0 * s - 1.0
            scale = ((1.0 - u * u) / s).sqrt()
            uvw[0, i], uvw[1, i], uvw[2, i] = u, a * scale, b * scale
            todo = todo[~ok]
        low = weight < 0.001
        u = _uniform(key, pid, pos)
        pos = pos + low.long()
        alive = ~(low & (u > 0.1))
        weight = torch.where(low, weight / 0.1, weight)
        pid, pos, weight = pid[alive], pos[alive], weight[alive]
        xyz, uvw = xyz[:, alive], uvw[:, alive]
    return heat, heat2


def exact(case, seed):
    """heat and heat2 (and the colour map's red) in 64 bits on the same draws.
    None for integer tallies, which have to be equal, and for long walks."""
    if case["kind"] not in ("host", "frame"):
        return None
    shells, mps, mu_a, mu_s = OPTICS[case["optics"]]
    per = tmc.expected_steps(mu_a, mu_s)
    if per > 500.0 or per * case["photons"] > 4e8:
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    heat, heat2 = 0.0, 0.0
    part = 1 << 20
    for first in range(0, case["photons"], part):
        h, h2 = _walk(shells, mps, mu_a, mu_s, _key(seed), first, min(part, case["photons"] - first), device)
        heat, heat2 = heat + h, heat2 + h2
    heat, heat2 = heat.cpu().numpy(), heat2.cpu().numpy()
    if case["kind"] == "host":
        return [heat, heat2]
    c = (np.arange(IMAGE) + 0.5) / 800.0 - 0.5
    r = np.sqrt(c[None, :] ** 2 + c[:, None] ** 2)
    shell = np.minimum((r / math.sqrt(0.5) * (shells - 1)).astype(np.int64), shells - 1)
    return [heat, heat2, 2.0 / (1.0 + np.exp(-0.004 * heat[shell])) - 1.0, None]
