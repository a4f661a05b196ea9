"""Performance cases of the gravity FMM library, through its public Python entry points.

A case is a dict of plain values: ``kind`` says which call it times
(``step``: preprocess, RK4 steps, postprocess of a Solver; ``batch``: the same
of a Batch of independent systems; ``accel``: one force evaluation, with or
without potentials; ``direct``: the FP64 direct sum on a sample of targets),
``model`` the particle distribution, and the rest the solver's parameters.
``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges,
``prepare`` the inputs and the solver a program keeps, ``run`` one pass,
``work`` the bytes and operations a pass cannot do without, ``exact`` the same
outputs from direct summation in 64 bits.

A pass starts from host arrays and ends with host arrays, as the solver's
preprocess / solve / postprocess boundary does; from 1,000,000 particles on
they are pinned buffers (upload_ptr / download_ptr), as bench.py's end-to-end
measurement has them (a batch's inputs always). The library's shipped tuning cache is in effect, as in
bench.py.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "vipp-nbody-bench_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
os.environ.setdefault("VIPP_GB_TUNE_FILE", os.path.join(PKG, "vipp_gb300", "tuning_gb300.txt"))

import vipp_gb300  # noqa: E402

PINNED_FROM = 1_000_000   # particles from which the host arrays are pinned buffers
EXACT_PAIRS = 6e10        # direct-sum pairs exact() computes at most


def _step(name, model, n, p, s, eps, dt, steps, precision, split="tf32", mode="ref"):
    return {"name": name, "kind": "step", "model": model, "n": n, "p": p, "s": s, "eps": eps, "dt": dt, "steps": steps,
            "precision": precision, "split": split, "mode": mode}


def listed():
    return [
        # The smallest call: one force evaluation at the library's default parameters, where latency and launches count.
        {"name": "accel_1k_fp64", "kind": "accel", "model": "plummer", "n": 1000, "p": 4, "s": 10, "eps": 0.01,
         "precision": "fp64", "split": "tf32", "potential": False},
        # A small simulation in mixed precision, an odd particle count.
        _step("step_3k_mixed", "plummer", 3001, 6, 32, 0.01, 5e-4, 4, "mixed"),
        # The reference's CPU-runnable configuration, ten RK4 steps in double precision as the reference runs them.
        _step("step_16k_fp64", "plummer", 16384, 4, 32, 0.01, 1e-3, 10, "fp64"),
        # An ordinary mixed-precision run at the library's default M2L split, ragged size.
        _step("step_100k_mixed", "plummer", 100003, 8, 64, 0.005, 5e-4, 4, "mixed"),
        # Forces and potentials of an ordinary system in double precision (energy diagnostics).
        {"name": "accel_phi_131k_fp64", "kind": "accel", "model": "plummer", "n": 131071, "p": 8, "s": 64, "eps": 0.005,
         "precision": "fp64", "split": "tf32", "potential": True},
        # Double-precision step of the unit-cube configuration.
        _step("step_cube_262k_fp64", "cube", 262144, 6, 64, 1e-3, 1e-4, 1, "fp64"),
        # The accuracy check: FP64 direct sum on a sample of targets.
        {"name": "direct_4k_of_262k", "kind": "direct", "model": "plummer", "n": 262144, "targets": 4096, "p": 8, "s": 64,
         "eps": 0.005, "precision": "mixed", "split": "bf16"},
        # The plain-at-scale unit cube, small leaves.
        _step("step_cube_1m_bf16", "cube", 1048576, 6, 64, 1e-3, 1e-4, 4, "mixed", "bf16"),
        # The accurate mode (softened far field) at its order, a size off the powers of two.
        _step("step_accurate_1m", "plummer", 1000003, 10, 64, 0.005, 5e-4, 2, "mixed", "tf32", "accurate"),
        # The headline: two steps of the 4M Plummer sphere.
        _step("step_plummer_4m_bf16", "plummer", 4194304, 8, 64, 0.005, 5e-4, 2, "mixed", "bf16"),
        # Many independent systems of uneven size advanced together.
        {"name": "batch_512_bf16", "kind": "batch", "model": "plummer", "systems": 512, "n_lo": 1024, "n_hi": 65536, "p": 6,
         "s": 64, "eps": 0.01, "dt": 5e-4, "steps": 2, "precision": "mixed", "split": "bf16"},
        # The largest: the adaptive-depth stress workload.
        _step("step_clusters_16m_bf16", "clusters", 16777216, 8, 64, 1e-4, 1e-4, 2, "mixed", "bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: sizes over their logarithm, odd ones among them."""
    family = rng.choice(["small", "fp64", "mixed", "mixed", "bf16", "bf16", "clusters", "accurate", "batch", "accel", "direct"])
    eps = rng.choice([0.005, 0.01])
    if family == "small":
        return {"kind": "accel", "model": rng.choice(["plummer", "cube"]), "n": _log_int(rng, 300, 20000), "p": rng.choice([2, 4, 5, 6]),
                "s": rng.choice([10, 16, 32]), "eps": eps, "precision": "fp64", "split": "tf32", "potential": rng.random() < 0.3}
    if family == "accel":
        return {"kind": "accel", "model": rng.choice(["plummer", "cube"]), "n": _log_int(rng, 20000, 300000), "p": rng.choice([4, 6, 7, 8]),
                "s": rng.choice([32, 64]), "eps": eps, "precision": "fp64", "split": "tf32", "potential": rng.random() < 0.5}
    if family == "direct":
        n = _log_int(rng, 20000, 1000000)
        return {"kind": "direct", "model": "plummer", "n": n, "targets": min(_log_int(rng, 200, 10000), int(2e9 / n)), "p": 8, "s": 64,
                "eps": eps, "precision": "mixed", "split": "bf16"}
    if family == "batch":
        lo = rng.choice([500, 1024, 2000])
        return {"kind": "batch", "model": "plummer", "systems": _log_int(rng, 8, 512), "n_lo": lo, "n_hi": rng.choice([8000, 30000, 65536]),
                "p": rng.choice([4, 6, 8]), "s": rng.choice([32, 64]), "eps": 0.01, "dt": 5e-4, "steps": 2, "precision": "mixed",
                "split": rng.choice(["bf16", "bf16", "tf32"])}
    c = _step("", "plummer", 0, 8, 64, eps, 5e-4, 2, "mixed")
    del c["name"]
    if family == "fp64":
        c.update(model=rng.choice(["plummer", "cube"]), n=_log_int(rng, 1000, 200000), p=rng.choice([4, 6, 7, 8]), s=rng.choice([32, 64]),
                 precision="fp64", dt=1e-3)
        c["steps"] = max(1, min(10, 100000 // c["n"]))
    elif family == "mixed":
        c.update(model=rng.choice(["plummer", "plummer", "cube"]), n=_log_int(rng, 1500, 1000000), p=rng.choice([4, 6, 8, 9, 10]),
                 s=rng.choice([32, 64]))
        c["steps"] = max(1, min(4, 200000 // c["n"]))
    elif family == "bf16":
        c.update(model=rng.choice(["plummer", "plummer", "cube"]), n=_log_int(rng, 100000, 8000000), p=rng.choice([6, 8]),
                 s=rng.choice([32, 64]), split="bf16")
    elif family == "clusters":
        c.update(model="clusters", n=_log_int(rng, 500000, 16000000), eps=1e-4, dt=1e-4, split="bf16")
    else:
        c.update(n=_log_int(rng, 10000, 3000000), p=10, mode="accurate")
    return c


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _isotropic(norm, g):
    z = (1 - 2 * _rand(g, norm.numel())) * norm
    w = (norm * norm - z * z).clamp_min(0).sqrt()
    a = 2 * math.pi * _rand(g, norm.numel())
    return torch.stack([w * a.cos(), w * a.sin(), z], 1)


def _plummer(n, g, r_max=10.0):
    """Plummer sphere, G = M = a = 1, radii capped at r_max, speeds from its distribution function."""
    cap = (1 + r_max ** -2) ** -1.5
    u = _rand(g, n) * cap
    r = (u.clamp_min(1e-12) ** (-2 / 3) - 1) ** -0.5
    q = torch.full((n,), -1.0, device="cuda", dtype=torch.float64)
    for _ in range(64):
        a, b = _rand(g, n), 0.1 * _rand(g, n)
        q = torch.where((q < 0) & (b < a * a * (1 - a * a) ** 3.5), a, q)
    q = q.clamp_min(0.0)
    return _isotropic(r, g), _isotropic(q * math.sqrt(2) * (1 + r * r) ** -0.25, g)


def _particles(case, seed):
    """Positions and velocities (n, 3), FP64 on the GPU, made from the seed alone."""
    g = _gen(seed)
    n = case["n"]
    if case["model"] == "plummer":
        return _plummer(n, g)
    if case["model"] == "cube":  # unit cube at about its virial velocity dispersion
        return _rand(g, n, 3), 0.5 * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    x, v, at = torch.empty(n, 3, device="cuda", dtype=torch.float64), torch.zeros(n, 3, device="cuda", dtype=torch.float64), 0
    inside = n - int(round(0.05 * n))  # 8 equal-mass Plummer clusters, the rest a uniform background at rest
    for k in range(8):
        m = inside // 8 + (k < inside % 8)
        centre, radius = _rand(g, 3), 0.01 + 0.09 * float(_rand(g, 1))
        bulk = 0.3 * torch.randn(3, generator=g, device="cuda", dtype=torch.float64)
        xc, vc = _plummer(m, g)
        x[at:at + m] = centre + radius * xc
        v[at:at + m] = bulk + math.sqrt(m / n / radius) * vc
        at += m
    x[at:] = _rand(g, n - at, 3)
    return x, v


def _sizes(case):
    rng = np.random.default_rng([case["systems"], case["n_lo"], case["n_hi"]])
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])  # uniform in the logarithm, as the batching workload
    return np.exp(rng.uniform(lo, hi, case["systems"])).round().astype(np.int64)


def _batch_particles(case, seed):
    """Every system a Plummer sphere of mass 1 scaled to a radius uniform in [0.5, 2]."""
    g, sizes = _gen(seed), _sizes(case)
    x, v = _plummer(int(sizes.sum()), g)
    of = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), torch.from_numpy(sizes).cuda())
    r = (0.5 + 1.5 * _rand(g, len(sizes)))[of][:, None]
    return sizes, x * r, v * r ** -0.5


def _flags(case):
    return vipp_gb300.FLAG_M2L_BF16 if case["split"] == "bf16" else 0


def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "batch":
        sizes, x, v = _batch_particles(case, seed)
        state["batch"] = vipp_gb300.Batch(sizes, p=case["p"], s=case["s"], eps=case["eps"], masses=1.0 / sizes,
                                          precision=case["precision"], flags=_flags(case))
        state["x"], state["v"] = (torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(q).numpy() for q in (x, v))
        return state
    x, v = _particles(case, seed)
    n = case["n"]
    state["solver"] = vipp_gb300.Solver(p=case["p"], s=case["s"], eps=case["eps"], m=1.0 / n, precision=case["precision"],
                                        flags=_flags(case), mode=case.get("mode", "ref"))
    if n >= PINNED_FROM and case["kind"] == "step":
        state["xv"] = torch.empty(2, n, 3, dtype=torch.float64, pin_memory=True)
        state["out"] = torch.empty(2, n, 3, dtype=torch.float64, pin_memory=True)
        state["xv"][0].copy_(x)
        state["xv"][1].copy_(v)
    else:
        state["x"], state["v"] = x.cpu().numpy(), v.cpu().numpy()
    if case["kind"] == "direct":
        state["targets"] = _targets(case, seed)
    return state


def _targets(case, seed):
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 11])
    return np.sort(rng.choice(case["n"], case["targets"], replace=False))


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.upload(state["x"], state["v"])
        for _ in range(case["steps"]):
            b.step(case["dt"])
        return b.download()
    s = state["solver"]
    if "xv" in state:
        xv, out = state["xv"], state["out"]
        s.upload_ptr(xv[0].data_ptr(), xv[1].data_ptr(), case["n"])
        for _ in range(case["steps"]):
            s.solve(case["dt"])
        s.download_ptr(out[0].data_ptr(), out[1].data_ptr())
        return out[0], out[1]
    s.preprocess(state["x"], state["v"])
    if case["kind"] == "accel":
        return s.accel(potential=case["potential"])
    if case["kind"] == "direct":
        return s.direct_accel(state["targets"])
    for _ in range(case["steps"]):
        s.solve(case["dt"])
    return s.postprocess()


def work(case):
    """State in and out once, plus the method's operations: 20 per near-field pair, 2 K^2 per M2L pair.

    Pairs per particle from the tree's typical occupancy: leaves of a
    centrally concentrated system hold about half their limit T = floor(sqrt(8) s)
    (27 neighbours each), those of a cube n / 8^L at the depth L its limit
    asks for; a cell has 189 M2L sources.
    """
    if case["kind"] == "direct":
        return {"bytes": 24.0 * case["n"] + 24.0 * case["targets"], "flops": 20.0 * case["n"] * case["targets"]}
    n = float(_sizes(case).sum()) if case["kind"] == "batch" else case["n"]
    limit = math.floor(math.sqrt(8) * case["s"])
    if case["model"] == "cube":
        depth = max(0, math.ceil(math.log(n / limit, 8))) if n > limit else 0
        leaf = n / 8 ** depth
    else:
        leaf = min(n, limit / 2)
    k = (case["p"] + 1) ** 2
    flops = 20.0 * n * min(n, 27 * leaf) + 2.0 * k * k * 189 * max(0.0, n / leaf - 8)
    evals = 1 if case["kind"] == "accel" else 4 * case["steps"]
    state = 48.0 * n if case["kind"] == "accel" and not case["potential"] else 56.0 * n if case["kind"] == "accel" else 96.0 * n
    return {"bytes": state, "flops": evals * flops}


def _direct(x, targets, m, eps, potential=False):
    """Softened direct sum, FP64 torch: accelerations (and potentials) of x[targets], G = 1."""
    n, nt = x.shape[0], targets.numel()
    a = torch.zeros(nt, 3, device=x.device, dtype=torch.float64)
    phi = torch.zeros(nt, device=x.device, dtype=torch.float64)
    rows = max(1, min(nt, (1 << 26) // n))
    for b in range(0, nt, rows):
        t = targets[b:b + rows]
        d = [x[:, k][None, :] - x[t, k][:, None] for k in range(3)]
        u = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps * eps).rsqrt_()
        u[torch.arange(t.numel(), device=x.device), t] = 0.0
        phi[b:b + rows] = -m * u.sum(1)
        u = u * u * u
        for k in range(3):
            a[b:b + rows, k] = m * (u * d[k]).sum(1)
    return (a, phi) if potential else a


def _rk4(x, v, m, eps, dt, steps):
    every = torch.arange(x.shape[0], device=x.device)
    for _ in range(steps):
        k1v, k1x = _direct(x, every, m, eps), v
        k2v, k2x = _direct(x + 0.5 * dt * k1x, every, m, eps), v + 0.5 * dt * k1v
        k3v, k3x = _direct(x + 0.5 * dt * k2x, every, m, eps), v + 0.5 * dt * k2v
        k4v, k4x = _direct(x + dt * k3x, every, m, eps), v + dt * k3v
        x = x + dt / 6 * (k1x + 2 * k2x + 2 * k3x + k4x)
        v = v + dt / 6 * (k1v + 2 * k2v + 2 * k3v + k4v)
    return x, v


def exact(case, seed):
    if case["kind"] == "batch":
        sizes = _sizes(case)
        if 4.0 * case["steps"] * float((sizes.astype(np.float64) ** 2).sum()) > EXACT_PAIRS:
            return None
        _, x, v = _batch_particles(case, seed)
        at = np.concatenate([[0], np.cumsum(sizes)])
        parts = [_rk4(x[b:e], v[b:e], 1.0 / (e - b), case["eps"], case["dt"], case["steps"]) for b, e in zip(at[:-1], at[1:])]
        return torch.cat([q[0] for q in parts]), torch.cat([q[1] for q in parts])
    n, m = case["n"], 1.0 / case["n"]
    pairs = float(n) * {"direct": case.get("targets", 0), "accel": n}.get(case["kind"], 4.0 * case.get("steps", 0) * n)
    if pairs > EXACT_PAIRS:
        return None
    x, v = _particles(case, seed)
    if case["kind"] == "direct":
        return _direct(x, torch.from_numpy(_targets(case, seed)).cuda(), m, case["eps"])
    if case["kind"] == "accel":
        return _direct(x, torch.arange(n, device="cuda"), m, case["eps"], case["potential"])
    return _rk4(x, v, m, case["eps"], case["dt"], case["steps"])
