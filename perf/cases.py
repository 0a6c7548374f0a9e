"""The force-evaluation work this library is timed on.

Every case is one call (or one short run of steps) that a simulation program
makes through the Python binding of libfmmgpu.so, over the sizes and options
the library is used with: force passes on device arrays (3D and 2D, FP32 and
tensor-core M2L, fixed and learned orders, uniform and adaptive targets, with
and without the potential), the host-array call, whole integrator calls, the
batched ensemble and the FP64 direct sum.

A program creates its context once and calls it for every step, so a case's
context is kept from one set of inputs to the next.  The FMM's arithmetic is
FP32 (split precision where it has to be), delivered in FP64 arrays; the
programs here keep the forces, potentials and velocities in FP32.  The direct
sum computes in FP64 and its results stay FP64, as do updated positions.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "nbody-fmm_b200"))
import fmmgpu  # noqa: E402

# what a case holds beside its name; `call` is the entry point
DEFAULTS = dict(call="device", dist="plummer", n=0, dim=3, p=8, leaf=64, m2l="tc", order="fixed", adaptive=0,
                direct_max=-1, chunk=0, run=0, eps=0.0, pot=False, method="se", steps=1, dt=1e-3, targets=0,
                soft="plummer", systems=0, lo=0, hi=0)


def listed():
    return [dict(DEFAULTS, **c) for c in (
        # a small interactive simulation: 500 particles, ten symplectic Euler steps from host arrays; launches
        # and host round trips are all it costs
        dict(name="integrate_se_500", call="integrate", dist="uniform", n=500, p=6, leaf=16, eps=1e-3, method="se",
             steps=10, dt=1e-3),
        # one force pass on a small cluster
        dict(name="pass_plummer_4096", dist="plummer", n=4096),
        # a mid-sized cluster, odd size, tensor cores at a fixed order, with the potential (an energy check)
        dict(name="pass_pot_plummer_65537", dist="plummer", n=65537, p=10, pot=True),
        # a homogeneous box, every interaction pair by the plain FP32 contraction, as the reference evaluates it
        dict(name="pass_uniform_200k_fp32", dist="uniform", n=200000, p=8, leaf=64, m2l="fp32", direct_max=0),
        # the same in the 2D tree at a moderate, odd size, with the potential
        dict(name="pass_2d_disk_50021_fp32", dist="disk", n=50021, dim=2, p=12, leaf=32, m2l="fp32", direct_max=0,
             pot=True),
        # the 2D benchmark configuration
        dict(name="pass_2d_clumps_4m", dist="clumps", n=1 << 22, dim=2, p=16, leaf=32),
        # one RK4 step of the 2^20 Plummer sphere from host arrays
        dict(name="integrate_rk4_plummer_1m", call="integrate", dist="plummer", n=1 << 20, p=8, leaf=64, method="rk4",
             steps=1, dt=1e-4),
        # the call of the README: host arrays, p = 12, learned orders on the tensor cores, uniform targets
        dict(name="host_plummer_1m_learned", call="host", dist="plummer", n=1 << 20, p=12, leaf=64,
             order="learned"),
        # the headline benchmark at the settings its autotuner keeps: 16M clustered mixture, learned orders,
        # adaptive targets
        dict(name="pass_mixture_16m_learned", dist="mixture", n=1 << 24, p=12, leaf=128, order="learned",
             adaptive=64, direct_max=807, chunk=512, run=24),
        # the ensemble benchmark: 256 independent Plummer systems of uneven size
        dict(name="batched_256_systems", call="batched", dist="plummer", systems=256, lo=1024, hi=65536, p=8, leaf=64),
        # the all-pairs update method with the reference's softening
        dict(name="direct_20011", call="direct", dist="uniform", n=20011, soft="naive_ref"),
        # an accuracy check of a large run: FP64 forces on sampled targets
        dict(name="direct_4096_of_1m", call="direct", dist="plummer", n=1 << 20, targets=4096, pot=True),
    )]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "mixture", "2d", "2d", "host", "integrate", "batched", "direct"])
    c = dict(DEFAULTS)
    if kind == "device":  # passes with uniform targets
        dist = rng.choice(["plummer", "uniform", "mixture"])
        c.update(dist=dist, n=_log_int(rng, 1000, 150000 if dist == "mixture" else 400000), p=rng.randint(4, 12),
                 leaf=rng.choice([16, 32, 64, 128]), pot=rng.random() < 0.3, eps=rng.choice([0.0, 0.0, 1e-3]))
        if dist == "uniform" and rng.random() < 0.5:
            c.update(m2l="fp32", direct_max=0)
    elif kind == "mixture":  # adaptive targets on the tensor cores
        # (a box that is not near a cube makes the library sum whole cell pairs directly: mixtures stay small)
        dist = rng.choice(["plummer", "plummer", "mixture"])
        c.update(dist=dist, n=_log_int(rng, 20000, 150000) if dist == "mixture" else _log_int(rng, 200000, 4000000),
                 p=rng.randint(8, 12), leaf=rng.choice([64, 128]), order=rng.choice(["fixed", "learned"]),
                 adaptive=rng.choice([16, 32, 64]), direct_max=rng.choice([-1, 571, 807]))
    elif kind == "2d":
        c.update(dist=rng.choice(["disk", "clumps"]), n=_log_int(rng, 1000, 2000000), dim=2, p=rng.randint(8, 16),
                 leaf=rng.choice([16, 32, 64]), pot=rng.random() < 0.3)
        if c["dist"] == "disk" and rng.random() < 0.5:
            c.update(m2l="fp32", direct_max=0)
    elif kind == "host":
        c.update(call="host", n=_log_int(rng, 1000, 500000), p=rng.choice([8, 10, 12]),
                 order=rng.choice(["fixed", "learned"]), adaptive=rng.choice([0, 32, 64]))
    elif kind == "integrate":
        c.update(call="integrate", dist=rng.choice(["plummer", "uniform"]), n=_log_int(rng, 300, 200000),
                 p=rng.choice([6, 8]), leaf=rng.choice([16, 32, 64]), eps=1e-3, method=rng.choice(["se", "rk4"]),
                 steps=rng.randint(1, 5), dt=rng.choice([1e-3, 1e-4]))
    elif kind == "batched":
        c.update(call="batched", systems=rng.randint(8, 100), lo=1024, hi=32768, p=rng.choice([6, 8]),
                 leaf=rng.choice([32, 64]))
    else:
        c.update(call="direct", dist=rng.choice(["plummer", "uniform", "disk"]), n=_log_int(rng, 1000, 60000),
                 soft=rng.choice(["plummer", "naive_ref"]), pot=rng.random() < 0.5,
                 targets=rng.choice([0, 0, 512, 3000]))
        c["dim"] = 2 if c["dist"] == "disk" else 3
        c["targets"] = min(c["targets"], c["n"])
    return c


# ------------------------------------------------------------------ inputs
# The distributions of fmmgpu.workloads, drawn on the GPU.
def _u(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _plummer(g, n, a=1.0, rmax=20.0):
    u = _u(g, n) * (rmax ** 3 / (rmax * rmax + 1.0) ** 1.5)  # enclosed-mass fraction, cut at rmax
    r = a / torch.sqrt(torch.clamp(u, min=1e-18) ** (-2.0 / 3.0) - 1.0)
    cz, ph = 2.0 * _u(g, n) - 1.0, 2.0 * math.pi * _u(g, n)
    sz = torch.sqrt(1.0 - cz * cz)
    return torch.stack([r * sz * torch.cos(ph), r * sz * torch.sin(ph), r * cz], 1)


def _disk(g, n):
    rad, th = torch.sqrt(_u(g, n)), 2.0 * math.pi * _u(g, n)
    return torch.stack([rad * torch.cos(th), rad * torch.sin(th)], 1)


def _system(g, dist, n):
    mass = torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    if dist == "uniform":
        return _u(g, n, 3), mass
    if dist == "plummer":
        return _plummer(g, n), mass
    if dist == "mixture":
        # the benchmark's 32 Plummer spheres (scale radii log-uniform in [0.01, 0.1], equal mass per sphere): its
        # centres and radii, other particles
        r, parts, k = np.random.default_rng(5), [], 0
        for s in range(32):
            m = n // 32 + (s < n % 32)
            a = float(np.exp(r.uniform(np.log(0.01), np.log(0.1))))
            centre = torch.tensor(r.random(3), device="cuda")
            r.integers(1 << 31)
            parts.append(_plummer(g, m, a) + centre)
            mass[k:k + m] = 1.0 / 32 / m
            k += m
        return torch.cat(parts).contiguous(), mass
    if dist == "disk":
        return _disk(g, n), mass
    # clumps: half uniform in the unit disk, half in 64 Gaussian clumps, log-normal masses
    nu = n // 2
    centres = _disk(g, 64)
    which = torch.randint(0, 64, (n - nu,), generator=g, device="cuda")
    off = torch.randn(n - nu, 2, generator=g, device="cuda", dtype=torch.float64) * 0.005
    mass = torch.exp(0.5 * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    return torch.cat([_disk(g, nu), centres[which] + off]).contiguous(), mass / mass.sum()


def _sizes(case, seed):
    # the ensemble's sizes, log-uniform in [lo, hi]: those of the benchmark, in an order given by the seed
    r = np.random.default_rng(4)
    sizes = np.floor(np.exp(r.uniform(np.log(case["lo"]), np.log(case["hi"]), case["systems"]))).astype(np.int64)
    return np.random.default_rng(seed).permutation(sizes)


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * seed + 17)
    s = dict(case=case)
    if case["call"] == "batched":
        s["offsets"] = np.concatenate([[0], np.cumsum(_sizes(case, seed))]).astype(np.int64)
        parts = [_system(g, case["dist"], int(k)) for k in np.diff(s["offsets"])]
        s["pos"] = torch.cat([p for p, _ in parts]).contiguous()
        s["mass"] = torch.cat([m for _, m in parts]).contiguous()
    else:
        s["pos"], s["mass"] = _system(g, case["dist"], case["n"])
    n = s["pos"].shape[0]
    if case["targets"]:
        s["targets"] = torch.randperm(n, generator=g, device="cuda")[:case["targets"]].contiguous()
    if case["call"] == "integrate":
        # a cluster in motion; the small interactive run starts at rest
        sigma = 0.3 if case["dist"] == "plummer" else 0.0
        s["vel"] = sigma * torch.randn(n, case["dim"], generator=g, device="cuda", dtype=torch.float64)
    return s


# ---------------------------------------------------------------- contexts
# The context of the case at hand and its stream, as a program keeps them for all its steps: a context's calls share
# its workspace, so they go to one stream.
_kept = {}


def _context(case, state):
    key = tuple((k, case[k]) for k in sorted(DEFAULTS))
    if key not in _kept:
        _kept.clear()
        learned = case["order"] == "learned"
        ctx = fmmgpu.Context(
            dim=case["dim"], p=case["p"], leaf_cap=case["leaf"], eps2=case["eps"] ** 2,
            m2l_mode=fmmgpu.FMM_M2L_TC if case["m2l"] == "tc" else fmmgpu.FMM_M2L_FP32,
            order_mode=fmmgpu.FMM_ORDER_LEARNED if learned else fmmgpu.FMM_ORDER_FIXED, order_tol=3e-6,
            judge_samples=512 if learned else 0, judge_every=8, direct_max=case["direct_max"],
            adaptive_leaf=case["adaptive"], p2p_chunk=case["chunk"], m2l_run=case["run"])
        if learned:  # the step before: learned orders budget with its RMS force
            ctx.evaluate_device(case["n"], state["pos"].data_ptr(), state["mass"].data_ptr(),
                                torch.empty_like(state["pos"]).data_ptr())
            ctx.synchronize()
        _kept[key] = ctx, torch.cuda.Stream()
    return _kept[key]


def prepare(case, seed):
    s = _inputs(case, seed)
    torch.cuda.synchronize()
    s["ctx"], s["stream"] = _context(case, s)
    n, dim = s["pos"].shape
    nt = case["targets"] or n
    if case["call"] in ("device", "batched", "direct"):
        s["acc"] = torch.empty(nt, dim, device="cuda", dtype=torch.float64)
        s["pot"] = torch.empty(nt, device="cuda", dtype=torch.float64) if case["pot"] else None
    elif case["call"] == "host":  # page-locked arrays, as a program that calls every step keeps them
        s["pos"], s["mass"] = s["pos"].cpu().pin_memory(), s["mass"].cpu().pin_memory()
        s["acc"] = torch.empty(n, dim, dtype=torch.float64).pin_memory()
        s["acc32"] = torch.empty(n, dim, dtype=torch.float32)
    else:
        s["pos"], s["vel"], s["mass"] = (s[k].cpu().numpy() for k in ("pos", "vel", "mass"))
    torch.cuda.synchronize()
    return s


def _ptr(t):
    return None if t is None else t.data_ptr()


def run(s):
    case, ctx = s["case"], s["ctx"]
    n = len(s["mass"])
    if case["call"] == "integrate":
        method = fmmgpu.FMM_INT_SYMPLECTIC_EULER if case["method"] == "se" else fmmgpu.FMM_INT_RK4
        pos, vel, acc = ctx.integrate(method, case["dt"], case["steps"], s["pos"], s["vel"], s["mass"])
        return {"pos": pos, "vel": vel.astype(np.float32), "acc": acc.astype(np.float32)}
    if case["call"] == "host":
        ctx.evaluate(s["pos"].numpy(), s["mass"].numpy(), out=s["acc"].numpy())
        return {"acc": s["acc32"].copy_(s["acc"])}
    if case["call"] == "batched":
        ctx.evaluate_batched(s["offsets"], _ptr(s["pos"]), _ptr(s["mass"]), _ptr(s["acc"]))
        return {"acc": s["acc"].float()}
    with torch.cuda.stream(s["stream"]):
        st = s["stream"].cuda_stream
        if case["call"] == "direct":
            soft = fmmgpu.FMM_SOFT_NAIVE_REF if case["soft"] == "naive_ref" else fmmgpu.FMM_SOFT_PLUMMER
            ctx.direct_device(n, _ptr(s["pos"]), _ptr(s["mass"]), case["targets"] or n, _ptr(s.get("targets")),
                              _ptr(s["acc"]), _ptr(s["pot"]), soft_mode=soft, stream=st)
            return {"acc": s["acc"]} if s["pot"] is None else {"acc": s["acc"], "pot": s["pot"]}
        ctx.evaluate_device(n, _ptr(s["pos"]), _ptr(s["mass"]), _ptr(s["acc"]), _ptr(s["pot"]), stream=st)
        out = {"acc": s["acc"].float()}
        if s["pot"] is not None:
            out["pot"] = s["pot"].float()
        return out


# -------------------------------------------------------------------- work
def _pass_flops(n, dim, p):
    """One force pass: the all-pairs sum, or a uniform-depth FMM at the leaf
    size that balances its near field (27 or 9 neighbours, 20 flops a pair)
    with its M2L (189 or 27 sources of 2 K^2 flops for every cell)."""
    K = (p + 1) ** 2 if dim == 3 else 2 * p + 1
    near, far = (27 * 20, 189 * 2 * K * K * 8 / 7) if dim == 3 else (9 * 20, 27 * 2 * K * K * 4 / 3)
    return min(20.0 * n * n, n * (2.0 * math.sqrt(near * far) + 8.0 * K))


def work(case):
    dim, n = case["dim"], case["n"]
    if case["call"] == "batched":
        sizes = _sizes(case, 0)
        return {"bytes": 8.0 * float(sizes.sum()) * (2 * dim + 1),
                "flops": float(sum(_pass_flops(int(k), dim, case["p"]) for k in sizes))}
    if case["call"] == "direct":
        nt = case["targets"] or n
        return {"bytes": 8.0 * (n * (dim + 1) + nt * (dim + (1 if case["pot"] else 0))), "flops": 20.0 * n * nt}
    if case["call"] == "integrate":
        passes = case["steps"] * (4 if case["method"] == "rk4" else 1)
        return {"bytes": 8.0 * n * (5 * dim + 1), "flops": passes * _pass_flops(n, dim, case["p"])}
    return {"bytes": 8.0 * n * (2 * dim + 1 + (1 if case["pot"] else 0)), "flops": _pass_flops(n, dim, case["p"])}


# ------------------------------------------------------------------- exact
MOST_PAIRS = 1.5e11  # all-pairs sums up to about ten seconds


def _sum(pos, mass, at, idx, eps2, soft):
    """FP64 all-pairs forces and potentials (G = 1) at positions `at`, the
    particles `idx` of pos themselves."""
    n, dim = pos.shape
    acc, pot = torch.empty_like(at), torch.empty_like(at[:, 0])
    step = max(1, (1 << 25) // n)
    for i in range(0, len(at), step):
        d = [at[i:i + step, k, None] - pos[None, :, k] for k in range(dim)]
        r2 = d[0] * d[0] + eps2
        for k in range(1, dim):
            r2 += d[k] * d[k]
        rows = torch.arange(r2.shape[0], device=r2.device)
        r2[rows, idx[i:i + step]] = math.inf
        if dim == 3 and soft == "naive_ref":
            w = mass / torch.sqrt(r2)
            f = w / (r2 + 1e-4)
        elif dim == 3:
            w = mass / torch.sqrt(r2)
            f = w / r2
        else:
            rr = r2 + 1e-4 if soft == "naive_ref" else r2
            f = mass / rr
            rr[rows, idx[i:i + step]] = 1.0
            w = -0.5 * mass * torch.log(rr)
        pot[i:i + step] = w.sum(1)
        for k in range(dim):
            acc[i:i + step, k] = -(f * d[k]).sum(1)
    return acc, pot


def exact(case, seed):
    passes = case["steps"] * (4 if case["method"] == "rk4" else 1) if case["call"] == "integrate" else 1
    s = _inputs(case, seed)
    pos, mass = s["pos"], s["mass"]
    n = len(mass)
    if case["call"] == "batched":
        off = s["offsets"]
        if float((np.diff(off).astype(float) ** 2).sum()) > MOST_PAIRS:
            return None
        acc = [_sum(pos[a:b], mass[a:b], pos[a:b], torch.arange(b - a, device="cuda"), 0.0, "plummer")[0]
               for a, b in zip(off[:-1], off[1:])]
        return {"acc": torch.cat(acc)}
    if passes * float(n) * (case["targets"] or n) > MOST_PAIRS:
        return None
    idx = s.get("targets", torch.arange(n, device="cuda"))
    eps2 = case["eps"] ** 2
    if case["call"] == "integrate":
        def force(x):
            return _sum(x, mass, x, idx, eps2, "plummer")[0]
        x, v, dt = pos.clone(), s["vel"].clone(), case["dt"]
        for _ in range(case["steps"]):
            if case["method"] == "se":
                a = force(x)
                v = v + dt * a
                x = x + dt * v
            else:
                a1, v1 = force(x), v
                a2, v2 = force(x + 0.5 * dt * v1), v + 0.5 * dt * a1
                a3, v3 = force(x + 0.5 * dt * v2), v + 0.5 * dt * a2
                a4, v4 = force(x + dt * v3), v + dt * a3
                a = a4
                x, v = x + dt / 6 * (v1 + 2 * v2 + 2 * v3 + v4), v + dt / 6 * (a1 + 2 * a2 + 2 * a3 + a4)
        return {"pos": x, "vel": v, "acc": a}
    acc, pot = _sum(pos, mass, pos[idx], idx, eps2, case["soft"])
    return {"acc": acc, "pot": pot} if case["pot"] else {"acc": acc}
