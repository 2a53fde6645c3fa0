"""The calls whose speed counts: what a program that uses this library has it do, through the
Python entry points (thin ctypes bindings of the C ABI), from the 64^3 heat configuration to the
512-patch batch.  Sizes are those of the repository's configurations and benchmark or lie between
them, odd and ragged ones included.

    listed()             the cases by name
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs on the GPU and the handles a program keeps
    run(state)           one pass
    work(case)           bytes and operations a pass cannot do without
    exact(case, seed)    the outputs of run() in 64-bit torch, without this library
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

N = __graft_entry__._import_pkg()

L2_BYTES = 129e6  # fields that fit in L2 need HBM once per pass, larger ones once per time step
F64 = torch.float64


def listed():
    return [
        # the plain heat configuration: 64^3, 100 explicit FP64 steps in one call, captured once by
        # the library and replayed (an implicit inner loop, a small patch: launches and latency count)
        dict(name="heat64_small", kind="heat", mode="exact", dtype="f64", nx=64, ny=64, nz=64, steps=100, graph=True,
             dx=1.0, dy=1.0, dz=1.0),
        # the same equation on a stretched mesh (every axis its own spacing), ragged sizes, launched
        # step by step as a program does that works between the steps
        dict(name="heat64_spacing", kind="heat", mode="exact", dtype="f64", nx=203, ny=131, nz=98, steps=4, graph=False,
             dx=0.5, dy=0.8, dz=1.25),
        # the FP64 throughput form at the benchmark's size
        dict(name="heat64_fixed_state", kind="heat", mode="fixed_state", dtype="f64", nx=256, ny=256, nz=256, steps=20,
             graph=False, dx=1.0, dy=1.0, dz=1.0),
        # FP32 storage on an odd, ragged patch wider than 256 cells
        dict(name="heat32_ragged", kind="heat", mode="exact", dtype="f32", nx=323, ny=197, nz=150, steps=10, graph=False,
             dx=1.0, dy=1.0, dz=1.0),
        # the deep fused chain with its box filter and reductions at the benchmark's size
        dict(name="deep", kind="deep", nx=256, ny=256, nz=256),
        # batched patches of uneven sizes (edges 16..96), FP64 and FP32 state
        dict(name="patches64", kind="patches", dtype="f64", count=128, lo=16, hi=96, steps=10),
        dict(name="patches32", kind="patches", dtype="f32", count=512, lo=16, hi=96, steps=20),
        # scalar transport, FP32 storage on a large patch and FP64 on an ordinary, odd one
        dict(name="transport32", kind="transport", dtype="f32", n=320, steps=5),
        dict(name="transport64", kind="transport", dtype="f64", n=127, steps=5),
        # the gradient of a heat run with sqrt(N) checkpoints (forward and reverse sweeps, all FP64)
        dict(name="gradient", kind="gradient", n=128, steps=64, products="f64", forward="f64"),
        # one particle <-> cell exchange: two particles per cell, one of random size and place
        dict(name="particles", kind="particles", nx=128, ny=120, nz=64, np=2000000),
        # nebo_sum, nebo_max and nebo_norm of a small field, read on the host: the diagnostics after
        # a run, the smallest calls there are
        dict(name="reduce_small", kind="reduce", dtype="f64", nx=64, ny=64, nz=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, cells):
    """Three edges in [lo, hi] whose product is at most `cells`."""
    while True:
        n = [_log(rng, lo, hi) for _ in range(3)]
        if n[0] * n[1] * n[2] <= cells:
            return dict(nx=n[0], ny=n[1], nz=n[2])


def draw(rng):
    kind = rng.choice(["heat", "heat", "heat", "deep", "patches", "transport", "gradient", "particles", "reduce"])
    if kind == "heat":
        dtype, mode = rng.choice([("f64", "exact"), ("f64", "exact"), ("f64", "fixed_state"), ("f32", "exact"),
                                  ("f32", "exact")])
        unit = mode != "exact" or rng.random() < 0.6
        sp = [1.0] * 3 if unit else [round(rng.uniform(0.4, 1.6), 3) for _ in range(3)]
        box = _box(rng, 16, 400, 1 << 24)
        most = max(2, min(100, int(8e7 / (box["nx"] * box["ny"] * box["nz"]))))
        return dict(kind=kind, mode=mode, dtype=dtype, **box, steps=_log(rng, 2, most), graph=rng.random() < 0.3,
                    dx=sp[0], dy=sp[1], dz=sp[2])
    if kind == "deep":
        return dict(kind=kind, **_box(rng, 16, 300, 1 << 24))
    if kind == "patches":
        dtype = rng.choice(["f64", "f32"])
        return dict(kind=kind, dtype=dtype, count=_log(rng, 8, 160 if dtype == "f64" else 512), lo=16,
                    hi=rng.randint(48, 96), steps=2 * rng.randint(1, 5 if dtype == "f64" else 10))
    if kind == "transport":
        dtype = rng.choice(["f64", "f32"])
        return dict(kind=kind, dtype=dtype, n=_log(rng, 24, 160 if dtype == "f64" else 320), steps=rng.randint(1, 5))
    if kind == "gradient":
        return dict(kind=kind, n=_log(rng, 16, 128), steps=rng.randint(9, 64), products=rng.choice(["f64", "f64", "f32"]),
                    forward=rng.choice(["f64", "f64", "f32"]))
    if kind == "particles":
        return dict(kind=kind, **_box(rng, 16, 200, 1 << 20), np=_log(rng, 1000, 2000000))
    return dict(kind="reduce", dtype=rng.choice(["f64", "f32"]), **_box(rng, 8, 500, 1 << 25))


# ----------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(gen, shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=gen, device="cuda", dtype=F64) * (hi - lo) + lo


def _bump(gen, n, sigma):
    """A Gaussian bump of amplitude 1 with N(0, 1e-3) noise on the interior (z, y, x)."""
    ax = [torch.arange(m, device="cuda", dtype=F64) + 0.5 - m / 2.0 for m in n]
    r2 = ax[2][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[0][None, None, :] ** 2
    noise = torch.randn(r2.shape, generator=gen, device="cuda", dtype=F64) * 1e-3
    return torch.exp(r2 / (-2.0 * sigma * sigma)) + noise


def _wrap(t, g):
    """The window of an interior with g periodic ghost layers."""
    for d in range(3):
        n = t.shape[d]
        t = torch.cat([t.narrow(d, n - g, g), t, t.narrow(d, 0, g)], dim=d)
    return t.contiguous()


def _size(case):
    return (case["nx"], case["ny"], case["nz"]) if "nx" in case else (case["n"],) * 3


def _heat_inputs(case, seed):
    n, gen = _size(case), _gen(seed)
    lam = _rand(gen, (n[2], n[1], n[0]), 0.5, 1.5)
    T0 = _bump(gen, n, 8.0)
    sp = (case.get("dx", 1.0), case.get("dy", 1.0), case.get("dz", 1.0))
    dt = 0.45 / (float(lam.max()) * sum(1.0 / d ** 2 for d in sp))  # stable; 0.15 / max(lambda) at unit spacing
    if case.get("dtype") == "f32":
        lam, T0 = lam.float(), T0.float()
    return lam, T0, sp, dt


def _field(loc, n, ghost, interior):
    f = N.Field(loc, n, ghost, dtype="f32" if interior.dtype == torch.float32 else "f64")
    f.tensor.copy_(_wrap(interior, ghost))
    return f


def _deep_inputs(case, seed):
    n, gen = _size(case), _gen(seed)
    shape = (n[2] + 2, n[1] + 2, n[0] + 2)
    a, b, c = (_rand(gen, shape, -1.0, 1.0) for _ in range(3))
    pick = torch.rand((n[2], n[1], n[0]), generator=gen, device="cuda") < 0.05
    for d in range(3):
        pick.select(d, 0).fill_(True)
        pick.select(d, -1).fill_(True)
    return a, b, c, pick


def _patch_inputs(case, seed):
    rng, gen = np.random.default_rng(seed), _gen(seed)
    # one mesh per case: a program's patches keep their shapes while their values change
    shapes = np.random.default_rng(7).integers(case["lo"], case["hi"] + 1, size=(case["count"], 3)).astype(np.int32)
    lam = rng.uniform(0.5, 1.5, size=case["count"])
    return shapes, lam, 0.15 / lam, [_bump(gen, [int(v) for v in s], min(s) / 6.0) for s in shapes]


def _transport_inputs(case, seed):
    """phi, u, v, w, lambda on the interior: the velocities are the discrete curl of a vector
    potential of four Fourier modes, so they are divergence free, with |u| <= 1."""
    n, gen, rng = case["n"], _gen(seed), np.random.default_rng(seed)
    ax = torch.arange(n, device="cuda", dtype=F64)
    A = [torch.zeros((n, n, n), device="cuda", dtype=F64) for _ in range(3)]
    for _ in range(4):
        k = rng.integers(1, 4, size=3) * rng.choice([-1, 1], size=3)
        arg = (2 * math.pi / n) * (int(k[0]) * ax[None, None, :] + int(k[1]) * ax[None, :, None]
                                   + int(k[2]) * ax[:, None, None]) + rng.uniform(0, 2 * math.pi)
        s, amp = torch.sin(arg), rng.normal(size=3)
        for d in range(3):
            A[d] += float(amp[d]) * s
    fwd = lambda f, d: torch.roll(f, -1, dims=d) - f  # noqa: E731
    u, v, w = fwd(A[2], 1) - fwd(A[1], 0), fwd(A[0], 0) - fwd(A[2], 2), fwd(A[1], 2) - fwd(A[0], 1)
    top = max(float(q.abs().max()) for q in (u, v, w))
    lam = _rand(gen, (n, n, n), 0.5, 1.5)
    out = [_bump(gen, (n, n, n), n / 8.0), u / top, v / top, w / top, lam]
    if case["dtype"] == "f32":
        out[1:] = [q.float() for q in out[1:]]
    return out, 0.4, 0.05


def _particle_inputs(case, seed):
    n, m, gen = _size(case), case["np"], _gen(seed)
    sp = tuple(1.0 / v for v in n)
    low = tuple(0.5 * d for d in sp)
    size = _rand(gen, (m,), 0.3, 2.5) * min(sp)
    pos = []
    for a in range(3):
        face = low[a] - sp[a] - sp[a] / 2
        pos.append(face + size / 2 + _rand(gen, (m,)) * ((n[a] + 2) * sp[a] - size))
    val, cell = _rand(gen, (m,), 0.5, 2.0), _rand(gen, (n[2] + 2, n[1] + 2, n[0] + 2), -1.0, 1.0)
    return pos, size, val, cell, sp, low


def _reduce_input(case, seed):
    t = _wrap(_bump(_gen(seed), _size(case), 8.0), 1)
    return t.float() if case["dtype"] == "f32" else t


# ----------------------------------------------------------------------------- passes
def prepare(case, seed):
    kind = case["kind"]
    if kind == "heat":
        lam, T0, sp, dt = _heat_inputs(case, seed)
        n = _size(case)
        T = _field("SVol", n, 1, T0)
        return dict(case=case, T=T, tmp=N.Field("SVol", n, 1, dtype=case["dtype"]), lam=_field("SVol", n, 1, lam), sp=sp,
                    dt=dt)
    if kind == "deep":
        a, b, c, pick = _deep_inputs(case, seed)
        n = _size(case)
        out, filt = N.Field("XVol", n, 1), N.Field("XVol", n, 1)
        pts = torch.nonzero(pick).flip(1).to(torch.int32).cpu().numpy()
        words = N.mask_from_points(N.mask_words(out.glob), out.glob, 1, pts)
        return dict(case=case, a=N.Field("SVol", n, 1, tensor=a), b=N.Field("XVol", n, 1, tensor=b),
                    c=N.Field("XVol", n, 1, tensor=c), out=out, filt=filt, words=words,
                    red=torch.zeros(4, device="cuda", dtype=F64))
    if kind == "patches":
        shapes, lam, dt, T0 = _patch_inputs(case, seed)
        ps = N.PatchSet(shapes, lam, dt, case["dtype"])
        ps.autotune()
        arena = ps.arena(0)
        arena.owner = ps  # the view does not own its memory: whoever holds it keeps the patch set
        ps.arena(1).zero_()
        arena.zero_()
        for p, t in enumerate(T0):
            ps.window(0, p)[1:-1, 1:-1, 1:-1].copy_(t)
        ps.fill_ghosts(0)
        return dict(case=case, ps=ps, arena=arena)
    if kind == "transport":
        fields, dt, nu = _transport_inputs(case, seed)
        z = np.zeros((1, 1, 1))
        t = N.Transport(z, z, z, z, z, case["n"], dt, nu, case["dtype"])
        t.phi = _wrap(fields[0], 2)
        t.coef = [_wrap(q, 2) for q in fields[1:]]
        return dict(case=case, t=t)
    if kind == "gradient":
        lam, T0, _, dt = _heat_inputs(case, seed)
        n = case["n"]
        target = T0 + 0.1 * torch.roll(T0, n // 8, dims=2)
        return dict(case=case, dt=dt, f=[_field("SVol", n, 1, q) for q in (T0, lam, target)])
    if kind == "particles":
        pos, size, val, cell, sp, low = _particle_inputs(case, seed)
        n = _size(case)
        return dict(case=case, pos=pos, size=size, val=val, sp=sp, low=low, cell=N.Field("SVol", n, 1, tensor=cell),
                    dest=N.Field("SVol", n, 1), out=torch.empty_like(val))
    t = _reduce_input(case, seed)
    return dict(case=case, f=N.Field("SVol", _size(case), 1, dtype=case["dtype"], tensor=t))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "heat":
        if case["mode"] == "exact":
            N.heat_run(s["T"], s["tmp"], s["lam"], case["steps"], s["dt"], s["sp"], use_graph=case["graph"])
        else:
            N.heat_run_ex(s["T"], s["tmp"], s["lam"], case["steps"], s["dt"], case["mode"], use_graph=case["graph"])
        return s["T"].tensor
    if kind == "deep":
        N.deep_chain(s["a"], s["b"], s["c"], s["words"], s["out"], s["filt"], reductions=s["red"])
        return dict(out=s["out"].tensor, filt=s["filt"].tensor, red=s["red"])
    if kind == "patches":
        which = s["ps"].run(case["steps"], start=0)  # an even number of steps: arena 0 again
        s["ps"].sync(which)
        return s["arena"]
    if kind == "transport":
        s["t"].run(case["steps"])
        return s["t"].phi
    if kind == "gradient":
        T0, lam, target = s["f"]
        J, gT, gl = N.heat_gradient(T0, lam, target, case["steps"], s["dt"], products=case["products"],
                                    forward=case["forward"])
        return dict(J=J, gT=gT.tensor, gl=gl.tensor)
    if kind == "particles":
        N.cell_to_particle(s["cell"], *s["pos"], s["size"], s["out"], s["sp"], s["low"])
        N.particle_to_cell(s["val"], *s["pos"], s["size"], s["dest"], s["sp"], s["low"])
        return dict(particles=s["out"], cells=s["dest"].tensor)
    return [N.nebo_sum(s["f"]), N.nebo_max(s["f"]), N.nebo_norm(s["f"])]


def work(case):
    kind = case["kind"]
    size = 4 if case.get("dtype") == "f32" else 8
    if kind == "patches":
        cells = float(case["count"]) * ((case["lo"] + case["hi"]) / 2.0) ** 3
        fields, state = cells * size, 2
        flops = 8 * cells * case["steps"]
        once = 16 * cells  # the FP64 state, read or written whole at either end
    else:
        n = _size(case)
        cells = float(n[0]) * n[1] * n[2]
    if kind == "heat":
        fields, state, flops, once = cells * size, 3, 16 * cells * case["steps"], 0
    if kind == "transport":
        # per stage: the stencil copy, three velocities, lambda and the FP64 state read, both written
        fields, state, once = cells * size, 0, 0
        per_step = 2 * cells * (6 * size + 20)
        flops = 100 * cells * case["steps"]
        return dict(bytes=per_step * case["steps"] if 5 * fields > L2_BYTES else cells * (16 + 4 * size), flops=flops)
    if kind == "gradient":
        # a forward sweep and a reverse sweep: T, lambda -> T'; T, A, lambda, dJ/dlambda -> A', dJ/dlambda
        flops = 40 * cells * case["steps"]
        return dict(bytes=cells * 8 * (9 * case["steps"] if cells * 48 > L2_BYTES else 5), flops=flops)
    if kind == "deep":
        return dict(bytes=cells * (32.125 + 16), flops=cells * 80)
    if kind == "particles":
        return dict(bytes=cells * 16 + case["np"] * (40.0 + 40.0), flops=case["np"] * 30.0 * 8)
    if kind == "reduce":
        return dict(bytes=cells * size, flops=3 * cells)
    steps = case["steps"] if state * fields > L2_BYTES else 1
    return dict(bytes=state * fields * steps + once, flops=flops)


# ----------------------------------------------------------------------------- in 64 bits
def _heat_rhs(T, k):
    """sum over the axes of (F_high - F_low) with F_low = k_d (T - T[-1]); k: three face arrays."""
    out = torch.zeros_like(T)
    for d in range(3):
        F = k[d] * (T - torch.roll(T, 1, dims=d))
        out += torch.roll(F, -1, dims=d) - F
    return out


def _face_coef(lam, sp):
    return [0.5 * (lam + torch.roll(lam, 1, dims=d)) / sp[2 - d] ** 2 for d in range(3)]


def _exact_deep(case, seed):
    a, b, c, pick = _deep_inputs(case, seed)
    n = _size(case)
    out, filt = torch.zeros_like(a), torch.zeros_like(a)
    g = 0.25 * ((a[:, :, 3:] - a[:, :, 1:-2]) + (a[:, :, 2:-1] - a[:, :, :-3]))
    v = g * torch.exp(b[:, :, 2:-1]) + torch.sin(c[:, :, 2:-1])
    m = torch.zeros(a.shape, dtype=torch.bool, device="cuda")
    m[1:-1, 1:-1, 1:-1] = pick
    out[:, :, 2:-1] = torch.where(m[:, :, 2:-1], torch.zeros_like(v), v)
    f = out
    for d in range(3):
        f = (f.narrow(d, 0, n[2 - d]) + f.narrow(d, 1, n[2 - d])) + f.narrow(d, 2, n[2 - d])
    filt[1:-1, 1:-1, 1:-1] = f / 27.0
    red = torch.stack([_sum(filt), filt.max(), filt.min(), _sum(filt * filt).sqrt()])
    return dict(out=out, filt=filt, red=red)


def _sum(t):
    """The sum of values around 1 in size, to a rounding or two: 2^-26 multiples and the rest apart."""
    t = t.double().reshape(-1)
    hi = torch.round(t * 2.0 ** 26) * 2.0 ** -26
    return hi.sum() + (t - hi).sum()


def _exact_patches(case, seed):
    shapes, lam, dt, T0 = _patch_inputs(case, seed)
    out = []
    for p, T in enumerate(T0):
        if case["dtype"] == "f32":
            T = T.float().double()
        k = float(lam[p]) * float(dt[p])
        for _ in range(case["steps"]):
            lap = -6.0 * T
            for d in range(3):
                lap += torch.roll(T, 1, dims=d) + torch.roll(T, -1, dims=d)
            T = T + k * lap
        w = _wrap(T, 1).reshape(-1)
        out += [w, torch.zeros(-w.numel() % 32, device="cuda", dtype=F64)]  # windows start on 256 bytes
    return torch.cat(out)


def _exact_transport(case, seed):
    (phi, u, v, w, lam), dt, nu = _transport_inputs(case, seed)
    vel = [q.double() for q in (w, v, u)]
    lam = lam.double()

    def rhs(p):
        out = torch.zeros_like(p)
        for d in range(3):
            m1, m2, p1 = torch.roll(p, 1, dims=d), torch.roll(p, 2, dims=d), torch.roll(p, -1, dims=d)
            g4 = (27.0 * (p - m1) - (p1 - m2)) / 24.0
            F = nu * 0.5 * (lam + torch.roll(lam, 1, dims=d)) * g4 - vel[d] * torch.where(vel[d] > 0, m1, p)
            out += torch.roll(F, -1, dims=d) - F
        return out

    for _ in range(case["steps"]):
        one = phi + dt * rhs(phi)
        phi = 0.5 * phi + 0.5 * (one + dt * rhs(one))
    return _wrap(phi, 2)


def _exact_gradient(case, seed):
    lam, T0, _, dt = _heat_inputs(case, seed)
    target = T0 + 0.1 * torch.roll(T0, case["n"] // 8, dims=2)
    k = _face_coef(lam, (1.0, 1.0, 1.0))
    states = [T0]
    for _ in range(case["steps"]):
        states.append(states[-1] + dt * _heat_rhs(states[-1], k))
    A = states.pop() - target
    J = 0.5 * float(_sum(A * A))
    gl = torch.zeros_like(lam)
    for T in reversed(states):
        for d in range(3):
            q = (T - torch.roll(T, 1, dims=d)) * (A - torch.roll(A, 1, dims=d))
            gl -= 0.5 * dt * (q + torch.roll(q, -1, dims=d))
        A = A + dt * _heat_rhs(A, k)
    whole = torch.zeros(tuple(v + 2 for v in gl.shape), device="cuda", dtype=F64)
    whole[1:-1, 1:-1, 1:-1] = gl
    return dict(J=J, gT=_wrap(A, 1), gl=whole)


def _exact_particles(case, seed):
    pos, size, val, cell, sp, low = _particle_inputs(case, seed)
    shape = cell.shape
    cells, vol = torch.zeros_like(cell).reshape(-1), size ** 3
    out = torch.zeros_like(val)
    lo = [p - size / 2 for p in pos]
    face = [low[a] - sp[a] - sp[a] / 2 for a in range(3)]
    first = [((lo[a] - face[a]) / sp[a]).floor().long() for a in range(3)]

    def part(a, i):
        c = first[a] + i
        left = face[a] + c.double() * sp[a]
        w = torch.minimum(left + sp[a], lo[a] + size) - torch.maximum(left, lo[a])
        n = shape[2 - a]
        return c.clamp(0, n - 1), torch.where((c >= 0) & (c < n), w.clamp_min(0.0), torch.zeros_like(w))

    reach = [int(2.5 * min(sp) / sp[a] + 2) for a in range(3)]
    for k in range(reach[2]):
        cz, wz = part(2, k)
        for j in range(reach[1]):
            cy, wy = part(1, j)
            for i in range(reach[0]):
                cx, wx = part(0, i)
                w = wx * wy * wz / vol
                at = cx + shape[2] * (cy + shape[1] * cz)
                out += w * cell.reshape(-1)[at]
                cells.index_add_(0, at, w * val)
    return dict(particles=out, cells=cells.reshape(shape))


def exact(case, seed):
    kind = case["kind"]
    if kind == "heat":
        lam, T, sp, dt = _heat_inputs(case, seed)
        T, k = T.double(), _face_coef(lam.double(), sp)
        for _ in range(case["steps"]):
            T = T + dt * _heat_rhs(T, k)
        return _wrap(T, 1)
    if kind == "deep":
        return _exact_deep(case, seed)
    if kind == "patches":
        return _exact_patches(case, seed)
    if kind == "transport":
        return _exact_transport(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "particles":
        return _exact_particles(case, seed)
    t = _reduce_input(case, seed)
    return [float(_sum(t)), float(t.max()), float(_sum(t.double() * t.double()).sqrt())]
