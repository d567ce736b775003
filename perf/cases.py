"""The work that users of this framework have it do, as measurable cases.

Every case goes through the public `phash` entry points: the spatial hash, the
vorticity query, the RBF strength fit, the two direct sums, the Monte-Carlo
step in its variants (plain, FP64, deformation, ensemble) and the adjoint.
Sizes are those of the repository's own workloads (lattices of 64^2 to 2048^2
particles, h_w of 4 to 16 lattice spacings, 16 to 64 samples per branch).
"""
import math

import numpy as np
import torch

from vortexparticlemc_cuda_gb300 import phash

#: The ensemble's lattice sizes (the batched workload draws its instances from these).
ENSEMBLE_NX = (96, 128, 192, 256, 320, 384)


def listed():
    return [
        # One frame of the reference's spatial-hashing app: ~10-12k particles, 128^2 cells, rebuilt every frame.
        dict(name="hash_frame", kind="hash", n=11003, rsh=128, subset=False),
        # The hash of one sign subset of the largest lattice, on cells of 2 h_w.
        dict(name="hash_subset", kind="hash", n=2048 * 2048, rsh=64, subset=True),
        # The vorticity at a ragged set of probe points (tracers, an output line) in a 512^2 run.
        dict(name="query_probes", kind="query", nx=512, hwr=16.0, m=20011, sign=1, signed=False),
        # The strength fit of one ensemble member from a sampled field (MINRES, the tolerance of the reference's CG).
        dict(name="fit_strengths", kind="fit", nx=192, hwr=8.0, tol=5e-3),
        # The deterministic particle method at the size of the reference's method comparison (40,000 particles).
        dict(name="direct_particles", kind="plummer", nx=200, eps=0.02),
        # The accuracy check of a 512^2 run: the FP64 mollified sum at 4096 particles of it.
        dict(name="direct_f64", kind="mollified", nx=512, hwr=16.0, m=4096),
        # The smallest simulation: 64^2 particles, 16 + 16 samples, one step.
        dict(name="step_small", kind="step", nx=64, hwr=4.0, n1=16, n2=16, k_walk=0, bits=32, deform=False, law=1),
        # The large single instance of the benchmark, with the tuning its autotuner settles on.
        dict(name="step_large", kind="step", nx=2048, hwr=16.0, n1=64, n2=64, k_walk=7, bits=32, deform=False, law=1),
        # The plain FP64 path of the same estimator (the precision study).
        dict(name="step_f64", kind="step", nx=256, hwr=8.0, n1=32, n2=32, k_walk=0, bits=64, deform=False, law=1),
        # The reference's own step: its sampling law, five-point auxiliary targets and the F update.
        dict(name="step_deform", kind="step", nx=256, hwr=8.0, n1=32, n2=32, k_walk=0, bits=32, deform=True, law=0),
        # A batch of independent simulations of uneven sizes in one step.
        dict(name="step_ensemble", kind="ensemble", instances=24, hwr=8.0, n1=32, n2=32),
        # The inverse problem's loop: some steps forward, the loss, and the gradient in positions and strengths.
        dict(name="gradient", kind="gradient", nx=256, hwr=8.0, n1=32, n2=32, steps=4, k_ckpt=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hash", "query", "fit", "plummer", "mollified", "step", "step", "step_f64", "deform", "ensemble",
                       "gradient"])
    if kind == "hash":
        return dict(kind="hash", n=_log_int(rng, 4000, 2048 * 2048), rsh=rng.choice([17, 64, 100, 128, 256]),
                    subset=rng.random() < 0.5)
    if kind == "query":
        sign = rng.choice([1, -1, 0])
        return dict(kind="query", nx=_log_int(rng, 64, 768), hwr=rng.choice([4.0, 8.0, 16.0]),
                    m=_log_int(rng, 1000, 1 << 20), sign=sign, signed=sign == 0)
    if kind == "fit":
        return dict(kind="fit", nx=_log_int(rng, 64, 384), hwr=rng.choice([4.0, 8.0]), tol=5e-3)
    if kind == "plummer":
        return dict(kind="plummer", nx=_log_int(rng, 40, 283), eps=rng.choice([0.01, 0.02, 0.05]))
    if kind == "mollified":
        return dict(kind="mollified", nx=_log_int(rng, 64, 512), hwr=rng.choice([4.0, 8.0, 16.0]),
                    m=_log_int(rng, 500, 4096))
    if kind == "step":
        nx, n = _log_int(rng, 64, 1024), rng.choice([16, 32, 64])
        return dict(kind="step", nx=nx, hwr=rng.choice([4.0, 8.0, 16.0]) if nx >= 96 else 4.0, n1=n, n2=n, k_walk=0,
                    bits=32, deform=False, law=rng.choice([0, 1, 1]))
    if kind == "step_f64":
        return dict(kind="step", nx=_log_int(rng, 64, 256), hwr=rng.choice([4.0, 8.0]), n1=32, n2=32, k_walk=0, bits=64,
                    deform=False, law=1)
    if kind == "deform":
        n = rng.choice([16, 32])
        return dict(kind="step", nx=_log_int(rng, 64, 512), hwr=rng.choice([4.0, 8.0]), n1=n, n2=n, k_walk=0, bits=32,
                    deform=True, law=rng.choice([0, 1]))
    if kind == "ensemble":
        return dict(kind="ensemble", instances=rng.randint(3, 40), hwr=8.0, n1=32, n2=32)
    return dict(kind="gradient", nx=_log_int(rng, 64, 256), hwr=rng.choice([4.0, 8.0]), n1=32, n2=32,
                steps=rng.randint(2, 5), k_ckpt=2)


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _positions(nx, g):
    """Particles some steps into a run: the cell-centred lattice, moved by about a third of its spacing, in [0, 1)^2."""
    a = (torch.arange(nx, device="cuda", dtype=torch.float64) + 0.5) / nx
    p = torch.stack(torch.meshgrid(a, a, indexing="ij"), -1).reshape(-1, 2)
    p = p + torch.randn(p.shape, device="cuda", dtype=torch.float64, generator=g) * (0.35 / nx)
    p = (p - torch.floor(p)).to(torch.float32)
    return torch.where(p >= 1.0, torch.zeros_like(p), p).contiguous()


def _taylor_green(p, g):
    """4 pi sin sin with a phase of its own, at the particles (float64)."""
    ph = torch.rand(2, device="cuda", dtype=torch.float64, generator=g)
    q = 2 * math.pi * (p.to(torch.float64) + ph)
    return 4 * math.pi * torch.sin(q[:, 0]) * torch.sin(q[:, 1])


def _vortices(p, g, k=8):
    """A sum of k Gaussian vortices (amplitudes N(0, 10^2), radii 0.03 to 0.1), nearest periodic image (float64)."""
    c = torch.rand((k, 2), device="cuda", dtype=torch.float64, generator=g)
    a = torch.randn(k, device="cuda", dtype=torch.float64, generator=g) * 10
    r = 0.03 + 0.07 * torch.rand(k, device="cuda", dtype=torch.float64, generator=g)
    w = torch.zeros(p.shape[0], device="cuda", dtype=torch.float64)
    for i in range(k):
        d = p.to(torch.float64) - c[i]
        d = d - torch.round(d)
        w += a[i] * torch.exp(-(d * d).sum(1) / (r[i] * r[i]))
    return w


def _hw(nx, hwr):
    return float(np.float32(np.float32(1.0) / np.float32(nx)) * np.float32(hwr))


def _ensemble_sizes(case):
    rng = np.random.default_rng(case["instances"])
    return [int(v) for v in rng.choice(ENSEMBLE_NX, case["instances"])]


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "hash":
        s["pos"] = torch.rand((case["n"], 2), device="cuda", generator=g)
        s["sub"] = None
        if case["subset"]:
            w = _taylor_green(s["pos"], g)
            top = torch.argsort(w)[case["n"] - case["n"] // 2:]   # the half with the larger vorticity, by index
            s["sub"] = torch.sort(top).values.to(torch.int32).contiguous()
        return s
    if kind == "ensemble":
        sizes = _ensemble_sizes(case)
        pos = [_positions(nx, g) for nx in sizes]
        om = [(_vortices(p, g) / (nx * nx)).to(torch.float32) for p, nx in zip(pos, sizes)]
        prm = [phash.SimParam(dt=1e-3, Nx=nx, hwr=case["hwr"], N1=case["n1"], N2=case["n2"], seed=seed + i)
               for i, nx in enumerate(sizes)]
        sim = phash.Simulation(prm, [nx * nx for nx in sizes])
        sim.set_particles(torch.cat(pos), torch.cat(om))
        sim.prepare()
        s["sim"] = sim
        return s
    nx = case["nx"]
    pos = _positions(nx, g)
    field = _taylor_green(pos, g)
    s["pos"], s["omega"] = pos, (field / (nx * nx)).to(torch.float32)
    if kind == "query":
        s["pts"] = torch.rand((case["m"], 2), device="cuda", generator=g)
        s["h_w"] = _hw(nx, case["hwr"])
    elif kind == "fit":
        s["b"] = (field + _vortices(pos, g, 4)).to(torch.float32)
        s["h_w"] = _hw(nx, case["hwr"])
    elif kind == "plummer":
        s["tidx"] = torch.arange(nx * nx, device="cuda", dtype=torch.int32)
    elif kind == "mollified":
        s["pts"] = pos[torch.randperm(nx * nx, device="cuda", generator=g)[:case["m"]]].contiguous()
        s["h_w"] = _hw(nx, case["hwr"])
    else:
        dt = 2.5e-4 if nx > 1024 else 5e-4 if nx > 256 else 1e-3
        prm = phash.SimParam(dt=dt, Nx=nx, hwr=case["hwr"], N1=case["n1"], N2=case["n2"], law=case.get("law", 1),
                             seed=seed)
        sim = phash.Simulation(prm, [nx * nx])
        s["sim"] = sim
        if kind == "step":
            if case["k_walk"]:
                sim.set_tuning(case["k_walk"], 4)
            if case["bits"] == 64:
                sim.set_precision(64)
            sim.set_particles(pos, s["omega"])
            sim.prepare()
            if case["deform"]:
                sim.set_deformation(True)
        else:
            s["target"] = _positions(nx, g)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "hash":
        return phash.hash_build(case["rsh"], case["rsh"], 1.0, 1.0, state["pos"], state["sub"])
    if kind == "query":
        return phash.query_vorticity(state["pos"], state["omega"], state["pts"], sign=case["sign"],
                                     use_signed=case["signed"], h_w=state["h_w"])
    if kind == "fit":
        omega, info = phash.minres_rbf(state["pos"], state["b"], state["h_w"], tol=case["tol"])
        return dict(omega=omega, iters=info["iters"], true_relres=info["true_relres"])
    if kind == "plummer":
        return phash.direct_velocity_f32(state["pos"], state["omega"], tidx=state["tidx"], param=case["eps"])
    if kind == "mollified":
        return phash.direct_velocity(state["pos"], state["omega"], pts=state["pts"], param=state["h_w"])
    sim = state["sim"]
    if kind == "gradient":
        x0 = state["pos"].clone().requires_grad_(True)
        w = state["omega"].clone().requires_grad_(True)
        xt = phash.trajectory(x0, w, sim, case["steps"], case["k_ckpt"])
        d = xt - state["target"]
        loss = ((d - torch.round(d)) ** 2).mean()
        loss.backward()
        return dict(xt=xt, dx0=x0.grad, domega=w.grad)
    sim.step(1)
    pos, _, vel = sim.particles()
    if kind == "step" and case["deform"]:
        return dict(pos=pos, vel=vel, F=sim.F())
    return dict(pos=pos, vel=vel)


def work(case):
    """What the path cannot do without: the inputs and outputs, and 16 flop for each pair of an evaluation point and a
    particle within its reach (a uniform spread: pi hwr^2 particles, half of them of one sign)."""
    kind = case["kind"]
    if kind == "hash":
        n = case["n"] // 2 if case["subset"] else case["n"]
        return dict(bytes=8 * n + (4 * n if case["subset"] else 0) + 8 * n + 8 * case["rsh"] ** 2, flops=4 * n)
    if kind == "ensemble":
        n = sum(nx * nx for nx in _ensemble_sizes(case))
    else:
        n = case["nx"] ** 2
    if kind == "plummer":
        return dict(bytes=20 * n + 8 * n, flops=14.0 * n * n)
    if kind == "mollified":
        return dict(bytes=12 * n + 24 * case["m"], flops=9 * 10.0 * n * case["m"])
    near = math.pi * case["hwr"] ** 2
    if kind == "query":
        part = 1.0 if case["sign"] == 0 else 0.5
        return dict(bytes=12 * n + 12 * case["m"], flops=16.0 * part * near * case["m"])
    if kind == "fit":  # some 25 products with the matrix; its entries need forming once
        return dict(bytes=16 * n, flops=(16.0 + 25 * 2) * near * n)
    sets = 5 if case.get("deform") else 1
    samples = 2 * n * (case["n1"] + sets * case["n2"])
    one = dict(bytes=12 * n + 24 * n, flops=samples * (8.0 * near + 40))
    if kind == "gradient":  # forward, recompute of a segment, value and gradient, transposed sum
        return dict(bytes=one["bytes"] * case["steps"], flops=4 * one["flops"] * case["steps"])
    return one


# ---------------------------------------------------------------- the same in 64 bits
def _spline(r, hw):
    q = r / hw
    t = torch.clamp(1 - q, min=0.0)
    return 40 / (7 * math.pi * hw * hw) * torch.where(q <= 0.5, 6 * (q * q * q - q * q) + 1, 2 * t * t * t)


def _field(pos, w, pts, hw, wrapped=True):
    """sum_j w_j W(|pts - x_j|) over the nearest images (float64, dense, in blocks of points)."""
    out = torch.empty(pts.shape[0], device="cuda", dtype=torch.float64)
    rows = max(1, (1 << 27) // pos.shape[0])
    for i in range(0, pts.shape[0], rows):
        d = pts[i:i + rows, None, :] - pos[None, :, :]
        if wrapped:
            d -= torch.round(d)
        out[i:i + rows] = _spline(torch.sqrt((d * d).sum(2)), hw) @ w
    return out


def _philox(c0, c1, c2, k0, k1):
    """Philox4x32-10 of counters (c0, c1, c2, 0) (uint64 arrays of 32-bit words) -> four arrays of 32-bit words."""
    lo = np.uint64(0xFFFFFFFF)
    x, y, z, w = c0, c1, np.full_like(c0, c2), np.zeros_like(c0)
    for r in range(10):
        a, b = np.uint64(0xD2511F53) * x, np.uint64(0xCD9E8D57) * z
        ka = np.uint64((k0 + r * 0x9E3779B9) & 0xFFFFFFFF)
        kb = np.uint64((k1 + r * 0xBB67AE85) & 0xFFFFFFFF)
        x, y, z, w = (b >> np.uint64(32)) ^ y ^ ka, b & lo, (a >> np.uint64(32)) ^ w ^ kb, a & lo
    return x, y, z, w


def _mix(v):
    m = (1 << 64) - 1
    v &= m
    v ^= v >> 33
    v = v * 0xFF51AFD7ED558CCD & m
    v ^= v >> 33
    v = v * 0xC4CEB9FE1A85EC53 & m
    v ^= v >> 33
    return v & 0xFFFFFFFF


def _radius_table():
    """Inverse of the spline's radial mass at i / 1024, rounded to float32 (the table is part of the sampling law)."""
    def mass(q):
        q2 = q * q
        inner = 1.2 * q2 * q2 * q - 1.5 * q2 * q2 + 0.5 * q2
        outer = q2 - 2 * q2 * q + 1.5 * q2 * q2 - 0.4 * q2 * q2 * q - 0.0125
        return 80 / 7 * np.where(q <= 0.5, inner, outer)
    u = np.arange(1025) / 1024
    lo, hi = np.zeros(1025), np.ones(1025)
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        below = mass(mid) < u
        lo, hi = np.where(below, mid, lo), np.where(below, hi, mid)
    t = (0.5 * (lo + hi)).astype(np.float32).astype(np.float64)
    t[0], t[-1] = 0.0, 1.0
    return torch.from_numpy(t).cuda()


def _exact_step(case, s, seed):
    """The first step of a plain simulation under the unbiased law: its draws, the field over the 3 x 3 images at each
    sample, the balance-heuristic estimate and the Euler update, in float64."""
    nx, n1, n2 = case["nx"], case["n1"], case["n2"]
    n, q = nx * nx, n1 + n2
    hw = _hw(nx, case["hwr"])
    dt = float(np.float32(2.5e-4 if nx > 1024 else 5e-4 if nx > 256 else 1e-3))
    pos, om = s["pos"].double(), s["omega"].double()
    k0 = _mix(seed * 0x9E3779B97F4A7C15 + 0x632BE59BD9B4E019)
    k1 = _mix(seed ^ 0xA4093822299F31D0)
    table = _radius_table()
    R = math.sqrt(2.0)
    alpha = 1 / (2 * math.pi * R)
    vel = torch.zeros_like(pos)
    t_idx = np.repeat(np.arange(n, dtype=np.uint64), q)
    j_idx = np.tile(np.arange(q, dtype=np.uint64), n)
    first = torch.from_numpy((j_idx < n1)).cuda()
    x = pos.repeat_interleave(q, 0)
    for sign in (0, 1):
        sub = torch.nonzero(om > 0 if sign == 0 else om < 0).reshape(-1)
        if not len(sub):
            continue
        cum = torch.cumsum(om[sub].abs(), 0)
        total = cum[-1]
        words = _philox(j_idx | np.uint64(sign << 31), t_idx, np.uint64(0), k0, k1)
        rx, ry, rz, rw = (torch.from_numpy(v.astype(np.int64)).cuda() for v in words)
        unit = lambda r: ((r >> 8).double() + 0.5) / 16777216.0  # noqa: E731
        pick = torch.searchsorted(cum / total, (rx.double() + 0.5) / 4294967296.0, right=True).clamp(max=len(sub) - 1)
        image = (unit(ry) * 9).floor().clamp(max=8)
        shift = torch.stack([torch.floor(image / 3) - 1, image % 3 - 1], 1)
        f = unit(rz) * 1024
        i0 = f.floor().clamp(max=1023).long()
        rad = (table[i0] + (table[i0 + 1] - table[i0]) * (f - i0)) * hw
        ang = 2 * math.pi * unit(rw)
        y1 = pos[sub[pick]] + shift + rad[:, None] * torch.stack([torch.cos(ang), torch.sin(ang)], 1)
        ang = 2 * math.pi * unit(rx)
        y2 = x + (R * unit(ry))[:, None] * torch.stack([torch.cos(ang), torch.sin(ang)], 1)
        y = torch.where(first[:, None], y1, y2)
        fv = torch.zeros(len(y), device="cuda", dtype=torch.float64)
        src, wt = pos[sub], om[sub].abs()
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                c = src + torch.tensor([a, b], device="cuda", dtype=torch.float64)
                hit = torch.nonzero(((y > c.min(0).values - hw) & (y < c.max(0).values + hw)).all(1)).reshape(-1)
                if len(hit):
                    fv[hit] += _field(c, wt, y[hit], hw, wrapped=False)
        d = x - y
        r2 = (d * d).sum(1)
        r = torch.sqrt(r2)
        w1, w2, c9 = n1 / q, n2 / q, 9 * total
        den = w1 * fv / c9 + torch.where(r < R, w2 * alpha / r, torch.zeros_like(r))
        sc = torch.where(fv > 0, fv / (den * 2 * math.pi * r2), torch.zeros_like(r))
        u = torch.stack([-d[:, 1] * sc, d[:, 0] * sc], 1).reshape(n, q, 2).sum(1) / q
        vel = vel + (u if sign == 0 else -u)
    new = pos + dt * vel
    return dict(pos=new - torch.floor(new), vel=vel)


def _exact_fit(case, s):
    """MINRES on the dense RBF matrix, started at b / W(0), to the same tolerance (float64)."""
    pos, b, hw = s["pos"].double(), s["b"].double(), s["h_w"]
    n = pos.shape[0]
    A = torch.empty((n, n), device="cuda", dtype=torch.float64)
    for i in range(0, n, 1024):
        d = pos[i:i + 1024, None, :] - pos[None, :, :]
        d -= torch.round(d)
        A[i:i + 1024] = _spline(torch.sqrt((d * d).sum(2)), hw)
    x = b / (40 / (7 * math.pi * hw * hw))
    r = b - A @ x
    bnorm, beta = float(b.norm()), float(r.norm())
    v, v_old = r / beta, torch.zeros_like(r)
    w, w_old = torch.zeros_like(r), torch.zeros_like(r)
    c0, c1, s0, s1, eta, its = 1.0, 1.0, 0.0, 0.0, beta, 0
    while its < 5000 and abs(eta) >= case["tol"] * bnorm:
        u = A @ v
        a = float(v @ u)
        u = u - a * v - beta * v_old
        nxt = float(u.norm())
        delta = c1 * a - c0 * s1 * beta
        rho = math.hypot(delta, nxt)
        new = (v - s0 * beta * w_old - (s1 * a + c0 * c1 * beta) * w) / rho
        c0, s0, c1, s1 = c1, s1, delta / rho, nxt / rho
        x = x + c1 * eta * new
        w_old, w, v_old, v = w, new, v, u / nxt
        eta, beta, its = -s1 * eta, nxt, its + 1
    return dict(omega=x, iters=None, true_relres=float((b - A @ x).norm()) / bnorm)


def exact(case, seed):
    kind = case["kind"]
    if kind == "query":
        if case["m"] * case["nx"] ** 2 > 2e10:
            return None
        s = prepare(case, seed)
        w = s["omega"].double()
        if case["sign"]:
            w = torch.clamp(w * case["sign"], min=0.0)
        return _field(s["pos"].double(), w, s["pts"].double(), s["h_w"])
    if kind == "fit":
        return _exact_fit(case, prepare(case, seed)) if case["nx"] <= 200 else None
    if kind == "plummer":
        s = prepare(case, seed)
        p, w, e = s["pos"].double(), s["omega"].double(), float(np.float32(case["eps"]))
        out = torch.empty_like(p)
        for i in range(0, len(p), 1024):
            d = p[i:i + 1024, None, :] - p[None, :, :]
            d -= torch.round(d)
            k = w / (2 * math.pi * ((d * d).sum(2) + e * e))
            out[i:i + 1024] = torch.stack([-(k * d[:, :, 1]).sum(1), (k * d[:, :, 0]).sum(1)], 1)
        return out
    if kind == "mollified":
        s = prepare(case, seed)
        p, w, y, hw = s["pos"].double(), s["omega"].double(), s["pts"].double(), s["h_w"]
        out = torch.zeros((len(y), 2), device="cuda", dtype=torch.float64)
        rows = max(1, (1 << 26) // len(p))
        for i in range(0, len(y), rows):
            for a in (-1, 0, 1):
                for b in (-1, 0, 1):
                    d = y[i:i + rows, None, :] - p[None, :, :]
                    d[..., 0] -= a
                    d[..., 1] -= b
                    r2 = (d * d).sum(2)
                    q = torch.clamp(torch.sqrt(r2) / hw, max=1.0)
                    q2 = q * q
                    inner = 1.2 * q2 * q2 * q - 1.5 * q2 * q2 + 0.5 * q2
                    outer = q2 - 2 * q2 * q + 1.5 * q2 * q2 - 0.4 * q2 * q2 * q - 0.0125
                    m = 80 / 7 * torch.where(q <= 0.5, inner, outer)
                    k = torch.where(r2 > 0, w * m / (2 * math.pi * r2), torch.zeros_like(r2))
                    out[i:i + rows, 0] -= (k * d[..., 1]).sum(1)
                    out[i:i + rows, 1] += (k * d[..., 0]).sum(1)
        return out
    if kind == "step" and case["law"] == 1 and not case["deform"]:
        samples = 2 * case["nx"] ** 2 * (case["n1"] + case["n2"])
        if samples * case["nx"] ** 2 <= 4e9:
            return _exact_step(case, prepare(case, seed), seed)
    # whole numbers (hash), and estimates whose draws and pairs are too many to repeat densely
    return None
