"""The RBF solves with the kept matrix and with values formed in each product,
a few iterations against MINRES and CG in numpy/torch float64."""
import math

import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu


def _matrix(pos, hw, L, periodic):
    d = pos[:, None, :] - pos[None, :, :]
    if periodic:
        Lt = torch.tensor(L, device=pos.device, dtype=torch.float64)
        d -= torch.round(d / Lt) * Lt
    q = torch.sqrt((d * d).sum(2)) / hw
    t = torch.clamp(1 - q, min=0.0)
    return 40 / (7 * math.pi * hw * hw) * torch.where(q <= 0.5, 6 * (q ** 3 - q * q) + 1, 2 * t ** 3)


def _minres(A, b, x, its):
    r = b - A @ x
    eta = beta = float(r.norm())
    v, v0, w, w0 = r / beta, 0 * r, 0 * r, 0 * r
    c0 = c1 = 1.0
    s0 = s1 = 0.0
    for _ in range(its):
        u = A @ v
        a = float(v @ u)
        u = u - a * v - beta * v0
        n = float(u.norm())
        d = c1 * a - c0 * s1 * beta
        rho = math.hypot(d, n)
        wn = (v - s0 * beta * w0 - (s1 * a + c0 * c1 * beta) * w) / rho
        c0, s0, c1, s1 = c1, s1, d / rho, n / rho
        x = x + c1 * eta * wn
        w0, w, v0, v, eta, beta = w, wn, v, u / n, -s1 * eta, n
    return x


def _cg(A, b, x, its):
    r = b - A @ x
    p, rr = r, float(r @ r)
    for _ in range(its):
        Ap = A @ p
        al = rr / float(p @ Ap)
        x, r = x + al * p, r - al * Ap
        new = float(r @ r)
        p, rr = r + (new / rr) * p, new
    return x


# 17,000 and 24,000 particles inside one support: 3.5 and 6.9 GB of matrix, on either side of what is kept
@pytest.mark.parametrize("n,hw,L,periodic,its", [
    (33, 0.11, (1.0, 1.0), True, 3), (32, 0.11, (1.0, 1.0), True, 1), (1000, 0.1, (1.0, 0.7), True, 3),
    (1023, 0.08, (1.3, 1.0), False, 6), (5000, 0.05, (1.0, 1.0), True, 9), (17000, 0.3, (1.0, 1.0), True, 2),
    (24000, 0.3, (1.0, 1.0), True, 2)])
def test_solves(cuda, n, hw, L, periodic, its):
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(n)
    hw = float(np.float32(hw))
    L = tuple(float(np.float32(v)) for v in L)
    # the crowded cases sit across the corner of the period
    p = rng.random((n, 2)) * L if n < 17000 else np.mod(rng.random((n, 2)) * 0.2 - 0.1, 1.0)
    pos = np.minimum(p, np.nextafter(np.float32(L), np.float32(0))).astype(np.float32)
    if not periodic:
        pos[:3] += np.float32(0.02) * np.array([[1, 0], [0, 1], [1, 1]], np.float32)
    b = rng.normal(size=n).astype(np.float32)
    dp, db = to_dev(pos, cuda), to_dev(b, cuda)
    A = _matrix(dp.double(), hw, L, periodic)
    x0 = db.double() / (40 / (7 * math.pi * hw * hw))
    for solve, want in ((P.minres_rbf, _minres(A, db.double(), x0, its)), (P.cg_rbf, _cg(A, db.double(), x0, its))):
        got, info = solve(dp, db, hw, L[0], L[1], periodic, tol=0.0, max_iter=its, allow_unconverged=True)
        assert info["iters"] == its
        # FP32 output; FP64 rounding of n-term sums grows with the iterations (and with the crowding's scale)
        tol = 2.0 ** -23 + its * n * 2.0 ** -44
        assert float((got.double() - want).abs().max()) <= tol * float(want.abs().max())
        res = float((db.double() - A @ want).norm() / db.double().norm())
        assert abs(info["true_relres"] - res) <= (1e-7 + its * n * 2.0 ** -44) * max(res, 1.0)


def test_one_particle(cuda):
    from vortexparticlemc_cuda_gb300 import phash as P
    pos, b = torch.tensor([[0.3, 0.4]], device=cuda), torch.tensor([2.0], device=cuda)
    for solve in (P.minres_rbf, P.cg_rbf):
        w, info = solve(pos, b, 0.1, tol=1e-6)
        want = 2.0 / (40 / (7 * math.pi * float(np.float32(0.1)) ** 2))
        assert abs(float(w[0]) / want - 1) < 1e-6 and info["iters"] == 0 and info["converged"]
    for solve in (P.minres_rbf, P.cg_rbf):
        w, info = solve(pos, 0 * b, 0.1, tol=1e-6)
        assert float(w[0]) == 0.0 and info["iters"] == 0
