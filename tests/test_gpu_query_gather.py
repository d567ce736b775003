"""Vorticity queries gathered point by point and binned, around the rule between
them, in every form the call takes, against the dense float64 sum."""
import math

import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,hw,L", [(1, 7, 0.3, (1.0, 1.0)), (3000, 1, 0.1, (1.0, 1.0)), (3000, 15999, 0.1, (1.0, 1.0)),
                                      (3000, 16001, 0.1, (1.0, 1.0)), (20000, 500, 0.08, (1.0, 0.5)),
                                      (500, 300, 0.02, (0.7, 1.3)), (5000, 700, 0.33, (1.0, 1.0))])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("sign,signed,exclude", [(1, False, False), (-1, False, True), (-1, True, False), (0, True, True),
                                                 (0, False, False)])
def test_forms(cuda, n, m, hw, L, periodic, sign, signed, exclude):
    """16,000 points over 20 x 20 half-supports are 40 a bin, the most that is gathered."""
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(n + m)
    hw = float(np.float32(hw))
    Lf = np.array(L, np.float32)
    pos, pts = (rng.random((n, 2)) * Lf).astype(np.float32), (rng.random((m, 2)) * Lf).astype(np.float32)
    pos, pts = np.minimum(pos, np.nextafter(Lf, np.float32(0))), np.minimum(pts, np.nextafter(Lf, np.float32(0)))
    pts[0] = pos[0]                                        # a coincident pair
    if m > 100:
        pts[1] = (np.nan, 0.1)
        pts[2] = pts[2] + Lf * np.float32(2) if periodic else -pts[2]     # another tile, or outside
        pos[1:3] += Lf * np.float32(1)                     # particles outside the domain
    om = rng.normal(size=n).astype(np.float32)
    om[::7] = 0.0
    got = P.query_vorticity(to_dev(pos, cuda), to_dev(om, cuda), to_dev(pts, cuda), sign=sign, use_signed=signed,
                            exclude_center=exclude, h_w=hw, Lx=L[0], Ly=L[1], periodic=periodic).double()
    p, y, w = to_dev(pos, cuda).double(), to_dev(pts, cuda).double(), to_dev(om, cuda).double()
    if sign:
        w = torch.clamp(w * sign, min=0.0) * (sign if signed else 1)
    elif not signed:
        w = w.abs()
    Lt = torch.tensor(Lf.astype(np.float64), device=cuda)
    want, size = torch.zeros(m, device=cuda, dtype=torch.float64), torch.zeros(m, device=cuda, dtype=torch.float64)
    for i in range(0, m, 4000):
        d = y[i:i + 4000, None] - p[None]
        if periodic:
            d -= torch.round(d / Lt) * Lt
        q = torch.sqrt((d * d).sum(2)) / hw
        t = torch.clamp(1 - q, min=0.0)
        k = 40 / (7 * math.pi * hw * hw) * torch.where(q <= 0.5, 6 * (q ** 3 - q * q) + 1, 2 * t ** 3)
        if exclude:
            k = torch.where(q * hw < 1e-6, torch.zeros_like(k), k)
        want[i:i + 4000], size[i:i + 4000] = k @ w, k @ w.abs()
    out = torch.isnan(y).any(1)
    if not periodic:
        out |= ((y < 0) | (y > Lt)).any(1)
    want[out] = 0.0
    # FP32 pairs: the differences' rounding (of the period) over h_w, a few roundings a term and of the sum
    tol = 4 * 2.0 ** -23 * max(L) * (3 if m > 100 else 1) / hw + 40 * 2.0 ** -24
    scale = float(w.abs().max()) * 40 / (7 * math.pi * hw * hw)
    got = torch.where(torch.isnan(got), torch.full_like(got, 1e30), got)
    assert bool(((got - want).abs() <= tol * (torch.nan_to_num(size) + scale)).all())


# 2^17 points are the most that are gathered whatever their bins hold, with 2^27 pairs at
# most in reach: 2,600 particles within h_w = 0.25 and 52,429 points are 2^27
@pytest.mark.parametrize("n,m,hw,L", [(700, 131072, 0.1, (1.0, 1.0)), (700, 131073, 0.1, (1.0, 1.0)),
                                      (13038, 52000, 0.25, (1.0, 1.0)), (13038, 53000, 0.25, (1.0, 1.0))])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("sign,signed,exclude", [(1, False, False), (0, True, True)])
def test_most_that_is_gathered(cuda, n, m, hw, L, periodic, sign, signed, exclude):
    test_forms(cuda, n, m, hw, L, periodic, sign, signed, exclude)
