"""Deformed and FP64 queries where the grid has few, some and all of its sub-rows a cell,
against the dense float64 sum."""
import math

import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu


# cells (2 / h_w)^2: 16 sub-rows to 1,000 of them (8 a particle; h_w 1 / 15.8), then fewer, 1 from 16,000 on
@pytest.mark.parametrize("inv", [7.3, 15.7, 16.0, 22.0, 44.0, 63.0, 257.0, 1030.0, 1500.0])
@pytest.mark.parametrize("periodic", [True, False])
def test_sub_rows(cuda, inv, periodic):
    from vortexparticlemc_cuda_gb300 import phash as P
    n, m, hw = 2000, 1500, float(np.float32(1 / inv))
    rng = np.random.default_rng(int(inv))
    side = min(1.0, 30 * hw)                    # a patch across the corner, dense enough to have neighbours
    pos = np.mod(rng.random((n, 2)) * side - (side / 2 if periodic else 0), 1.0).astype(np.float32)
    pts = np.mod(rng.random((m, 2)) * side - (side / 2 if periodic else 0), 1.0).astype(np.float32)
    pos, pts = (np.minimum(v, np.nextafter(np.float32(1), np.float32(0))) for v in (pos, pts))
    om = rng.normal(size=n).astype(np.float32)
    F = np.tile(np.array([1.3, 0.2, 0.0, 1 / 1.3], np.float32), (n, 1))
    p, y, w = to_dev(pos, cuda).double(), to_dev(pts, cuda).double(), to_dev(om, cuda).double()
    d = y[:, None] - p[None]
    if periodic:
        d -= torch.round(d)
    Fi = torch.linalg.inv(torch.tensor(F[0].reshape(2, 2).astype(np.float64), device=cuda))
    args = dict(sign=0, use_signed=True, h_w=hw, periodic=periodic)
    for got, e, eps in ((P.query_vorticity(to_dev(pos, cuda), to_dev(om, cuda), to_dev(pts, cuda), F=to_dev(F, cuda), **args),
                         d @ Fi.T, 2.0 ** -24),
                        (P.query_vorticity_f64(to_dev(pos, cuda), to_dev(om, cuda), to_dev(pts, cuda), **args), d, 2.0 ** -53)):
        q = torch.sqrt((e * e).sum(2)) / hw
        t = torch.clamp(1 - q, min=0.0)
        k = 40 / (7 * math.pi * hw * hw) * torch.where(q <= 0.5, 6 * (q ** 3 - q * q) + 1, 2 * t ** 3)
        size = k @ w.abs() + 40 / (7 * math.pi * hw * hw) * float(w.abs().max())
        # FP32: the differences' rounding (of the period) over h_w and some 60 of a deformed pair and
        # of the sum; FP64: the differences are exact
        tol = (4 * 2.0 ** -23 / hw if eps > 1e-10 else 0.0) + 60 * eps
        assert bool(((got.double() - k @ w).abs() <= tol * size).all())
        assert bool((k > 0).any())
