"""Which domains a vorticity query accepts: those the default walk of two cells a h_w has
room for, by either path, against the dense float64 sum."""
import math

import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu
ERR_GEOMETRY, ERR_CAPACITY = 7, 8
GATHERED, BINNED = 500, 140000      # more than 2^17 points, and than 40 a half-support cell, are binned


def inputs(n, m):
    rng = np.random.default_rng(n + m)
    return rng.random((n, 2)).astype(np.float32), rng.normal(size=n).astype(np.float32), rng.random((m, 2)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 4, 100, 300])
@pytest.mark.parametrize("hw,periodic", [(0.34, True), (0.38, True), (0.399, True), (0.4, True), (1.2, False), (1.9, False)])
@pytest.mark.parametrize("m", [GATHERED, BINNED])
def test_accepted(cuda, n, hw, periodic, m):
    from vortexparticlemc_cuda_gb300 import phash as P
    pos, om, pts = inputs(n, m)
    hw = float(np.float32(hw))
    p, w, y = to_dev(pos, cuda), to_dev(om, cuda), to_dev(pts, cuda)
    got = P.query_vorticity(p, w, y, sign=0, use_signed=True, h_w=hw, periodic=periodic).double()
    d = y.double()[:, None] - p.double()[None]
    if periodic:
        d -= torch.round(d)
    q = torch.sqrt((d * d).sum(2)) / hw
    t = torch.clamp(1 - q, min=0.0)
    k = 40 / (7 * math.pi * hw * hw) * torch.where(q <= 0.5, 6 * (q ** 3 - q * q) + 1, 2 * t ** 3)
    # FP32 pairs: the differences' rounding over h_w, a few roundings a term and of the sum
    tol = 4 * 2.0 ** -23 / hw + 40 * 2.0 ** -24
    size = k @ w.double().abs() + float(w.abs().max()) * 40 / (7 * math.pi * hw * hw)
    assert bool(((got - k @ w.double()).abs() <= tol * size).all())


# a period of 2.4 h_w, an open domain of h_w / 3, and 6,000^2 cells, with few and many particles
@pytest.mark.parametrize("n", [10, 3000])
@pytest.mark.parametrize("hw,periodic,status", [(1 / 2.4, True, ERR_GEOMETRY), (3.0, False, ERR_GEOMETRY),
                                                (1 / 3000, True, ERR_CAPACITY)])
@pytest.mark.parametrize("m", [GATHERED, BINNED])
def test_refused(cuda, n, hw, periodic, status, m):
    from vortexparticlemc_cuda_gb300 import phash as P
    from vortexparticlemc_cuda_gb300._lib import VpmcError
    pos, om, pts = inputs(n, m)
    with pytest.raises(VpmcError) as e:
        P.query_vorticity(to_dev(pos, cuda), to_dev(om, cuda), to_dev(pts, cuda), h_w=hw, periodic=periodic)
    assert e.value.status == status
