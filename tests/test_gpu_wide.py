"""The FP64 field on the FP32 pipe against sums in extended precision."""
import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu
Q = np.longdouble


def _field(pos, om, pts, hw, periodic):
    hw = Q(np.float32(hw))
    d = pts[:, None].astype(Q) - pos[None].astype(Q)
    if periodic:
        d -= np.round(d)
    r = np.sqrt((d * d).sum(-1))
    t = np.maximum(1 - r / hw, 0)
    q = r / hw
    w = np.where(q <= 0.5, 6 * (q * q * q - q * q) + 1, 2 * t * t * t)
    w = w * (Q(40) / (7 * Q(np.pi) * hw * hw)) * om[None].astype(Q)
    return w.sum(1), np.abs(w).sum(1)


@pytest.mark.parametrize("n,m,hw,scale", [(1, 3, 0.1, 1.0), (33, 129, 0.2, 1.0), (700, 257, 0.05, 1e-6), (900, 64, 0.3, 1.0),
                                          (500, 40, 0.02, 1e-30), (500, 40, 0.11, 1e30)])
@pytest.mark.parametrize("periodic", [True, False])
def test_query_f64(cuda, n, m, hw, scale, periodic):
    """Weights of any size (the last two take FP64 pairs), points near and across the edges, coincident points."""
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(n + m)
    pos, pts = rng.random((n, 2)).astype(np.float32), rng.random((m, 2)).astype(np.float32)
    pos[: n // 3] *= np.float32(0.02)               # near the origin: differences that need a second float
    pts[: m // 3] *= np.float32(0.02)
    pts[0] = pos[0]
    pts[-1] = (pos[0] + np.float32(0.97)) % np.float32(1) if periodic else pos[-1]
    om = (rng.random(n) * scale + scale * 0.1).astype(np.float32)
    got = P.query_vorticity_f64(to_dev(pos, cuda), to_dev(om, cuda), to_dev(pts, cuda), sign=0, use_signed=True, h_w=hw,
                                periodic=periodic).cpu().numpy()
    want, size = _field(pos, om, pts, hw, periodic)
    # the strengths' two floats (2^-48), pi in FP64 and the result's last roundings
    assert (np.abs(got - want) <= 2.0 ** -47 * size).all()


def test_error_is_below_fp64_arithmetic(cuda):
    """With strengths that are exact, the sums' error stays within the rounding of the result."""
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(2)
    pos, pts = rng.random((2000, 2)).astype(np.float32), rng.random((200, 2)).astype(np.float32)
    hw = 0.125
    om = rng.random(2000).astype(np.float32)
    s = 80.0 / (7.0 * np.pi * hw * hw)
    w = om.astype(np.float64) * s                   # the library's weights: two floats
    w0 = w.astype(np.float32)
    w1 = (w - w0.astype(np.float64)).astype(np.float32)
    got = P.query_vorticity_f64(to_dev(pos, cuda), to_dev(om, cuda), to_dev(pts, cuda), sign=1, h_w=hw).cpu().numpy()
    d = pts[:, None].astype(Q) - pos[None].astype(Q)
    d -= np.round(d)
    q = np.sqrt((d * d).sum(-1)) / Q(hw)
    t = np.maximum(1 - q, 0)
    v = np.where(q <= 0.5, Q(0.5) - 3 * q * q * t, t * t * t) * (w0.astype(Q) + w1.astype(Q))[None]
    want = v.sum(1)
    assert (np.abs(got - want) <= 3 * 2.0 ** -53 * want).all()


def test_items_of_either_size(cuda):
    """A member whose items hold 64 samples alone and 128 in a large ensemble: the same velocities, bit for bit."""
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(8)
    sizes = [64, 300]                     # 1 M and 24 M samples, on either side of 2^24
    prm = [P.SimParam(dt=1e-3, Nx=s, hwr=3, N1=64, N2=64, seed=s) for s in sizes]
    parts = [(rng.random((s * s, 2)).astype(np.float32), (rng.normal(size=s * s) / (s * s)).astype(np.float32)) for s in sizes]

    def velocity(which):
        sim = P.Simulation([prm[i] for i in which], [sizes[i] ** 2 for i in which])
        sim.set_precision(64)
        sim.set_particles(*(to_dev(np.concatenate([parts[i][j] for i in which]), cuda) for j in (0, 1)))
        sim.prepare()
        v = sim.velocity(3)
        sim.close()
        return v

    assert torch.equal(velocity([0, 1])[:64 * 64], velocity([0]))
