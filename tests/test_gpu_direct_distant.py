"""The FP32 Plummer sum where r^2 comes near the largest float."""
import numpy as np
import pytest

from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dist", [2e18, 2.4e18, 5e18, 9.3e18, 1.2e19, 1.8e19])
@pytest.mark.parametrize("periodic,L", [(False, 1.0), (True, 4.0e19), (True, 2.0 ** 65)])
def test_distant_pairs(cuda, dist, periodic, L):
    from vortexparticlemc_cuda_gb300 import phash as P
    pos = np.array([[0, 0], [dist, 0], [0, dist]], np.float32)
    om = np.array([1.0, 3.0, -2.0], np.float32)
    idx = np.arange(3, dtype=np.int32)
    got = P.direct_velocity_f32(to_dev(pos, cuda), to_dev(om, cuda), P.DIRECT_PLUMMER, tidx=to_dev(idx, cuda), param=0.02,
                                Lx=L, Ly=L, periodic=periodic).cpu().numpy()
    d = pos[:, None].astype(np.float64) - pos[None]
    r2 = (d ** 2).sum(-1)
    c = np.where((r2 > 0) & (r2 < 2.0 ** 128), om / (2 * np.pi * np.where(r2 > 0, r2, 1.0)), 0.0)   # r2 beyond the floats: no term
    t = np.stack([-c * d[..., 1], c * d[..., 0]], -1)
    # a strength over r2 rounds to a multiple of 2^-149 where it is subnormal; otherwise a few roundings
    tol = (np.abs(d) * 2.0 ** -149).sum(1) + 16 * 2.0 ** -24 * np.abs(t).sum(1)
    assert (np.abs(got - t.sum(1)) <= tol).all()


@pytest.mark.parametrize("at", [3e19, np.float32(3e38)])
def test_lone_particle(cuda, at):
    from vortexparticlemc_cuda_gb300 import phash as P
    pos, om = np.full((1, 2), at, np.float32), np.ones(1, np.float32)
    got = P.direct_velocity_f32(to_dev(pos, cuda), to_dev(om, cuda), P.DIRECT_PLUMMER,
                                tidx=to_dev(np.zeros(1, np.int32), cuda), param=0.02, periodic=False)
    assert (got.cpu().numpy() == 0).all()
