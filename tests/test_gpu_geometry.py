"""Which domains a simulation accepts: those the default walk of two cells a h_w has room
for, whatever number of cells the library would rather take."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ERR_GEOMETRY, ERR_CAPACITY = 7, 8


def particles(n, seed=0):
    rng = np.random.default_rng(seed)
    return (torch.from_numpy(rng.random((n, 2)).astype(np.float32)).cuda(),
            torch.from_numpy((rng.normal(size=n) / n).astype(np.float32)).cuda())


def velocity(n, walk, F=None, **kw):
    from vortexparticlemc_cuda_gb300 import phash as P
    sim = P.Simulation(P.SimParam(dt=1e-3, seed=4, **kw), [n])
    sim.set_tuning(walk, 4)
    if F is not None:
        sim.set_deformation(True)
        sim.set_F(F)
    sim.set_particles(*particles(n))
    sim.prepare()
    out = sim.velocity(1), sim.tuning()[0]
    sim.close()
    return out


# a period of 2.5 to 3 h_w, an open domain of 0.5 to 1 h_w: two cells a h_w fit, one does not
@pytest.mark.parametrize("n,kw", [(64, dict(Nx=8, hwr=3, N1=16, N2=16)), (256, dict(Nx=16, hwr=6, N1=2, N2=2)),
                                  (100, dict(Nx=10, hwr=3.5, N1=64, N2=64)), (121, dict(Nx=11, hwr=4, N1=16, N2=16)),
                                  (4, dict(Nx=2, hwr=3, N1=16, N2=16, periodic=False)),
                                  (1, dict(Nx=2, hwr=4, N1=16, N2=16, periodic=False)),
                                  (1600, dict(Nx=40, hwr=16, N1=1, N2=0))])   # 2.5 h_w, the FP32 h_w a rounding longer
@pytest.mark.parametrize("law", [0, 1])
def test_accepted(cuda, n, kw, law):
    got, k = velocity(n, 0, law=law, **kw)
    want, _ = velocity(n, 2, law=law, **kw)
    assert k == 2 and torch.equal(got, want)


def test_accepted_as_kernels_stretch(cuda):
    """h_w times the largest stretch crosses a third of the period."""
    F = torch.tensor([1.8, 0.0, 0.0, 1 / 1.8], device=cuda).repeat(256, 1)
    got, k = velocity(256, 0, F=F, Nx=16, hwr=3, N1=16, N2=16)
    want, _ = velocity(256, 2, F=F, Nx=16, hwr=3, N1=16, N2=16)
    assert k == 2 and torch.equal(got, want)


# a period of 2.4 h_w and an open domain of h_w / 3 leave no room for two cells a h_w, however
# many samples there are; 6,000^2 cells are too many although one cell a h_w makes 3,000^2
@pytest.mark.parametrize("status,n,kw", [(ERR_GEOMETRY, 576, dict(Nx=24, hwr=10, N1=128, N2=128)),
                                         (ERR_GEOMETRY, 16, dict(Nx=4, hwr=12, N1=1024, N2=1024, periodic=False)),
                                         (ERR_CAPACITY, 100, dict(Nx=3000, hwr=1, N1=16, N2=16))])
def test_refused(cuda, status, n, kw):
    from vortexparticlemc_cuda_gb300 import phash as P
    from vortexparticlemc_cuda_gb300._lib import VpmcError
    with pytest.raises(VpmcError) as e:
        P.Simulation(P.SimParam(dt=1e-3, **kw), [n])
    assert e.value.status == status
