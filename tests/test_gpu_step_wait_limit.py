"""A step whose evaluation gives up leaves the particles where they are, and the run goes
on from there."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,hwr,n,k", [("pairs", 4, 16, 3), ("pairs", 4, 16, 0), ("boxes", 16, 64, 7), ("tensor", 4, 16, 3),
                                          ("f64", 4, 16, 0), ("deform", 4, 16, 0)])
@pytest.mark.parametrize("graph", [False, True])
def test_particles_stay(cuda, mode, hwr, n, k, graph):
    from vortexparticlemc_cuda_gb300 import phash as P
    from vortexparticlemc_cuda_gb300._lib import WAIT_LIMIT_DEFAULT, VpmcError
    rng = np.random.default_rng(2)
    sim = P.Simulation(P.SimParam(dt=1e-2, Nx=64, hwr=hwr, N1=n, N2=n, seed=5), [4096])
    sim.set_tuning(k, 1 if mode == "tensor" else 4)
    if mode == "f64":
        sim.set_precision(64)
    if mode == "deform":
        sim.set_deformation(True)
    sim.set_particles(torch.from_numpy(rng.random((4096, 2)).astype(np.float32)).cuda(),
                      torch.from_numpy((rng.normal(size=4096) / 4096).astype(np.float32)).cuda())
    sim.prepare()
    sim.step(1, use_graph=False)
    want = sim.particles()[0]
    sim.ctx.set_wait_limit(0)
    try:
        for _ in range(2):
            with pytest.raises(VpmcError) as e:
                sim.step(1, use_graph=graph)
            assert e.value.status == 5   # VPMC_ERR_TIMEOUT
    finally:
        sim.ctx.set_wait_limit(WAIT_LIMIT_DEFAULT)
    assert torch.equal(sim.particles()[0], want)
    if not graph:   # (a captured step keeps the limit it was captured with)
        sim.step(1, use_graph=False)
        assert not torch.equal(sim.particles()[0], want)
    sim.close()
