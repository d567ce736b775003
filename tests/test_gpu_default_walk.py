"""The walk the library chooses by itself against two cells per h_w."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,hwr,n,k", [(64, 4, 16, 1), (128, 4, 32, 2), (96, 8, 32, 3), (96, 16, 64, 6), (48, 16, 16, None)])
@pytest.mark.parametrize("mode", ["unbiased", "reference", "f64", "deform"])
def test_velocities_agree(cuda, nx, hwr, n, k, mode):
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(nx)
    pos = torch.from_numpy(rng.random((nx * nx, 2)).astype(np.float32)).cuda()
    om = torch.from_numpy((rng.normal(size=nx * nx) / nx ** 2).astype(np.float32)).cuda()
    v = []
    for walk in (0, 2):
        sim = P.Simulation(P.SimParam(dt=1e-3, Nx=nx, hwr=hwr, N1=n, N2=n, law=0 if mode == "reference" else 1, seed=3),
                           [nx * nx])
        sim.set_tuning(walk, 4)
        if mode == "f64":
            sim.set_precision(64)
        if mode == "deform":
            sim.set_deformation(True)
        sim.set_particles(pos, om)
        sim.prepare()
        if walk == 0 and mode != "deform" and k:
            assert sim.tuning()[0] == k
        v.append(sim.velocity(4).double())
        sim.close()
    # the same samples and terms, field sums grouped differently (FP32: 1e-6 of the RMS, as between tunings)
    assert float((v[0] - v[1]).norm() / v[1].norm()) < (1e-7 if mode == "f64" else 2e-6)
