"""Where the library takes the boxes of the local expansions: more samples a box are asked for
the fewer particles lie within h_w."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# boxes of h_w / 14 (7 cells a h_w, halved) on either side of 28 + 7000 / reach samples a box
@pytest.mark.parametrize("hwr", [5.2, 6.5, 8.0, 11.0, 16.0])
@pytest.mark.parametrize("more", [False, True])
def test_line(cuda, hwr, more):
    from vortexparticlemc_cuda_gb300 import phash as P
    nx = 48
    reach = math.pi * hwr ** 2
    h_w = float(np.float32(1) / np.float32(nx) * np.float32(hwr))
    boxes = (2 * math.floor(7 / h_w + 1e-9)) ** 2
    n = (28 + 7000 / reach) * boxes / (2 * nx * nx)            # N1 = N2 with so many a box
    n = math.ceil(n * 1.03) if more else math.floor(n * 0.97)
    rng = np.random.default_rng(n)
    sim = P.Simulation(P.SimParam(dt=1e-3, Nx=nx, hwr=hwr, N1=n, N2=n), [nx * nx])
    sim.set_particles(torch.from_numpy(rng.random((nx * nx, 2)).astype(np.float32)).cuda(),
                      torch.from_numpy((rng.normal(size=nx * nx) / nx ** 2).astype(np.float32)).cuda())
    sim.prepare()
    v = []
    for qpt in (4, 6):                                         # 6 queries a thread: pair by pair
        sim.set_tuning(7, qpt)
        v.append(sim.velocity(1))
    assert torch.equal(*v) == (not more)
    assert float((v[0] - v[1]).norm()) <= 2e-6 * float(v[1].norm())
    sim.close()
