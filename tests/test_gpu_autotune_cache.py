"""What the autotuner remembers: a choice made for one precision or share of the targets
is not handed to another."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_precision_and_shard_have_their_own(cuda):
    from vortexparticlemc_cuda_gb300 import phash as P

    def tuned(bits, end):   # (whether the choice was remembered, k)
        nx = 53             # a shape that no other test tunes
        rng = np.random.default_rng(1)
        sim = P.Simulation(P.SimParam(dt=1e-3, Nx=nx, hwr=9, N1=17, N2=18, seed=1), [nx * nx])
        sim.set_precision(bits)
        sim.set_target_range(0, end)
        sim.set_particles(torch.from_numpy(rng.random((nx * nx, 2)).astype(np.float32)).cuda(),
                          torch.from_numpy((rng.normal(size=nx * nx) / nx ** 2).astype(np.float32)).cuda())
        k, q, ms = sim.autotune()
        assert sim.tuning() == (k, q)
        sim.close()
        return ms == -1.0, k, q

    n = 53 * 53
    for case in ((32, n), (64, n), (32, n // 8)):
        first, again = tuned(*case), tuned(*case)
        assert not first[0] and again[0] and first[1:] == again[1:]
