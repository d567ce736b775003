"""Direct and staged placement of the samples on both sides of their limit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# 2^21 samples a chunk is the most that is placed directly; 127^2 and 129^2
# particles with 64 samples a sign are on either side of 128^2.  The shard
# draws a part of the same samples in a chunk of its own.
@pytest.mark.parametrize("nx", [127, 128, 129])
@pytest.mark.parametrize("law", [0, 1])
def test_shards_agree_with_the_whole_run(cuda, nx, law):
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(nx)
    n = nx * nx
    pos = torch.from_numpy(rng.random((n, 2)).astype(np.float32)).cuda()
    om = torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda()

    def run(ranges):
        sim = P.Simulation(P.SimParam(dt=1e-3, Nx=nx, hwr=4, N1=32, N2=32, law=law, seed=5), [n])
        sim.set_particles(pos, om)
        sim.prepare()
        out = torch.empty_like(pos)
        for a, b in ranges:
            sim.set_particles(pos)
            sim.set_step(0)
            sim.set_target_range(a, b)
            sim.step(1)
            out[a:b] = sim.particles()[0][a:b]
        assert sim.step_count == 1
        sim.close()
        return out

    whole = run([(0, n)])
    assert torch.equal(whole, run([(0, 1), (1, 700), (700, n)]))
    assert not torch.equal(whole, pos)


# bins of 260, 576 and 1,040 samples on average (the three sizes of the window assembly),
# spread evenly and clustered, where most of the samples lie in windows that overflow.
# The whole run is staged, its shards are placed directly.
@pytest.mark.parametrize("hwr,walk", [(4, 2), (3, 1), (4, 1)])
@pytest.mark.parametrize("clustered", [False, True])
def test_windows_of_every_size(cuda, hwr, walk, clustered):
    from vortexparticlemc_cuda_gb300 import phash as P
    nx = 129
    n = nx * nx
    rng = np.random.default_rng(hwr + walk)
    p = rng.random((n, 2))
    if clustered:
        p[: n * 4 // 5] = (0.02 * rng.normal(size=(n * 4 // 5, 2))) % 1.0
    pos = torch.from_numpy(p.astype(np.float32)).cuda()
    om = torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda()
    sim = P.Simulation(P.SimParam(dt=1e-3, Nx=nx, hwr=hwr, N1=32, N2=32, seed=5), [n])
    sim.set_tuning(walk, 4)
    sim.set_particles(pos, om)
    sim.prepare()
    whole = sim.velocity(2)
    for a, b in [(0, 5000), (5000, n)]:
        sim.set_target_range(a, b)
        assert torch.equal(whole[a:b], sim.velocity(2)[a:b])
    sim.close()
