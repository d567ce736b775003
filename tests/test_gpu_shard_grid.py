"""The grid of a shard of the targets: the whole run's, and with it the run's sums bit for
bit, unless the library chooses the walk and the shard's samples are too thin for it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def simulation(P, counts, walk=0, qpt=4, **kw):
    n = sum(counts)
    rng = np.random.default_rng(n)
    sim = P.Simulation([P.SimParam(dt=1e-3, seed=5 + i, **kw) for i in range(len(counts))], counts)
    sim.set_tuning(walk, qpt)
    sim.set_particles(torch.from_numpy(rng.random((n, 2)).astype(np.float32)).cuda(),
                      torch.from_numpy((rng.normal(size=n) / n).astype(np.float32)).cuda())
    sim.prepare()
    return sim


# 64^2 particles, 804 of them within h_w, 128 samples of a sign each: boxes ask for 36.7; 6 cells
# a h_w in boxes of 1 / 4 cell hold to 2,643 targets, then 7 in boxes of 1 / 2 cell to 900, then
# pairs on 6 and fewer
DENSE = dict(Nx=64, hwr=16, N1=64, N2=64)


@pytest.mark.parametrize("begin,end,k,qpt", [(0, 4095, 6, 4), (1400, 4050, 6, 4), (0, 2640, 7, 4), (100, 1002, 7, 4),
                                             (0, 898, 6, 6), (5, 55, 2, 6)])   # 6 queries a thread: pair by pair
def test_dense_run(cuda, begin, end, k, qpt):
    from vortexparticlemc_cuda_gb300 import phash as P
    sim = simulation(P, [4096], **DENSE)
    assert sim.tuning()[0] == 6
    whole = sim.velocity(3)[begin:end]
    sim.set_target_range(begin, end)
    assert sim.tuning()[0] == k
    got = sim.velocity(3)[begin:end]
    assert torch.equal(got, whole) == ((k, qpt) == (6, 4))
    assert float((got - whole).norm()) <= 2e-6 * float(whole.norm())
    alone = simulation(P, [4096], k, qpt, **DENSE)
    alone.set_target_range(begin, end)
    assert torch.equal(got, alone.velocity(3)[begin:end])
    alone.close()
    sim.set_target_range(0, 4096)
    assert sim.tuning()[0] == 6 and torch.equal(sim.velocity(3)[begin:end], whole)
    sim.close()


@pytest.mark.parametrize("bits", [32, 64])
def test_thin_bins(cuda, bits):
    """96^2 particles, 32 samples of a sign each, on 35^2 bins: 64 a bin are 2,450 targets."""
    from vortexparticlemc_cuda_gb300 import phash as P
    sim = simulation(P, [96 * 96], Nx=96, hwr=8, N1=16, N2=16)
    sim.set_precision(bits)
    whole = sim.velocity(3)
    for begin, end, k in ((10, 2460, 3), (10, 2459, 2), (0, 1, 2), (0, 9216, 3)):
        sim.set_target_range(begin, end)
        assert sim.tuning()[0] == k
        got = sim.velocity(3)[begin:end]
        assert torch.equal(got, whole[begin:end]) or k == 2
        assert float((got - whole[begin:end]).norm()) <= 2e-6 * float(whole[begin:end].norm())
    sim.close()


@pytest.mark.parametrize("walk,qpt", [(7, 4), (4, 4), (6, 6), (3, 1)])
def test_explicit_walk_is_kept(cuda, walk, qpt):
    from vortexparticlemc_cuda_gb300 import phash as P
    sim = simulation(P, [4096], walk, qpt, **DENSE)
    whole = sim.velocity(3)
    for begin, end in ((0, 4000), (7, 300), (4000, 4096)):
        sim.set_target_range(begin, end)
        assert sim.tuning() == (walk, qpt) and torch.equal(sim.velocity(3)[begin:end], whole[begin:end])
    sim.close()


def test_instances_of_a_range(cuda):
    """A range that takes one instance, a sliver of the next and nothing of the last: steps and positions."""
    from vortexparticlemc_cuda_gb300 import phash as P
    counts = [4096, 1024, 4096]
    sim, ref = simulation(P, counts, **DENSE), simulation(P, counts, **DENSE)
    for s in (sim, ref):
        if s is sim:
            s.set_target_range(0, 4096 + 40)
        s.step(2)
    got, want, start = (s.particles()[0] for s in (sim, ref, simulation(P, counts, **DENSE)))
    assert torch.equal(got[4096 + 40:], start[4096 + 40:])
    # the second step's sources differ from the whole run's in the last two instances only
    assert torch.equal(got[:4096], want[:4096])
    sim.close()
    ref.close()
