"""Densely sampled steps summed by local expansions of boxes: against the FP64 sums of
the same samples, at box sizes, grids and images where the box walk can go wrong."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def run(P, counts, pos, om, walk, bits, qpt=4, **kw):
    sim = P.Simulation(P.SimParam(dt=1e-3, seed=5, **kw), counts)
    sim.set_tuning(walk, qpt)
    if bits == 64:
        sim.set_precision(64)
    sim.set_particles(pos, om)
    sim.prepare()
    v = sim.velocity(3)
    out = v.double(), sim.tuning()[0]
    sim.close()
    return out


def particles(n, seed, Lx=1.0, Ly=1.0, kind="uniform"):
    rng = np.random.default_rng(seed)
    p = rng.random((n, 2))
    if kind == "clustered":   # most particles in one corner cell, across both edges
        p[: n * 3 // 4] = (rng.normal(size=(n * 3 // 4, 2)) * 0.02) % 1.0
    p = (p * [Lx, Ly]).astype(np.float32)
    w = rng.normal(size=n) / n
    if kind == "positive":    # one sign set empty
        w = np.abs(w)
    return torch.from_numpy(p).cuda(), torch.from_numpy(w.astype(np.float32)).cuda()


# walk cells 4 and 5: boxes of a quarter cell; 7 and 8: half a cell; 3 and below: pairs only.
# 40: h_w 16/40, the periodic grid barely wider than the walk
@pytest.mark.parametrize("nx,hwr,n,walk", [(64, 16, 64, 4), (64, 16, 64, 5), (64, 16, 64, 7), (64, 16, 64, 8), (64, 16, 48, 0),
                                           (40, 16, 192, 7), (50, 11, 160, 7), (33, 13, 224, 6), (64, 16, 33, 7)])
@pytest.mark.parametrize("kind", ["uniform", "clustered", "positive"])
@pytest.mark.parametrize("law,periodic", [(0, 1), (1, 1), (1, 0)])
def test_against_fp64(cuda, nx, hwr, n, walk, kind, law, periodic):
    from vortexparticlemc_cuda_gb300 import phash as P
    pos, om = particles(nx * nx, nx + walk, kind=kind)
    kw = dict(Nx=nx, hwr=hwr, N1=n, N2=n, law=law, periodic=bool(periodic))
    box, _ = run(P, [nx * nx], pos, om, walk, 32, **kw)
    pair, _ = run(P, [nx * nx], pos, om, walk, 32, qpt=6, **kw)
    ref, _ = run(P, [nx * nx], pos, om, walk, 64, **kw)
    assert torch.isfinite(box).all()
    e_box, e_pair = float((box - ref).norm()), float((pair - ref).norm())
    # no further from the FP64 sums than the pairwise FP32 sums are (both share the FP32
    # generation and accumulation, which dominate: a tenth for their rounding)
    assert e_box <= 1.1 * e_pair + 1e-8 * float(ref.norm())


def test_instances_by_either_path(cuda):
    """An ensemble of boxed and pairwise instances: each equals its run alone, bit for bit."""
    from vortexparticlemc_cuda_gb300 import phash as P
    sizes, hwr, n = [64, 24, 96], [16.0, 3.0, 16.0], 64
    parts = [particles(s * s, s) for s in sizes]
    prm = [P.SimParam(dt=1e-3, Nx=s, hwr=h, N1=n, N2=n, law=1, seed=5 + s) for s, h in zip(sizes, hwr)]
    sim = P.Simulation(prm, [s * s for s in sizes])
    sim.set_particles(torch.cat([p for p, _ in parts]), torch.cat([w for _, w in parts]))
    sim.prepare()
    v = sim.velocity(3)
    sim.close()
    at = 0
    for i, s in enumerate(sizes):
        one = P.Simulation([prm[i]], [s * s])
        one.set_particles(*parts[i])
        one.prepare()
        assert torch.equal(one.velocity(3), v[at:at + s * s])
        one.close()
        at += s * s


def test_no_polls_allowed(cuda):
    """A wait limit of 0 ends a boxed pass with the timeout status, as it does a pairwise one."""
    from vortexparticlemc_cuda_gb300 import phash as P
    from vortexparticlemc_cuda_gb300._lib import WAIT_LIMIT_DEFAULT, VpmcError
    pos, om = particles(64 * 64, 1)
    sim = P.Simulation(P.SimParam(dt=1e-3, Nx=64, hwr=16, N1=64, N2=64, seed=5), [64 * 64])
    sim.set_particles(pos, om)
    sim.prepare()
    want = sim.velocity(3)
    sim.ctx.set_wait_limit(0)
    try:
        with pytest.raises(VpmcError):
            sim.velocity(3)
            sim.ctx.sync()
    finally:
        sim.ctx.set_wait_limit(WAIT_LIMIT_DEFAULT)
    assert torch.equal(sim.velocity(3), want)
    sim.close()
