"""Boxed field values where a particle lies at a box's centre, a rounding beside it, or
far outside an open domain: sample by sample against the FP64 values of the same samples."""
import numpy as np
import pytest
import torch

from vortexparticlemc_cuda_gb300.inputs import lattice

pytestmark = pytest.mark.gpu


def fields(pos, om, walk, nx, hwr, n, periodic=True):
    """Field values of one pass: boxed, pair by pair, and in FP64."""
    from vortexparticlemc_cuda_gb300 import phash as P
    out = []
    for bits, qpt in ((32, 4), (32, 6), (64, 4)):
        sim = P.Simulation(P.SimParam(dt=1e-3, Nx=nx, hwr=hwr, N1=n, N2=n, law=1, seed=11, periodic=periodic), [len(pos)])
        sim.set_tuning(walk, qpt)
        sim.set_precision(bits)
        sim.set_particles(torch.from_numpy(pos).cuda(), torch.from_numpy(om).cuda())
        sim.prepare()
        sim.velocity(2)
        out.append(sim.read_field(0, len(pos) * 4 * n)[1])
        sim.close()
    return out


def check(pos, om, *args, **kw):
    box, pair, ref = fields(pos, om, *args, **kw)
    assert (box != pair).any()            # the expansions ran
    assert np.isfinite(box).all()
    assert np.abs(box - ref).max() <= 1e-5 * ref.max()   # the bound of every FP32 field value


# boxes of h_w / 14 are this lattice's cells: each holds a particle at its centre, or, by
# the rounding of the two expressions, an ulp beside it
@pytest.mark.parametrize("nx", [56, 98, 448])
def test_lattice_of_the_boxes(cuda, nx):
    om = (np.random.default_rng(nx).normal(size=nx * nx) / nx ** 2).astype(np.float32)
    check(lattice(nx), om, 0, nx, 14.0, 32)


@pytest.mark.parametrize("ulps", [0, 1, 2, 40])
def test_particle_beside_a_centre(cuda, ulps):
    rng = np.random.default_rng(ulps)
    pos, om = rng.random((4096, 2)).astype(np.float32), (rng.normal(size=4096) / 4096).astype(np.float32)
    c = np.float32(0.25) * (np.float32(1) / np.float32(28))      # centre of the first half-cell box of 28 cells
    x = c
    for _ in range(ulps):
        x = np.nextafter(x, np.float32(1))
    pos[17], pos[18] = (x, c), (x, x)
    check(pos, om, 7, 64, 16.0, 64)


@pytest.mark.parametrize("far", [3e19, -1e25])
def test_particle_far_outside(cuda, far):
    rng = np.random.default_rng(3)
    pos, om = rng.random((4096, 2)).astype(np.float32), (rng.normal(size=4096) / 4096).astype(np.float32)
    pos[5], pos[6] = (far, 0.4), (0.6, -far)
    check(pos, om, 7, 64, 16.0, 64, periodic=False)
