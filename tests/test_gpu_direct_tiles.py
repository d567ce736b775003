"""The packed Plummer sum and the row-wise FP64 mollified sum at the edges of
their tiles and of the rules that choose them, against sums in numpy."""
import numpy as np
import pytest

from conftest import to_dev

pytestmark = pytest.mark.gpu


def _plummer(pos, om, tidx, eps, Lx, Ly, periodic):
    """The sum in float64 over the images that the FP32 quotient dx / L chooses; and the sum of the terms' sizes."""
    e2 = float(np.float32(eps) * np.float32(eps))
    d = pos[tidx][:, None, :] - pos[None, :, :]                      # FP32 differences
    if periodic:
        L = np.array([Lx, Ly], np.float32)
        k = np.rint(d / L)                                           # FP32 quotients
        d = d.astype(np.float64) - k.astype(np.float64) * L.astype(np.float64)
    d = d.astype(np.float64)
    c = om.astype(np.float64) / (2 * np.pi) / ((d ** 2).sum(-1) + e2)
    c[np.arange(len(tidx)), tidx] = 0.0
    t = np.stack([-c * d[..., 1], c * d[..., 0]], -1)
    return t.sum(1), np.abs(t).sum(1)


@pytest.mark.parametrize("n,m,Lx,Ly,periodic", [
    (1, 1, 1.0, 1.0, True), (63, 63, 1.0, 1.0, True), (64, 5, 1.0, 1.0, True), (65, 65, 2.0, 0.5, True),
    (511, 511, 1.0, 1.0, False), (513, 513, 0.7, 3.0, True), (4097, 1025, 1.0, 1.0, True),
    (4096, 700, 6.2831855, 0.3, True)])
def test_plummer_tiles(cuda, n, m, Lx, Ly, periodic):
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(n + m)
    L = np.array([Lx, Ly], np.float32)
    if n == 4096:     # a lattice: many pairs exactly (or within rounding of) half a period apart
        g = (np.stack(np.meshgrid(np.arange(64), np.arange(64), indexing="ij"), -1).reshape(-1, 2) + 0.5) / 64
        pos = (g * L).astype(np.float32)
    else:
        pos = (rng.random((n, 2)) * L).astype(np.float32)
    om = rng.normal(size=n).astype(np.float32)
    tidx = rng.permutation(n)[:m].astype(np.int32)
    got = P.direct_velocity_f32(to_dev(pos, cuda), to_dev(om, cuda), P.DIRECT_PLUMMER, tidx=to_dev(tidx, cuda),
                                param=0.02, Lx=Lx, Ly=Ly, periodic=periodic).cpu().numpy()
    want, size = _plummer(pos, om, tidx, 0.02, Lx, Ly, periodic)
    # a term: the difference, image, r2, reciprocal and products round ~8 times (r2 counts twice);
    # the sum: 64 a tile, the tiles of a chunk and the chunks
    tol = (64 + 2 * (n / 64) + 20) * 2.0 ** -24
    # a difference rounded at the scale of the period moves r2 near the core
    tol_d = 2.0 ** -23 * max(Lx, Ly) / 0.02 * 4
    assert (np.abs(got - want) <= (tol + tol_d) * size + 1e-30).all()


@pytest.mark.parametrize("what", ["far", "inf", "huge"])
def test_plummer_general_tiles(cuda, what):
    """Particles many periods away, and strengths that overflow, as the general arithmetic gives them."""
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(3)
    pos = rng.random((300, 2)).astype(np.float32)
    om = rng.normal(size=300).astype(np.float32)
    if what == "far":
        pos[7] += np.float32(3.0e6)
        pos[200] -= np.float32(900.0)
    om[100] = dict(far=om[100], inf=np.inf, huge=2e38)[what]
    tidx = np.arange(300, dtype=np.int32)
    for L in (1.0, 0.7):
        got = P.direct_velocity_f32(to_dev(pos, cuda), to_dev(om, cuda), P.DIRECT_PLUMMER, tidx=to_dev(tidx, cuda),
                                    param=0.02, Lx=L, Ly=L).cpu().numpy()
        if what == "far":
            want, size = _plummer(pos, om, tidx, 0.02, L, L, True)
            assert (np.abs(got - want) <= ((64 + 30) * 2.0 ** -24 + 2.0 ** -23 / 0.02 * 4) * size).all()
        else:   # only the particle itself does not see its own strength
            assert np.isfinite(got[100]).all()
            if what == "inf":
                assert not np.isfinite(np.delete(got, 100, 0)).any()


# periods that are floats take the three-float sums, 0.7 and 1.3 the FP64 rows; a
# core of 0.3 has many images inside it (more than a thread notes); "range" has a
# tile of strengths too far apart for the floats
@pytest.mark.parametrize("n,m,param,Lx,Ly,what", [
    (1, 3, 0.05, 1.0, 1.0, ""), (255, 1, 0.3, 1.0, 1.0, ""), (256, 257, 0.05, 0.7, 1.3, ""), (257, 256, 1e-5, 1.0, 1.0, ""),
    (3000, 100, 0.02, 1.0, 2.0, ""), (600, 40, 0.05, 1.0, 1.0, "range"), (300, 40, 0.05, 1.0, 1.0, "small")])
def test_mollified_periodic(cuda, n, m, param, Lx, Ly, what):
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(n)
    L = np.array([Lx, Ly])
    pos = (rng.random((n, 2)) * L).astype(np.float32)
    om = rng.normal(size=n).astype(np.float32)
    om[::5] = 0.0
    if what == "range":
        om[1] = 1e25
    if what == "small":
        om *= np.float32(1e-33)
    pts = (rng.random((m, 2)) * L).astype(np.float32)
    pts[0] = pos[0]                                   # an image at r = 0
    got = P.direct_velocity(to_dev(pos, cuda), to_dev(om, cuda), pts=to_dev(pts, cuda), param=param, Lx=Lx,
                            Ly=Ly).cpu().numpy()
    u, size = np.zeros((m, 2)), np.zeros((m, 2))
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            d = pts[:, None, :].astype(np.float64) - (pos.astype(np.float64) + np.array([a * Lx, b * Ly]))[None]
            r2 = (d ** 2).sum(-1)
            q = np.minimum(np.sqrt(r2) / param, 1.0)
            inner = 1.2 * q ** 5 - 1.5 * q ** 4 + 0.5 * q ** 2
            outer = q ** 2 - 2 * q ** 3 + 1.5 * q ** 4 - 0.4 * q ** 5 - 0.0125
            mass = np.where(r2 < param ** 2, 80 / 7 * np.where(q <= 0.5, inner, outer), 1.0)
            with np.errstate(divide="ignore", invalid="ignore"):
                k = np.where(r2 > 0, om.astype(np.float64) / (2 * np.pi) * mass / r2, 0.0)
            t = np.stack([-k * d[..., 1], k * d[..., 0]], -1)
            u += t.sum(1)
            size += np.abs(np.sqrt(r2) * k).sum(1)[:, None]
    # ~20 roundings a term, one add a source and chunk; the mass near the edge of the inner pieces cancels ~10 digits' units
    assert (np.abs(got - u) <= (n + 60) * 2.0 ** -52 * size + 1e-300).all()
