"""Entries of the RBF matrix one by one: the residual of two particles, of which one has a
right-hand side of 1, is the spline's value at their distance, in FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def around(v, n=3):
    out, lo, hi = [np.float32(v)], np.float32(v), np.float32(v)
    for _ in range(n):
        lo, hi = np.nextafter(lo, np.float32(0)), np.nextafter(hi, np.float32(1))
        out += [lo, hi]
    return out


@pytest.mark.parametrize("hw", [0.25, 0.11, 0.3])
@pytest.mark.parametrize("solver", ["cg_rbf", "minres_rbf"])
def test_against_extended_precision(cuda, hw, solver):
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(7)
    h = np.float32(hw)
    # nothing, distances whose squares leave the estimate's range, and the spline's pieces and knots
    ds = [(0.0, 0.0), (1e-45, 0.0), (3e-39, 1e-38), (1e-30, 0.0), (2e-20, 1e-19), (1e-10, 0.0)]
    ds += [(v, 0.0) for r in (h / 2, h, h / 4, 0.9 * h) for v in around(r)]
    ds += [(0.6 * v, 0.8 * v) for r in (h / 2, h) for v in around(r)]
    ds += list(rng.uniform(-0.72, 0.72, (60, 2)) * hw)
    b = torch.tensor([1.0, 0.0], device="cuda")
    for dx, dy in ds:
        d = np.array([dx, dy], np.float32)
        pos = np.stack([np.zeros(2, np.float32), d]) + (np.float32(0.5) if min(d) < 0 else np.float32(0))
        got = getattr(P, solver)(torch.from_numpy(pos).cuda(), b, float(h), tol=0.0, max_iter=0,
                                 allow_unconverged=True)[1]["true_relres"]
        e = (pos[1].astype(np.longdouble) - pos[0].astype(np.longdouble))
        q = np.sqrt((e * e).sum()) / np.longdouble(h)
        t = max(1 - q, np.longdouble(0))
        want = 6 * (q ** 3 - q ** 2) + 1 if q <= 0.5 else 2 * t ** 3
        slope = q * (12 * q - 18 * q * q) if q <= 0.5 else q * 6 * t * t    # |dW / dq| q
        # q: its square, root and quotient round; W and the residual's norm a few times more; and
        # the other component, 1 - W(0) (1 / W(0)), is a rounding instead of 0
        tol = 3 * U * slope + 16 * U * want + 4 * U * (want < 1e-6) + 2 * U
        assert abs(got - want) <= tol, (d, got, want)
