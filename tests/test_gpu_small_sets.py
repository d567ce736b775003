"""The one-CTA builds of small hashes and grids on both sides of their limits."""
import math

import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu


# 16,384 particles and 65,536 cells are the largest the one-CTA hash takes
@pytest.mark.parametrize("n,rx,ry,sub", [(1, 1, 1, False), (31, 2, 1, True), (1024, 128, 128, False),
                                         (1025, 3, 5, True), (11003, 128, 128, False), (16383, 256, 256, True),
                                         (16384, 256, 256, False), (16385, 256, 256, False), (16384, 256, 257, True),
                                         (5000, 1, 65536, False)])
def test_hash_is_a_stable_counting_sort(cuda, n, rx, ry, sub):
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(n + rx)
    pos = (rng.random((2 * n, 2)) * 1.2 - 0.1).astype(np.float32)      # some outside: clamped
    if n != 11003 and n != 16383:
        pos[::7] = pos[0]                                               # a crowded cell: the radix passes
    s = np.sort(rng.permutation(2 * n)[:n]).astype(np.int32) if sub else None
    p = pos[s] if sub else pos[:n]
    f = np.floor(p * np.array([np.float32(rx) / np.float32(1), np.float32(ry) / np.float32(1)], np.float32))
    cell = (np.clip(f[:, 0], 0, rx - 1) * ry + np.clip(f[:, 1], 0, ry - 1)).astype(np.int64)
    h = P.hash_build(rx, ry, 1.0, 1.0, to_dev(pos if sub else p, cuda), None if s is None else to_dev(s, cuda))
    assert np.array_equal(h["vp_cell"].cpu().numpy(), cell)
    assert np.array_equal(h["vp_sort"].cpu().numpy(), np.argsort(cell, kind="stable"))
    acc = np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=rx * ry))[:-1]])
    assert np.array_equal(h["cell_acc"].cpu().numpy(), acc)
    assert not h["cell_num"].any()


@pytest.mark.parametrize("n,m", [(1, 5), (33, 40), (16384, 999), (16385, 1000)])
@pytest.mark.parametrize("sign", [1, -1, 0])
def test_query_on_small_grids(cuda, n, m, sign):
    """Field of a random set against the dense float64 sum (1e-5 of its scale, as elsewhere)."""
    from vortexparticlemc_cuda_gb300 import phash as P
    rng = np.random.default_rng(n)
    hw = float(np.float32(0.07))
    pos, pts = rng.random((n, 2)).astype(np.float32), rng.random((m, 2)).astype(np.float32)
    om = rng.normal(size=n).astype(np.float32)
    om[::9] = 0.0
    got = P.query_vorticity(to_dev(pos, cuda), to_dev(om, cuda), to_dev(pts, cuda), sign=sign, use_signed=sign == 0,
                            h_w=hw)
    w = torch.from_numpy(om).cuda().double()
    w = torch.clamp(w * sign, min=0.0) if sign else w
    d = to_dev(pts, cuda).double()[:, None] - to_dev(pos, cuda).double()[None]
    d -= torch.round(d)
    q = torch.sqrt((d * d).sum(2)) / hw
    t = torch.clamp(1 - q, min=0.0)
    k = 40 / (7 * math.pi * hw * hw) * torch.where(q <= 0.5, 6 * (q ** 3 - q * q) + 1, 2 * t ** 3)
    want, scale = k @ w, float((k @ w.abs()).max())
    assert float((got.double() - want).abs().max()) <= 1e-5 * max(scale, 1e-30)


# 4,096 cells are the most that sort in one counting pass (tiles of 512 to 16,384 members)
@pytest.mark.parametrize("n,rx,ry,sub", [(16385, 64, 64, False), (17000, 1, 1, True), (20000, 2, 1, False), (33000, 1, 3, False),
                                         (40000, 3, 5, True), (60000, 3, 11, False), (70000, 5, 205, True),
                                         (77824, 64, 64, True), (77825, 63, 65, False), (200001, 64, 64, False),
                                         (200001, 17, 241, True), (2500001, 50, 81, False), (3000000, 64, 64, True)])
def test_counting_pass_is_a_stable_counting_sort(cuda, n, rx, ry, sub):
    test_hash_is_a_stable_counting_sort(cuda, n, rx, ry, sub)
