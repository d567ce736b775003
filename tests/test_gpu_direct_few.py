"""The FP32 Plummer sum of few targets over many sources, around its chunks of 256 sources."""
import numpy as np
import pytest

from test_gpu_direct_tiles import test_plummer_tiles as tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(255, 3), (256, 1), (257, 200), (513, 512), (5000, 511), (5000, 1024), (5000, 1025)])
@pytest.mark.parametrize("Lx,Ly,periodic", [(1.0, 1.0, True), (0.7, 3.0, True), (1.0, 1.0, False)])
def test_chunks(cuda, n, m, Lx, Ly, periodic):
    tiles(cuda, n, m, Lx, Ly, periodic)
