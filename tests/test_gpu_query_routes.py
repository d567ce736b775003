"""The lines between gathered and binned vorticity queries and between one and two cells a
h_w, with more than 2^17 points, in the forms of the call."""
import pytest

from test_gpu_query_gather import test_forms as forms

pytestmark = pytest.mark.gpu


# cells (2 / h_w)^2: 1 point each in 500^2 is the most that is gathered of any number of points;
# 3 2^16 points the most of 40 a cell; 64 a cell in 50^2 the most that one cell a h_w takes
@pytest.mark.parametrize("n,m,hw", [(900, 249000, 0.004), (900, 251500, 0.004), (700, 3 << 16, 0.02), (700, (3 << 16) + 1, 0.02),
                                    (400, 159000, 0.04), (400, 161500, 0.04)])
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("sign,signed,exclude", [(-1, True, False), (0, True, True)])
def test_lines(cuda, n, m, hw, periodic, sign, signed, exclude):
    forms(cuda, n, m, hw, (1.0, 1.0), periodic, sign, signed, exclude)
