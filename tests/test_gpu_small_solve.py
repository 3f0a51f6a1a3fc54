"""The plain form's LU and solves below the tensor cores' order: 16-wide panels
with the rows of a CTA on one to four column groups, the FP64 update and
few-column kernels, and the 64-row triangular solves, at the orders where
their tiles, groups and blocks end."""
import numpy as np
import pytest

import __graft_entry__ as g

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


# 16 CTAs x 32, 64, 128, 256 rows are where the panel changes its threads; 16, 64 and 256 the widths of panels,
# triangular steps and blocks; 1024 the first order on the tensor cores
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 255, 257, 511, 512, 513, 1023, 1024, 1025, 2047, 2049])
@pytest.mark.parametrize("nrhs", [1, 9])
def test_plain_solve_backward_error(n, nrhs):
    pkg = g.load_package()
    rng = np.random.default_rng(1000 * n + nrhs)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    s = pkg.hamsgpu.Solver()
    lu, ipiv, x, it, info = s.gesv(a, b)
    s.close()
    assert info == 0 and it == 0
    # partial pivoting: every multiplier at most 1 in |re| + |im| up to the pivot rule's measure
    low = np.tril(lu, -1)
    assert np.abs(low).max(initial=0.0) <= np.sqrt(2.0) * (1 + 8 * EPS)
    pa = a.copy()
    for k, p in enumerate(ipiv):
        pa[[k, p - 1]] = pa[[p - 1, k]]
    lower = low + np.eye(n)
    upper = np.triu(lu)
    # |P A - L U| <= c n eps |L| |U| entry by entry (Higham, Accuracy and Stability, thm 9.3; complex products take
    # up to 2 sqrt(2) eps each, and U12 of the tensor-core orders one refinement step of its explicit inverse)
    bound = 8 * n * EPS * (np.abs(lower) @ np.abs(upper)) + EPS
    assert (np.abs(pa - lower @ upper) <= bound).all()
    # |b - A x| <= c n eps (|L| |U|) |x| after the row exchanges
    res = np.abs(a @ x - b).max()
    scale = (np.abs(lower) @ (np.abs(upper) @ np.abs(x))).max() + np.abs(b).max()
    assert res <= 16 * n * EPS * scale
