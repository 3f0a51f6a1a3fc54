"""Rounding of the plain form's kernels against extended precision: no further
from it than the straightforward evaluation in double precision."""
import numpy as np
import pytest
import scipy.linalg as sl

import __graft_entry__ as g

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def test_solve_of_collocation_like_systems():
    """Forward error of systems with 2 pi on the diagonal and small entries beside it.

    One rounding at C's size a 16-column update, and one a column inside the panel and a step inside a triangle of 64,
    are at order 627 some 36 roundings of a diagonal entry and 37 of a solution entry in each triangle, each 0.29
    units in the last place as a root mean square: 4.7e-16 together, 4.2 u.  The bound is twice that; a sum formed
    in place (two roundings for each of up to 627 columns) comes to 9 u from the diagonal alone.
    """
    n, errs = 627, []
    s = g.load_package().hamsgpu.Solver()
    for seed in range(4):
        rng = np.random.default_rng(seed)
        a = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * (0.05 / np.sqrt(n)) + 2 * np.pi * np.eye(n)
        b = rng.standard_normal((n, 8)) + 1j * rng.standard_normal((n, 8))
        x = s.gesv(a, b)[2]
        f = sl.lu_factor(a)
        y, al = sl.lu_solve(f, b).astype(np.clongdouble), a.astype(np.clongdouble)
        for _ in range(3):
            y = y + sl.lu_solve(f, (b - al @ y).astype(complex))
        errs.append(np.linalg.norm((x - y).astype(complex)) / np.linalg.norm(y.astype(complex)))
    s.close()
    assert np.exp(np.mean(np.log(errs))) <= 8.4 * U, errs


# the last column's diagonal entry so far from its other entries that their quotient leaves the range of doubles
@pytest.mark.parametrize("n", [2, 64, 130])
@pytest.mark.parametrize("diag,entry", [(1e-300, 1e10), (1e300, 1e-10), (1e-300 + 1e-300j, -1e12j)])
def test_graded_triangle(n, diag, entry):
    a = np.eye(n, dtype=complex) * min(1.0, abs(entry))
    a[:-1, -1], a[-1, -1] = entry, diag
    b = np.full((n, 3), a[0, 0] + entry)
    b[-1] = diag
    s = g.load_package().hamsgpu.Solver()
    x, _, info = s.gesv(a, b)[2:]
    s.close()
    # x = 1 throughout; each b was rounded once at |entry| and the entry's product is rounded there again, so rows
    # above the last carry up to 4 units of |entry| / |diagonal| of their own
    bound = np.full(n, 4 * 2 * U * max(1.0, abs(entry)) + 8 * U)
    assert info == 0 and (np.abs(x - 1.0).max(axis=1) <= bound).all()
