"""The digit kernels of the sliced complex128 products: inner dimensions that
are odd (one entry a thread) and even (two), at the edges of their 32-wide
tiles and of a 256-wide pass, with few and many row blocks (the tiles of a row
block spread over several CTAs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 33, 4900])
@pytest.mark.parametrize("k", [1, 2, 31, 32, 33, 34, 63, 66, 255, 256, 257, 290])
def test_sliced_product_per_entry(pkg, m, k):
    rng = np.random.default_rng(1000 * m + k)
    cx = lambda r, c: np.asfortranarray(rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c)))  # noqa: E731
    a, b, c = cx(m, k), cx(k, 7), cx(m, 7)
    s = pkg.hamsgpu.Solver(precision=pkg.hamsgpu.HG_PREC_FP64)
    got = s.gemm_check(5, a, b, c)
    s.close()
    # eight digits leave 2^-57 of the row's and the column's largest entries, two roundings 2^-53 each; numpy's own
    # sums of up to 290 terms are taken in extended precision
    al, bl = a.astype(np.clongdouble), b.astype(np.clongdouble)
    ref = (c - al @ bl).astype(np.complex128)
    bound = k * np.abs(a).max(1, keepdims=True) * np.abs(b).max(0, keepdims=True) * 2.0 ** -54 + \
        (np.abs(a) @ np.abs(b) + np.abs(c)) * 2.0 ** -51
    assert (np.abs(got - ref) <= bound).all()
