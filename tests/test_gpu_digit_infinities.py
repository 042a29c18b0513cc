"""Infinities and nans in the operands of FP64 digit products: every output of
an affected row or column is the infinity, with its sign, or the nan that the
plain sum of products gives (an infinity times zero and opposite infinities
are nan); all other outputs keep their accuracy, k 2^-50 of the largest
elements' product."""
import numpy as np
import pytest

from test_gpu_dgemm import _gemm

pytestmark = pytest.mark.gpu


def _row(u, b):
    """u . b by plain products and sums."""
    with np.errstate(all="ignore"):
        if not np.iscomplexobj(b):
            return (u[:, None] * b).sum(0)
        re = (u.real[:, None] * b.real).sum(0) + (-u.imag[:, None] * b.imag).sum(0)
        im = (u.real[:, None] * b.imag).sum(0) + (u.imag[:, None] * b.real).sum(0)
        return np.stack([re, im])


def _parts(x):
    return np.stack([x.real, x.imag]) if np.iscomplexobj(x) else x


# output tiles of one CTA each, and shared by a cluster; K that ends inside a step
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,k,n", [(640, 150, 576), (300, 301, 300), (383, 1100, 63)])
def test_infinities_as_in_a_plain_sum(cplx, m, k, n):
    rng = np.random.default_rng(m + k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if cplx:
        a, b = a + 1j * rng.standard_normal((m, k)), b + 1j * rng.standard_normal((k, n))
    inf, nan = np.inf, np.nan
    b[11, 5:9] = 0.0                     # meets the infinities below
    b[:, 10] = 0.0
    a[3] = 0.0
    a[8, 11] = inf
    a[9, 11], a[9, 12] = -inf, inf
    a[10, k - 1] = -inf
    a[11, 4], a[11, 5] = nan, inf
    a[m - 1, 0] = complex(1.0, inf) if cplx else inf
    b[20, n - 1] = inf                   # the last column; row 13 holds an infinity at the same k
    a[13, 20] = -inf
    b[21, 1] = nan
    b[k - 1, 2] = complex(-inf, 2.0) if cplx else -inf
    c, need = _gemm(a, b)
    assert need > 0
    rows, cols = [8, 9, 10, 11, 13, m - 1], [1, 2, n - 1]
    for i in rows:
        got, ref = _parts(c[i]), _row(a[i], b)
        assert np.array_equal(np.isnan(got), np.isnan(ref)), i
        assert np.array_equal(got[~np.isnan(ref)], ref[~np.isnan(ref)]), i
    with np.errstate(all="ignore"):
        for j in cols:
            got, ref = _parts(c[:, j]), _row(b[:, j], np.ascontiguousarray(a.T))
            assert np.array_equal(np.isnan(got), np.isnan(ref)), j
            ok = ~np.isnan(ref)
            assert np.array_equal(got[ok], ref[ok]), j
        plain = a @ b
    fin = np.ones((m, n), bool)
    fin[rows] = False
    fin[:, cols] = False
    lim = np.max(np.abs(a[np.isfinite(a)])) * np.max(np.abs(b[np.isfinite(b)])) * k * 2.0 ** -50
    assert np.all(np.isfinite(c[fin])) and np.max(np.abs(c[fin] - plain[fin])) <= lim
    assert np.all(c[3][fin[3]] == 0.0) and np.all(c[:, 10][fin[:, 10]] == 0.0)
