"""Digit products of more K than one launch sums (20480 real, 10240 complex):
later launches add to the first's result.

Bound per output, beside the digit product's own (test_gpu_dgemm.py): each of
the later launches rounds its part and the sum, 2^-53 of at most sum |a||b|.
Checked on a sample of rows and columns in extended precision, and on whole
numbers, exactly."""
import numpy as np
import pytest

from test_gpu_dgemm import _gemm

pytestmark = pytest.mark.gpu


# the last step alone in the second launch; three launches; complex
@pytest.mark.parametrize("cplx,m,k,n", [(False, 640, 20481, 576), (False, 300, 41000, 300), (True, 200, 10300, 150)])
def test_k_over_several_launches(cplx, m, k, n):
    rng = np.random.default_rng(k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if cplx:
        a, b = a + 1j * rng.standard_normal((m, k)), b + 1j * rng.standard_normal((k, n))
    c, need = _gemm(a, b)
    assert need > 0
    rows, cols = [0, 127, 128, m - 1], [0, 63, 64, n - 1]
    kr = 2 * k if cplx else k
    launches = -(-kr // 20480)
    assert launches > 1
    for i in rows:
        for j in cols:
            u, v = a[i], b[:, j]
            if cplx:
                us = (np.stack([u.real, -u.imag]), np.stack([u.imag, u.real]))
                vs = np.stack([v.real, v.imag])
                parts = ((c[i, j].real, us[0], vs), (c[i, j].imag, us[1], vs))
            else:
                parts = ((c[i, j], u[None], v[None]),)
            for got, x, y in parts:
                p = x.astype(np.longdouble) * y.astype(np.longdouble)
                lim = np.abs(x).max() * np.abs(y).max() * (kr * 2.0 ** -58.7 + (kr / 128 + launches) * 2.0 ** -56) \
                    + launches * 2.0 ** -52 * float(np.abs(p).sum())
                assert abs(np.longdouble(got) - p.sum()) <= lim


def test_whole_numbers_over_several_launches():
    rng = np.random.default_rng(1)
    a = rng.integers(-(1 << 15), 1 << 15, (640, 25000)).astype(np.float64)
    b = rng.integers(-(1 << 15), 1 << 15, (25000, 576)).astype(np.float64)
    c, need = _gemm(a, b)
    assert need > 0
    assert np.array_equal(c, a @ b)      # every partial sum is below 2^53
