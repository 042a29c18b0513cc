"""FP64 products by exact digit products on the tensor cores (dmrg_gemm with
a workspace) against extended-precision sums.

Error bound per output, from the splitting: with s_a, s_b the powers of two
above the largest element of the row of A and column of B (at most twice
it), every product errs by the two operands' rounding (2^-64 s_a s_b each)
and the digit pairs of order 8 and beyond (7 pairs of at most 2^14 units of
2^-78 s_a s_b, and smaller), together below 2^-60.7 s_a s_b, i.e. 2^-58.7
max|a| max|b|; every run of at least 128 products by its last place, 2^-63
s_a s_b (with random digits the sums of order 6 stay far below 2^24, so the
tensor core adds them exactly), for which 2^-56 max|a| max|b| leaves room;
the result by its rounding, 2^-53 |c|.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gemm(a, b):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    cplx = np.iscomplexobj(a)
    dt = _lib.COMPLEX128 if cplx else _lib.REAL64
    (m, k), n = a.shape, b.shape[1]
    A, B = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
    C = torch.full((m, n), 7.0, dtype=A.dtype, device="cuda")
    need = lib.dmrg_gemm_workspace_bytes(dt, _lib.PREC_FP64, m, k, n)
    w = torch.empty(max(int(need), 256), dtype=torch.uint8, device="cuda")
    _lib.check("dmrg_gemm", lib.dmrg_gemm(dt, _lib.PREC_FP64, m, k, n, A.data_ptr(), B.data_ptr(), C.data_ptr(),
                                          w.data_ptr(), w.numel(),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return C.cpu().numpy(), int(need)


def _exact(a, b):
    if np.iscomplexobj(a):
        r = np.matmul(a.real.astype(np.longdouble), b.real.astype(np.longdouble)) \
            - np.matmul(a.imag.astype(np.longdouble), b.imag.astype(np.longdouble))
        i = np.matmul(a.real.astype(np.longdouble), b.imag.astype(np.longdouble)) \
            + np.matmul(a.imag.astype(np.longdouble), b.real.astype(np.longdouble))
        return r, i
    return np.matmul(a.astype(np.longdouble), b.astype(np.longdouble)), None


def _check(a, b):
    c, need = _gemm(a, b)
    assert need > 0, "shape not routed to the digit product"
    er, ei = _exact(a, b)
    k = a.shape[1] * (2 if np.iscomplexobj(a) else 1)
    ma = np.maximum(np.abs(a.real), np.abs(a.imag)).max(axis=1)
    mb = np.maximum(np.abs(b.real), np.abs(b.imag)).max(axis=0)
    bound = np.outer(ma, mb) * (k * 2.0 ** -58.7 + (k / 128 + 1) * 2.0 ** -56)
    for got, ex in ((c.real, er),) + (((c.imag, ei),) if ei is not None else ()):
        err = np.abs(got.astype(np.longdouble) - ex)
        lim = bound + 2.0 ** -53 * np.abs(ex)
        assert np.all(err <= lim), float(np.max(err / np.maximum(lim, 1e-300)))


def _graded(rng, r, c, cplx):
    x = rng.standard_normal((r, c)) * np.exp(rng.uniform(-12, 12, (r, 1))) * np.exp(-rng.uniform(0, 9, (1, c)))
    if cplx:
        x = x + 1j * rng.standard_normal((r, c)) * np.abs(x)
    return np.ascontiguousarray(x)


# edges of the 128 x 64 tile, of the K step (16), of the run (128) and of the stage ring
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,k,n", [(640, 128, 576), (641, 129, 577), (639, 111, 575), (1200, 16, 1216),
                                   (385, 1100, 321), (700, 300, 450)])
def test_digit_product_matches_extended_precision(m, k, n, cplx):
    rng = np.random.default_rng(m * 1000 + k)
    _check(_graded(rng, m, k, cplx), _graded(rng, k, n, cplx))


def test_digit_product_is_exact_at_the_digit_extremes():
    """All-ones significands of one sign drive every order's accumulator to
    its largest value; integers below 2^53 whose sums fit FP64 come out
    exactly."""
    k = 640
    x = np.nextafter(1.0, 0.0)
    a = np.full((640, k), x)
    b = np.full((k, 576), x)
    c, need = _gemm(a, b)
    assert need > 0
    exact = np.matmul(a[:1].astype(np.longdouble), b[:, :1].astype(np.longdouble))[0, 0]
    assert np.all(np.abs(c.astype(np.longdouble) - exact) <= 2.0 ** -53 * exact)
    rng = np.random.default_rng(3)
    ai = rng.integers(-(1 << 21), 1 << 21, (600, k)).astype(np.float64)
    bi = rng.integers(-(1 << 21), 1 << 21, (k, 640)).astype(np.float64)
    c, _ = _gemm(ai, bi)
    assert np.array_equal(c, (ai.astype(np.int64) @ bi.astype(np.int64)).astype(np.float64))


def test_digit_product_special_values():
    """Zero rows, subnormals, huge and tiny rows, and non-finite elements
    (whose row or column becomes non-finite, as in a plain product)."""
    rng = np.random.default_rng(9)
    a, b = rng.standard_normal((640, 150)), rng.standard_normal((150, 576))
    a[3] = 0.0
    a[4] *= 1e300
    a[5] *= 1e-300
    b[:, 6] *= 1e-200
    a[7] = 5e-324 * rng.integers(-3, 4, 150)
    a[8, 11] = np.inf
    b[9, 12] = np.nan
    c, need = _gemm(a, b)
    assert need > 0
    with np.errstate(all="ignore"):
        # extended precision: FP64 would round every product of the subnormal row
        ref = _exact(a, b)[0]
    fin = np.isfinite(ref)
    assert not np.isfinite(c[8]).any() and not np.isfinite(c[:, 12]).any()
    fin[8] = False
    fin[:, 12] = False
    scale = np.abs(np.where(np.isfinite(a), a, 0)).max(1)[:, None] * np.abs(np.where(np.isfinite(b), b, 0)).max(0)
    assert np.all(np.abs(c - ref)[fin] <= (150 * 2.0 ** -52 * scale + 1e-323)[fin])
    assert np.all(c[3][fin[3]] == 0.0)


# few output tiles: clusters of 2, 4 and 8 CTAs share a tile's K steps, at the
# first and last tile counts of each (76, 36, 15 tiles) and with steps that do
# not divide evenly
@pytest.mark.parametrize("cplx,m,k,n", [(0, 640, 300, 960), (0, 600, 79, 960), (0, 1152, 129, 256), (0, 520, 500, 400),
                                        (0, 300, 300, 300), (0, 640, 643, 192), (0, 383, 1100, 63), (1, 200, 131, 250),
                                        (1, 129, 300, 65)])
def test_digit_product_with_split_k(cplx, m, k, n):
    rng = np.random.default_rng(m * 1000 + k)
    _check(_graded(rng, m, k, cplx), _graded(rng, k, n, cplx))
