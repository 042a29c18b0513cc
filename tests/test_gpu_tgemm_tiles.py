"""The CUDA-core FP64 contraction at the edges of its output tiles
(8, 16, 32, 64), against NumPy.

Bound: both sums run over K products in FP64 in some order, so each errs by
at most K 2^-53 sum |a| |b| (complex: 2 K products per part)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 8 and 16: few outputs; 32: just under 152 tiles of 32 x 32; 64: many tiles of 64 x 64
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (17, 33, 15), (8, 32, 16), (60, 60, 60), (9, 150, 31), (150, 30, 120),
                                   (380, 17, 383), (1500, 20, 1601)])
def test_cuda_core_product_tiles(m, k, n, cplx):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if cplx:
        a = a + 1j * rng.standard_normal((m, k))
        b = b + 1j * rng.standard_normal((k, n))
    A, B = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
    C = torch.full((m, n), 3.0, dtype=A.dtype, device="cuda")
    _lib.check("dmrg_gemm", lib.dmrg_gemm(_lib.COMPLEX128 if cplx else _lib.REAL64, _lib.PREC_FP64, m, k, n,
                                          A.data_ptr(), B.data_ptr(), C.data_ptr(), None, 0,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    kk = 2 * k if cplx else k
    lim = 2 * kk * 2.0 ** -53 * (np.abs(a) @ np.abs(b)) * 1.01
    assert np.all(np.abs(C.cpu().numpy() - a @ b) <= lim)


def test_cuda_core_gram_tiles():
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    for m, k in ((5, 3), (40, 100), (33, 545), (20, 1601)):
        x = np.random.default_rng(k).standard_normal((m, k))
        X = torch.as_tensor(x, device="cuda")
        G = torch.empty((k, k), dtype=torch.float64, device="cuda")
        _lib.check("dmrg_gram", lib.dmrg_gram(_lib.GRAM_FP64, m, k, X.data_ptr(), k, G.data_ptr(), None, 0,
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        g = G.cpu().numpy()
        assert np.array_equal(g, g.T)
        assert np.all(np.abs(g - x.T @ x) <= 2 * m * 2.0 ** -53 * (np.abs(x).T @ np.abs(x)) * 1.01)
