"""The two error bounds of an FP64 contraction that the header states, on
matrices where they differ: large elements of a row of A meet zeros or far
smaller elements of the columns of B (block-sparse, and graded along k in
opposite directions).

With the workspace (digit product): 2^-53 |c| + (K + 128) 2^-58 max|row of A|
max|column of B|.  Without it (FP64 pipe): K 2^-53 sum |a||b|."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gemm(a, b, digits):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    (m, k), n = a.shape, b.shape[1]
    A, B = torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda")
    C = torch.full((m, n), 7.0, dtype=torch.float64, device="cuda")
    need = int(lib.dmrg_gemm_workspace_bytes(_lib.REAL64, _lib.PREC_FP64, m, k, n))
    assert need > 0
    w = torch.empty(need, dtype=torch.uint8, device="cuda") if digits else None
    _lib.check("dmrg_gemm", lib.dmrg_gemm(_lib.REAL64, _lib.PREC_FP64, m, k, n, A.data_ptr(), B.data_ptr(),
                                          C.data_ptr(), w.data_ptr() if digits else None, need if digits else 0,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return C.cpu().numpy().astype(np.longdouble)


def _case(kind):
    m, k, n = 640, 300, 576
    rng = np.random.default_rng(len(kind))
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if kind == "one element":            # (1, 1e-20, 0, ...) against (0, 1, 0, ...)
        a, b = np.zeros((m, k)), np.zeros((k, n))
        a[:, 0], a[:, 1] = 1.0, 1e-20 * rng.uniform(1.0, 2.0, m)
        b[1] = rng.uniform(1.0, 2.0, n)
    elif kind == "blocks":               # rows' large halves meet zeros
        a[:, :150] *= 1e15
        b[:150, ::2] = 0.0
    else:                                # opposite grading along k
        g = np.exp(-80.0 * np.linspace(0.0, 1.0, k))
        a, b = a * g, b * g[::-1, None]
    return a, b


@pytest.mark.parametrize("kind", ["one element", "blocks", "graded"])
def test_both_bounds(kind):
    a, b = _case(kind)
    k = a.shape[1]
    al, bl = a.astype(np.longdouble), b.astype(np.longdouble)
    exact, mags = al @ bl, np.abs(al) @ np.abs(bl)
    norm = np.outer(np.abs(al).max(1), np.abs(bl).max(0))
    err = np.abs(_gemm(a, b, True) - exact)
    assert np.all(err <= 2.0 ** -53 * np.abs(exact) + (k + 128) * 2.0 ** -58 * norm)
    err = np.abs(_gemm(a, b, False) - exact)
    assert np.all(err <= k * 2.0 ** -53 * mags)
