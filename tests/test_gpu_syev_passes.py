"""Symmetric eigensolver (FP32 sweeps between FP64 products) at the edges of
its launch shapes, on spectra with multiplets, of both signs and graded as
the Gram matrices of a truncation are.

Bounds: a rotation is skipped below 1e-14 sqrt|g_ii g_jj| or 1e-15 |A| (the
passes stop within 3 times that), at most n couplings a row; the products
V^T A V and the last Newton-Schulz step round at n 2^-53 each.  Residual
below n (3e-14 + 4 2^-53) |A|, orthonormality below 4 n 2^-53, both with a
factor of 2 for the norm taken (largest element).
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one 32-wide block pair, the 64-wide one launch and the blocked rounds, each
# at its first, last and a ragged size
@pytest.mark.parametrize("n", [2, 17, 32, 33, 60, 64, 65, 96, 130, 200])
@pytest.mark.parametrize("kind", ["graded", "multiplets", "indefinite"])
def test_syev_launch_shapes(n, kind):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(n)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    if kind == "graded":
        w = np.exp(-18.0 * np.linspace(0.0, 1.0, n) ** 0.5)
    elif kind == "multiplets":
        w = 0.5 ** (np.arange(n) // 5)
    else:
        w = rng.uniform(-1.0, 1.0, n)
    A = (q * w) @ q.T
    A = 0.5 * (A + A.T)
    Ad = torch.as_tensor(A, device="cuda")
    V = torch.empty_like(Ad)
    got, sweeps = np.zeros(n), ctypes.c_int()
    work = torch.empty(lib.dmrg_syev_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    _lib.check("dmrg_syev", lib.dmrg_syev(n, Ad.data_ptr(), n, got.ctypes.data_as(_lib.P_double), V.data_ptr(), n,
                                          ctypes.byref(sweeps), work.data_ptr(), work.numel(),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    v = V.cpu().numpy()
    norm = np.max(np.abs(w))
    lim = 2 * n * (3e-14 + 4 * 2.0 ** -53) * norm
    assert np.max(np.abs(A @ v - v * got)) <= lim
    assert np.max(np.abs(v.T @ v - np.eye(n))) <= 8 * n * 2.0 ** -53
    assert np.max(np.abs(got - np.sort(w)[::-1])) <= lim
