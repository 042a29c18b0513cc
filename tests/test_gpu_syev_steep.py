"""Symmetric eigensolver below n = 256 on steep spectra, most eigenvalues far below rounding
of the largest, as in the Gram matrices of a truncation: together the
eigenvalues err by no more than 2^-52 of the largest each, on average.  (Each
comes from products that round at 2^-53; couplings left between the small ones
would add up beyond that.)"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [50, 200, 255])
@pytest.mark.parametrize("kind", ["exponential", "gram"])
def test_sum_of_eigenvalue_errors(n, kind):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(n)
    q, r = (np.linalg.qr(rng.standard_normal((n, n)))[0] for _ in range(2))
    if kind == "gram":
        B = (q * np.exp(-25.0 * np.linspace(0.0, 1.0, n) ** 0.7)) @ r.T
        A = B @ B.T
    else:
        A = (q * np.exp(-60.0 * np.linspace(0.0, 1.0, n))) @ q.T
    A = 0.5 * (A + A.T)
    Ad = torch.as_tensor(A, device="cuda")
    got, sweeps = np.zeros(n), ctypes.c_int()
    work = torch.empty(lib.dmrg_syev_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    _lib.check("dmrg_syev", lib.dmrg_syev(n, Ad.data_ptr(), n, got.ctypes.data_as(_lib.P_double), None, n,
                                          ctypes.byref(sweeps), work.data_ptr(), work.numel(),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    w = np.linalg.eigvalsh(A)[::-1]
    assert np.sum(np.abs(got - w)) <= n * 2.0 ** -52 * w[0]
