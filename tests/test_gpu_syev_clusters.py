"""Symmetric eigensolver beyond n = 64 on eigenvalues that agree to many digits:
the FP32 passes resolve them (at most four passes: 12 + 3 x 8 sweeps), and the
results keep the bounds of the launch-shape tests (residual 2 n (3e-14 +
4 2^-53) |A|, orthonormality 8 n 2^-53)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _syev(A):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    n = A.shape[0]
    Ad = torch.as_tensor(A, device="cuda")
    V = torch.empty_like(Ad)
    got, sweeps = np.zeros(n), ctypes.c_int()
    work = torch.empty(lib.dmrg_syev_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    _lib.check("dmrg_syev", lib.dmrg_syev(n, Ad.data_ptr(), n, got.ctypes.data_as(_lib.P_double), V.data_ptr(), n,
                                          ctypes.byref(sweeps), work.data_ptr(), work.numel(),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return got, V.cpu().numpy(), sweeps.value


@pytest.mark.parametrize("n", [65, 100, 256])
@pytest.mark.parametrize("kind", ["1 + 1e-6 x", "1 + 1e-9 x", "pairs"])
def test_eigenvalues_that_agree(n, kind):
    rng = np.random.default_rng(n)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    if kind == "pairs":
        w = np.repeat(np.exp(-10.0 * np.linspace(0.0, 1.0, (n + 1) // 2)), 2)[:n] * (1.0 + 1e-12 * rng.random(n))
    else:
        w = 1.0 + float(kind.split()[2]) * rng.random(n)
    A = (q * w) @ q.T
    A = 0.5 * (A + A.T)
    got, v, sweeps = _syev(A)
    lim = 2 * n * (3e-14 + 4 * 2.0 ** -53) * np.max(w)
    assert np.max(np.abs(A @ v - v * got)) <= lim
    assert np.max(np.abs(v.T @ v - np.eye(n))) <= 8 * n * 2.0 ** -53
    assert np.max(np.abs(got - np.linalg.eigvalsh(A)[::-1])) <= lim
    assert sweeps <= 36
