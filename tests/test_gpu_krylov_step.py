"""The one-launch Krylov step on both sides of its size limit, against a
dense eigenproblem and a dense exponential.

Zero-site operators (L, R) make H = sum_k L_k (x) R_k dense and cheap at any
vector length.  Tolerance: the loops stop when the Ritz value moves by less
than 1e-13 of max(1, |E|), or the exponential's residual is below 1e-13; the
dense references err by n 2^-53 |H| ~ 1e-13 |H|, so 1e-11 |H| leaves a
decade or more.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(cl, cr, cplx):
    import torch
    from dmrgpy_gb300 import _lib
    rng = np.random.default_rng(cl * 1000 + cr)

    def herm(n):
        x = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0.0)
        return (x + x.conj().T) / np.sqrt(8 * n)

    # H = A (x) 1 + 1 (x) B: spectrum and exponential follow from the factors'
    A, B = herm(cl), herm(cr)
    L = np.stack([A, np.eye(cl)], axis=1).astype(A.dtype)
    R = np.stack([np.eye(cr), B], axis=1).astype(A.dtype)
    x = rng.standard_normal((cl, cr)) + (1j * rng.standard_normal((cl, cr)) if cplx else 0.0)
    x /= np.linalg.norm(x)
    dev = [torch.as_tensor(np.ascontiguousarray(t), device="cuda") for t in (L, R, x)]
    h = _lib.HeffDesc()
    h.kind, h.dtype, h.precision = 0, _lib.COMPLEX128 if cplx else _lib.REAL64, _lib.PREC_FP64
    h.chil, h.d1, h.d2, h.chir, h.wl, h.wm, h.wr = cl, 1, 1, cr, 2, 2, 2
    h.L, h.R = dev[0].data_ptr(), dev[1].data_ptr()
    return A, B, x, dev, h


# one element, one CTA's chunk and just past it, ragged slices, the last
# length of the one-launch step (152 x 1536) and the first past it
@pytest.mark.parametrize("cl,cr", [(1, 1), (8, 16), (43, 3), (61, 37), (456, 512), (457, 512)])
@pytest.mark.parametrize("cplx", [False, True])
def test_krylov_loops_match_dense(cl, cr, cplx):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    A, B, x, dev, h = _problem(cl, cr, cplx)
    wa, va = np.linalg.eigh(A)
    wb, vb = np.linalg.eigh(B)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    kmax = min(120, cl * cr)
    need = max(lib.dmrg_lanczos_workspace_bytes(ctypes.byref(h), kmax),
               lib.dmrg_expm_workspace_bytes(ctypes.byref(h), kmax))
    work = torch.empty(need, dtype=torch.uint8, device="cuda")
    e, it = ctypes.c_double(), ctypes.c_int()
    if cplx:
        y = dev[2].clone()
        _lib.check("dmrg_krylov_expm", lib.dmrg_krylov_expm(ctypes.byref(h), y.data_ptr(), 0.0, -0.5, kmax, 1e-13,
                                                            1e-13, ctypes.byref(it), work.data_ptr(), need, s))
        # exp(-i t (A (x) 1 + 1 (x) B)) X = exp(-i t A) X exp(-i t B)^T
        ea = (va * np.exp(-0.5j * wa)) @ va.conj().T
        eb = (vb * np.exp(-0.5j * wb)) @ vb.conj().T
        assert np.linalg.norm(y.cpu().numpy() - ea @ x @ eb.T) <= 1e-11
    y = dev[2].clone()
    _lib.check("dmrg_lanczos_ground", lib.dmrg_lanczos_ground(ctypes.byref(h), y.data_ptr(), kmax, 1e-13,
                                                              ctypes.byref(e), ctypes.byref(it), work.data_ptr(),
                                                              need, s))
    want = wa[0] + wb[0]
    got = y.cpu().numpy()
    # the value is the state's own, never below the lowest; equal to it where the space is exhausted
    hy = A @ got + got @ B.T
    scale = max(1.0, abs(want))
    assert abs(np.vdot(got, hy).real / np.vdot(got, got).real - e.value) <= 1e-11 * scale
    assert e.value >= want - 1e-11 * scale
    if cl * cr <= 129:
        assert abs(e.value - want) <= 1e-11 * scale
