"""Split-TF32 operands whose K is no multiple of 32 are padded with zeros:
the same results from a workspace full of NaN as from one full of zeros,
bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cl,cr,d,w", [(37, 45, 2, 5), (64, 32, 2, 4), (33, 31, 3, 1)])
def test_tf32x3_ignores_what_the_workspace_held(cl, cr, d, w):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(cl)
    dev = [torch.as_tensor(rng.standard_normal(sh), device="cuda")
           for sh in ((cl, w, cl), (w, d, d, w), (w, d, d, w), (cr, w, cr), (cl, d, d, cr), (cl, d, cr))]
    L, W1, W2, R, x, A = dev
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    h = _lib.HeffDesc()
    h.kind, h.dtype, h.precision = 2, _lib.REAL64, _lib.PREC_TF32X3
    h.chil, h.d1, h.d2, h.chir, h.wl, h.wm, h.wr = cl, d, d, cr, w, w, w
    h.L, h.W1, h.W2, h.R = L.data_ptr(), W1.data_ptr(), W2.data_ptr(), R.data_ptr()
    env = (_lib.REAL64, _lib.PREC_TF32X3, cl, d, cr, w, w)
    runs = []
    for fill in (0, 255):
        y = torch.zeros_like(x)
        ln, rn = (torch.zeros((c, w, c), dtype=x.dtype, device="cuda") for c in (cr, cl))
        work = torch.full((lib.dmrg_heff_workspace_bytes(ctypes.byref(h)),), fill, dtype=torch.uint8, device="cuda")
        _lib.check("dmrg_heff_apply", lib.dmrg_heff_apply(ctypes.byref(h), x.data_ptr(), y.data_ptr(),
                                                          work.data_ptr(), work.numel(), s))
        work = torch.full((lib.dmrg_env_workspace_bytes(*env),), fill, dtype=torch.uint8, device="cuda")
        for f, E, out in (("dmrg_env_extend_left", L, ln), ("dmrg_env_extend_right", R, rn)):
            _lib.check(f, getattr(lib, f)(*env, E.data_ptr(), W1.data_ptr(), A.data_ptr(), out.data_ptr(),
                                          work.data_ptr(), work.numel(), s))
        runs.append([t.cpu().numpy() for t in (y, ln, rn)])
    for a, b in zip(*runs):
        assert np.isfinite(a).all() and np.array_equal(a, b)
