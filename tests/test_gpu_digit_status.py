"""dmrg_heff_status reports a wait that gave up in an FP64 operator's digit
products: the word they record it in, found by its mark in the workspace and
set by the test, comes back, and the next matvec clears it.  (The wait itself
running out is covered by the bounded-wait probe.)"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MARK = 0x64675f30


@pytest.mark.parametrize("cplx,cl,cr", [(False, 300, 280), (False, 300, 40), (True, 160, 150)])
def test_status_word_of_digit_products(cplx, cl, cr):
    import torch
    from dmrgpy_gb300 import Engine, _lib
    from dmrgpy_gb300 import mpo
    terms = [(1.0 + 0j, [(op, i), (op, i + 1)]) for i in range(1, 6) for op in ("Sx", "Sy", "Sz")]
    W, _ = mpo.build_mpo([2] * 6, terms)
    eng = Engine(W, real=not cplx, precision="fp64")
    lib, w = eng.lib, eng.W[2].shape[0]
    rng = np.random.default_rng(cl)
    L, R, x = (torch.as_tensor(rng.standard_normal(s) + (0j if cplx else 0.0), device="cuda")
               for s in ((cl, w, cl), (cr, w, cr), (cl, 2, 2, cr)))
    h = eng.heff2(L, eng.W[2], eng.W[3], R, x.shape)
    r = ctypes.byref(h)
    work = torch.zeros(int(lib.dmrg_heff_workspace_bytes(r)) // 4 * 4, dtype=torch.uint8, device="cuda")
    words = work.view(torch.int32)
    args = (work.data_ptr(), work.numel(), eng.stream)
    y = torch.empty_like(x)

    def apply():
        _lib.check("dmrg_heff_apply", lib.dmrg_heff_apply(r, x.data_ptr(), y.data_ptr(), *args))

    # a workspace that no matvec has used, whatever it holds
    words.fill_(_lib.DMRG_ERR_TIMEOUT)
    assert lib.dmrg_heff_status(r, *args) == _lib.DMRG_OK
    apply()
    assert lib.dmrg_heff_status(r, *args) == _lib.DMRG_OK
    at = torch.nonzero((words[1:] == MARK) & (words[:-1] == 0)).flatten().tolist()
    assert len(at) == 1
    words[at[0]] = _lib.DMRG_ERR_TIMEOUT
    assert lib.dmrg_heff_status(r, *args) == _lib.DMRG_ERR_TIMEOUT
    apply()
    assert lib.dmrg_heff_status(r, *args) == _lib.DMRG_OK
    assert torch.isfinite(torch.view_as_real(y) if cplx else y).all()
