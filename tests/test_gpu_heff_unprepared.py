"""FP64 operators keep nothing in the workspace: dmrg_heff_apply_prepared
without a prepare, on a workspace of arbitrary contents, with the workspace
overwritten in between, with a larger one than at the prepare, and after a
change of the environment in place gives dmrg_heff_apply's bits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# row lists alone; digit products for both, one or none of the contractions
@pytest.mark.parametrize("cplx,cl,cr,d", [(False, 12, 9, 2), (False, 300, 280, 2), (False, 300, 40, 3),
                                          (True, 20, 33, 2), (True, 160, 150, 2)])
def test_apply_prepared_needs_no_prepare(cplx, cl, cr, d):
    import torch
    from dmrgpy_gb300 import Engine, _lib
    from dmrgpy_gb300 import mpo
    code = {2: 2, 3: 3}[d]
    terms = [(1.0 + 0j, [(op, i), (op, i + 1)]) for i in range(1, 6) for op in ("Sx", "Sy", "Sz")]
    W, _ = mpo.build_mpo([code] * 6, terms)
    eng = Engine(W, real=not cplx, precision="fp64")
    lib, w = eng.lib, eng.W[2].shape[0]
    rng = np.random.default_rng(cl)

    def rnd(*shape):
        v = rng.standard_normal(shape)
        return torch.as_tensor(v + 1j * rng.standard_normal(shape) if cplx else v, device="cuda")

    L, R, x = rnd(cl, w, cl), rnd(cr, w, cr), rnd(cl, d, d, cr)
    h = eng.heff2(L, eng.W[2], eng.W[3], R, x.shape)
    r = ctypes.byref(h)
    need = int(lib.dmrg_heff_workspace_bytes(r))
    work = torch.full((2 * need + 4096,), 255, dtype=torch.uint8, device="cuda")
    y = torch.empty_like(x)

    def prepared(size):
        y.fill_(7.0)
        _lib.check("dmrg_heff_apply_prepared", lib.dmrg_heff_apply_prepared(
            r, x.data_ptr(), y.data_ptr(), work.data_ptr(), size, eng.stream))
        return y.clone()

    ref = eng.apply(h, x)
    assert torch.isfinite(torch.view_as_real(ref) if cplx else ref).all()
    assert torch.equal(prepared(need), ref)
    work.fill_(171)
    assert torch.equal(prepared(need), ref)
    _lib.check("dmrg_heff_prepare", lib.dmrg_heff_prepare(r, work.data_ptr(), need, eng.stream))
    assert torch.equal(prepared(work.numel()), ref)
    old = ref
    L.mul_(-2.0)
    ref = eng.apply(h, x)
    assert torch.equal(prepared(work.numel()), ref)
    assert torch.linalg.vector_norm(ref + 2.0 * old) <= 1e-12 * torch.linalg.vector_norm(ref)
    # the two intermediates alone (FP64 pipe, dense MPO steps) and back
    es = 16 if cplx else 8
    lean = sum((n * es + 255) // 256 * 256 for n in (cl * w * d * d * cr, cl * d * w * d * cr))
    z = prepared(lean)
    assert torch.linalg.vector_norm(z - ref) <= 1e-12 * torch.linalg.vector_norm(ref)
    assert torch.equal(prepared(need), ref)
