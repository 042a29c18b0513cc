"""FP64 matvecs and environment extensions: row-list MPO steps and digit
products against plain tensor contractions, with the full workspace and with
one that only holds the two intermediates (FP64 pipe, dense MPO step).

Tolerance: three to four chained FP64 contractions of at most K = 4 w chi
products each, compared by 2-norm; each side errs by less than K 2^-53 of
the product of the factors' norms, which exceeds the result's by a modest
factor for these random tensors: 1e-12 leaves two decades."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _rnd(rng, shape, cplx, keep=1.0):
    x = rng.standard_normal(shape)
    if cplx:
        x = x + 1j * rng.standard_normal(shape) * (rng.random(shape) < 0.5)   # some entries real
    return x * (rng.random(shape) < keep)


def _close(got, ref):
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)


# row lists: empty, one entry, full; inner index around a warp; digit and FP64-pipe sizes
@pytest.mark.parametrize("kind,cplx,cl,cr,d1,d2,w,keep", [
    (2, False, 1, 31, 2, 2, 5, 0.15), (2, False, 33, 32, 3, 2, 5, 1.0), (2, True, 40, 33, 2, 3, 4, 0.3),
    (2, False, 200, 161, 2, 2, 5, 0.1), (2, True, 130, 97, 2, 2, 3, 0.2), (1, False, 300, 129, 3, 1, 5, 0.2),
    (1, True, 65, 64, 2, 1, 4, 0.5), (0, False, 90, 250, 1, 1, 5, 1.0), (0, True, 64, 31, 1, 1, 3, 1.0)])
def test_matvec_routes(kind, cplx, cl, cr, d1, d2, w, keep):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(cl + cr)
    wl, wm, wr = (w, w + 1, w) if kind == 2 else (w, w, w)
    L, R = _rnd(rng, (cl, wl, cl), cplx), _rnd(rng, (cr, wr, cr), cplx)
    if kind == 2:
        W1, W2 = _rnd(rng, (wl, d1, d1, wm), cplx, keep), _rnd(rng, (wm, d2, d2, wr), cplx, keep)
        W1[0, 0, 0, 0] = W2[0, 0, 0, 0] = 1.0
        x = _rnd(rng, (cl, d1, d2, cr), cplx)
        ref = np.einsum("pka,astb->pkstb", L, x)
        ref = np.einsum("pkstb,ksum->pumtb", ref, W1)
        ref = np.einsum("pumtb,mtvn->puvnb", ref, W2)
        ref = np.einsum("puvnb,qnb->puvq", ref, R)
    elif kind == 1:
        W1, W2 = _rnd(rng, (wl, d1, d1, wr), cplx, keep), None
        W1[0, 0, 0, 0] = 1.0
        x = _rnd(rng, (cl, d1, cr), cplx)
        ref = np.einsum("pksb,ksum->pumb", np.einsum("pka,asb->pksb", L, x), W1)
        ref = np.einsum("pumb,qmb->puq", ref, R)
    else:
        W1 = W2 = None
        x = _rnd(rng, (cl, cr), cplx)
        ref = np.einsum("pkb,qkb->pq", np.einsum("pka,ab->pkb", L, x), R)
    dev = [None if t is None else torch.as_tensor(t, device="cuda") for t in (L, W1, W2, R, x)]
    h = _lib.HeffDesc()
    h.kind, h.dtype, h.precision = kind, _lib.COMPLEX128 if cplx else _lib.REAL64, _lib.PREC_FP64
    h.chil, h.d1, h.d2, h.chir, h.wl, h.wm, h.wr = cl, d1, d2, cr, wl, wm, wr
    h.L, h.R = dev[0].data_ptr(), dev[3].data_ptr()
    h.W1 = dev[1].data_ptr() if dev[1] is not None else None
    h.W2 = dev[2].data_ptr() if dev[2] is not None else None
    es = 16 if cplx else 8
    dd = d1 * d2
    up = lambda n: (n + 255) // 256 * 256   # noqa: E731
    lean = up(es * max(cl * wl * dd * cr, cl * dd * wr * cr if kind == 2 else 0)) + \
        up(es * (cl * d1 * wm * d2 * cr if kind == 2 else cl * d1 * wr * cr if kind == 1 else 0))
    full = lib.dmrg_heff_workspace_bytes(ctypes.byref(h))
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for size in (full, lean):
        work = torch.empty(size, dtype=torch.uint8, device="cuda")
        y = torch.full_like(dev[4], float("nan"))
        _lib.check("dmrg_heff_apply", lib.dmrg_heff_apply(ctypes.byref(h), dev[4].data_ptr(), y.data_ptr(),
                                                          work.data_ptr(), size, s))
        _close(y.cpu().numpy(), ref)
    small = min(full, lean) // 2
    assert lib.dmrg_heff_apply(ctypes.byref(h), dev[4].data_ptr(), y.data_ptr(), work.data_ptr(), small, s) == \
        _lib.DMRG_ERR_WORKSPACE


@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("cplx,clb,crb,clk,crk,d,wl,wr", [
    (False, 1, 9, 1, 7, 2, 1, 5), (False, 33, 40, 64, 31, 3, 5, 4), (True, 40, 33, 25, 50, 2, 4, 5),
    (False, 200, 150, 170, 190, 2, 5, 5), (True, 120, 100, 90, 130, 2, 3, 3)])
def test_environment_routes(side, cplx, clb, crb, clk, crk, d, wl, wr):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(clb + crk)
    B, A = _rnd(rng, (clb, d, crb), cplx), _rnd(rng, (clk, d, crk), cplx)
    W = _rnd(rng, (wl, d, d, wr), cplx, 0.4)
    W[0, 0, 0, 0] = 1.0
    if side == 0:
        E = _rnd(rng, (clb, wl, clk), cplx)
        ref = np.einsum("pksb,ksum->pumb", np.einsum("pka,asb->pksb", E, A), W)
        ref = np.einsum("puq,pumb->qmb", B.conj(), ref)
        n = clb * wl * d * crk + clb * d * wr * crk
    else:
        E = _rnd(rng, (crb, wr, crk), cplx)
        ref = np.einsum("qmas,ksum->qkua", np.einsum("qmb,asb->qmas", E, A), W)
        ref = np.einsum("puq,qkua->pka", B.conj(), ref)
        n = crb * wr * clk * d + crb * wl * d * clk
    dt = _lib.COMPLEX128 if cplx else _lib.REAL64
    dev = [torch.as_tensor(t, device="cuda") for t in (E, W, B, A)]
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    dims = (clb, crb, clk, crk, d, wl, wr)
    full = lib.dmrg_env_mixed_workspace_bytes(side, dt, *dims)
    for size in (full, n * (16 if cplx else 8)):
        work = torch.empty(size, dtype=torch.uint8, device="cuda")
        out = torch.full(ref.shape, float("nan"), dtype=dev[0].dtype, device="cuda")
        _lib.check("dmrg_env_extend_mixed", lib.dmrg_env_extend_mixed(
            side, dt, *dims, *[t.data_ptr() for t in dev], out.data_ptr(), work.data_ptr(), size, s))
        _close(out.cpu().numpy(), ref)
    assert lib.dmrg_env_extend_mixed(side, dt, *dims, *[t.data_ptr() for t in dev], out.data_ptr(), work.data_ptr(),
                                     n * 4, s) == _lib.DMRG_ERR_WORKSPACE
