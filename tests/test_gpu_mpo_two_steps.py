"""Bond MPO steps on both sides of the line between one pass over the product
of the two site tensors and one step per site, dense and sparse, with unequal
links, against plain contractions (1e-12 of the result's norm, as in the other
FP64 contraction tests), with prepared digits (Krylov loop) and without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# elements of the product, against 16384: d = 2 (always one pass), below, above,
# unequal links above, digit products above, a site dimension of 1
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("cl,cr,d1,d2,wl,wm,wr,keep", [
    (20, 33, 2, 2, 40, 41, 40, 1.0), (20, 17, 3, 3, 14, 13, 14, 1.0), (20, 17, 3, 3, 15, 15, 15, 0.3),
    (7, 5, 4, 3, 17, 9, 23, 1.0), (1, 1, 4, 4, 16, 16, 16, 1.0), (200, 180, 4, 4, 10, 10, 9, 0.1),
    (30, 40, 8, 1, 20, 3, 20, 1.0)])
def test_two_site_matvec_of_wide_mpos(cplx, cl, cr, d1, d2, wl, wm, wr, keep):
    import torch
    from dmrgpy_gb300 import Engine
    rng = np.random.default_rng(wl * 100 + wr)

    def rnd(*s):
        x = rng.standard_normal(s)
        return x + 1j * rng.standard_normal(s) if cplx else x

    W1, W2 = rnd(wl, d1, d1, wm), rnd(wm, d2, d2, wr)
    W1, W2 = W1 * (rng.random(W1.shape) < keep), W2 * (rng.random(W2.shape) < keep)
    L, R, x = rnd(cl, wl, cl), rnd(cr, wr, cr), rnd(cl, d1, d2, cr)
    eng = Engine([W1, W2], real=not cplx, precision="fp64")
    Ld, Rd, xd = (torch.as_tensor(v, device="cuda") for v in (L, R, x))
    y = eng.apply(eng.heff2(Ld, eng.W[0], eng.W[1], Rd, x.shape), xd).cpu().numpy()
    ref = np.einsum("pka,astb->pkstb", L, x, optimize=True)
    ref = np.einsum("pkstb,ksum->pumtb", ref, W1, optimize=True)
    ref = np.einsum("pumtb,mtvn->puvnb", ref, W2, optimize=True)
    ref = np.einsum("puvnb,qnb->puvq", ref, R, optimize=True)
    assert np.linalg.norm(y - ref) <= 1e-12 * np.linalg.norm(ref)
