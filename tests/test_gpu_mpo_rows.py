"""MPO steps of few CTAs, whose rows are spread over several: environments and
one-site matvecs of narrow bonds with wide dense MPOs against plain
contractions.  Tolerance as in the other FP64 contraction tests: three chained
contractions of K <= 400, 1e-12 of the result's norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one CTA and many row groups; rows that do not divide by eight; a leg beyond a warp
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("cl,cr,d,w", [(1, 1, 2, 3), (2, 3, 3, 41), (5, 40, 4, 13), (33, 4, 2, 60)])
def test_rows_over_several_ctas(cplx, cl, cr, d, w):
    import torch
    from dmrgpy_gb300 import Engine
    rng = np.random.default_rng(cl * 100 + w)

    def rnd(*s):
        x = rng.standard_normal(s)
        return x + 1j * rng.standard_normal(s) if cplx else x

    W = rnd(w, d, d, w)
    eng = Engine([W, W], real=not cplx, precision="fp64")
    L, R, A = rnd(cl, w, cl), rnd(cr, w, cr), rnd(cl, d, cr)
    Ld, Rd, Ad = (torch.as_tensor(x, device="cuda") for x in (L, R, A))

    def close(got, ref):
        assert np.linalg.norm(got.cpu().numpy() - ref) <= 1e-12 * np.linalg.norm(ref)

    x = np.einsum("pka,asb->pksb", L, A)
    x = np.einsum("pksb,ksum->pumb", x, W)
    close(eng.env_left(Ld, eng.W[0], Ad), np.einsum("puq,pumb->qmb", A.conj(), x))
    close(eng.apply(eng.heff1(Ld, eng.W[0], Rd, A.shape), Ad), np.einsum("pumb,qmb->puq", x, R))
    z = np.einsum("qmb,asb->qmsa", R, A)
    z = np.einsum("qmsa,ksum->qkua", z, W)
    close(eng.env_right(Rd, eng.W[0], Ad), np.einsum("puq,qkua->pka", A.conj(), z))
