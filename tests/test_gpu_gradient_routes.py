"""dmrg_env_gradient_mixed on both of its contraction orders (the right
tensor first, or the bra first where d crk <= clb wr) against NumPy sums.

Error bound per output: at most clk + clb + crk crb products and sums follow
one another (clk + crk + clb crb in the other order), each rounded to 2^-53
of the sum of absolute products; complex products double the count.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# bra first at and around the line d crk = clb wr, m tiles of 8 full and
# ragged, chunks of (b', b) shorter and longer than one (1024), bonds of 1
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("clb,crb,clk,crk,d,wl,wr", [
    (24, 20, 22, 18, 2, 3, 5), (6, 9, 6, 9, 2, 5, 3), (6, 9, 6, 10, 2, 5, 3), (33, 70, 31, 67, 2, 4, 8),
    (12, 37, 40, 41, 4, 2, 17), (40, 1, 30, 1, 3, 1, 1), (1, 2, 1, 2, 2, 1, 9), (5, 300, 7, 1, 2, 2, 2)])
def test_gradient_orders_match_numpy(cplx, clb, crb, clk, crk, d, wl, wr):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(clb * 100 + crk)

    def rand(*shape):
        x = rng.standard_normal(shape)
        return x + 1j * rng.standard_normal(shape) if cplx else x

    L, A, B, R = rand(clb, wl, clk), rand(clk, d, crk), rand(clb, d, crb), rand(crb, wr, crk)
    dt = _lib.COMPLEX128 if cplx else _lib.REAL64
    dev = [torch.as_tensor(x, device="cuda") for x in (L, B, A, R)]
    G = torch.full((wl, d, d, wr), 7.0, dtype=dev[0].dtype, device="cuda")
    need = int(lib.dmrg_env_gradient_mixed_workspace_bytes(dt, clb, crb, clk, crk, d, wl, wr))
    w = torch.full((need,), 255, dtype=torch.uint8, device="cuda")   # NaN wherever it is read unwritten
    _lib.check("dmrg_env_gradient_mixed", lib.dmrg_env_gradient_mixed(
        dt, clb, crb, clk, crk, d, wl, wr, *(x.data_ptr() for x in dev), G.data_ptr(), w.data_ptr(), need,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))

    def contract(l, a, b, r):
        y = np.einsum("pka,asb->pksb", l, a, optimize=True)
        v = np.einsum("pksb,ptq->kstqb", y, b, optimize=True)
        return np.einsum("kstqb,qmb->kstm", v, r, optimize=True)

    want = contract(L, A, B.conj(), R)
    size = contract(np.abs(L), np.abs(A), np.abs(B), np.abs(R))
    n = clk + clb + crk + max(crk * crb, clb * crb)
    assert np.all(np.abs(G.cpu().numpy() - want) <= 2 * (2 if cplx else 1) * n * 2.0 ** -53 * size)
