"""One-sided Jacobi SVD on its three launch shapes (one CTA up to 7 pairs a
round, a cluster up to 64 columns, a cooperative grid beyond) against NumPy.

Bound: a column meets at most c rotations a sweep, each rounded to a few
2^-53 of the larger column, over at most 20 sweeps: 20 c 2^-52 of the largest
singular value, for values, product and orthonormality alike.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# pairs 7, 8 (first of the cluster); odd counts; 64 columns (last of the
# cluster), 65 and 66; real matrices of these shapes take this route because
# the kept side is more than twice the other
@pytest.mark.parametrize("cplx,m,n,absorb", [
    (False, 60, 14, 0), (False, 15, 47, 1), (False, 60, 16, 0), (False, 140, 64, 0), (False, 66, 140, 1),
    (True, 14, 20, 0), (True, 16, 15, 1), (True, 33, 33, 0), (True, 64, 64, 1), (True, 65, 70, 0), (True, 70, 66, 0)])
def test_svd_routes_match_numpy(cplx, m, n, absorb):
    import torch
    from dmrgpy_gb300 import Engine
    from dmrgpy_gb300 import mpo
    rng = np.random.default_rng(m * 100 + n)
    c = min(m, n)

    def iso(r):
        x = rng.standard_normal((r, c)) + (1j * rng.standard_normal((r, c)) if cplx else 0.0)
        return np.linalg.qr(x)[0]

    # singular values over five decades, one of them five times over
    s = np.exp(-11.5 * np.linspace(0.0, 1.0, c) ** 0.5)
    s[c // 2:c // 2 + 5] = s[c // 2]
    M = (iso(m) * s) @ iso(n).conj().T
    W, _ = mpo.build_mpo([2] * 4, [(1.0 + 0j, [("Sz", 1), ("Sz", 2)])])
    eng = Engine(W, real=not cplx, precision="fp64")
    lo, ro, sv, keep, _ = eng.svd(torch.as_tensor(np.ascontiguousarray(M), device="cuda"), 0.0, c, 1, absorb)
    lo, ro = lo.cpu().numpy(), ro.cpu().numpy()
    lim = 20 * c * 2.0 ** -52
    assert keep == c
    assert np.max(np.abs(np.asarray(sv)[:c] - np.linalg.svd(M, compute_uv=False))) <= lim
    assert np.linalg.norm(lo @ ro - M, 2) <= lim * np.sqrt(c)
    q = lo.conj().T @ lo if absorb == 0 else ro @ ro.conj().T
    assert np.max(np.abs(q - np.eye(c))) <= lim
