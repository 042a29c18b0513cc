"""One-sided Jacobi SVD of matrices far from unit scale whose columns differ
by many orders: the kept factor stays orthonormal.

Columns (s, 0, 0) and (r s, r s, 0): their coupling is 0.7 of the norms'
product whatever r, so it has to be rotated away.  Bound as in the SVD route
tests: 20 c 2^-52 (c = 2 columns) on orthonormality and, relative to the
largest, on the singular values.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("s,r", [(1e90, 1e-20), (1e-75, 1e-20), (1.0, 1e-20), (1.2e154, 0.1), (1e-140, 1e-3)])
def test_kept_factor_is_orthonormal_at_any_scale(cplx, s, r):
    import torch
    from dmrgpy_gb300 import Engine
    from dmrgpy_gb300 import mpo
    unit = np.array([[1.0, r], [0.0, r], [0.0, 0.0]])
    if cplx:
        unit = unit * np.array([[1.0, (0.6 + 0.8j)], [1.0, 1.0j], [1.0, 1.0]])
    W, _ = mpo.build_mpo([2] * 4, [(1.0 + 0j, [("Sz", 1), ("Sz", 2)])])
    eng = Engine(W, real=not cplx, precision="fp64")
    lo, ro, sv, keep, _ = eng.svd(torch.as_tensor(unit * s, device="cuda"), 0.0, 2, 2, 0)
    lim = 20 * 2 * 2.0 ** -52
    lo = lo.cpu().numpy()
    assert keep == 2
    assert np.max(np.abs(lo.conj().T @ lo - np.eye(2))) <= lim
    assert np.max(np.abs(np.asarray(sv)[:2] / s - np.linalg.svd(unit, compute_uv=False))) <= lim
    assert np.max(np.abs((lo @ ro.cpu().numpy()) / s - unit)) <= lim
