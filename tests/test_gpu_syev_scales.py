"""Symmetric eigensolver on matrices whose largest element is off the
diagonal, far from unit scale: hollow ones and ones with a diagonal of 1e-20
of the rest.  Bounds as in the tests of its launch shapes (residual and
eigenvalues 2 n (3e-14 + 4 2^-53) |A|, orthonormality 8 n 2^-53), with |A| at
most n times the largest element.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _syev(A):
    import torch
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    n = A.shape[0]
    Ad = torch.as_tensor(A, device="cuda")
    V = torch.empty_like(Ad)
    got, sweeps = np.zeros(n), ctypes.c_int()
    work = torch.empty(lib.dmrg_syev_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    st = lib.dmrg_syev(n, Ad.data_ptr(), n, got.ctypes.data_as(_lib.P_double), V.data_ptr(), n, ctypes.byref(sweeps),
                       work.data_ptr(), work.numel(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return st, got, V.cpu().numpy()


# one launch of one block pair, of two, and the blocked rounds
@pytest.mark.parametrize("n", [2, 20, 50, 100])
@pytest.mark.parametrize("diag", [0.0, 1e-20])
@pytest.mark.parametrize("scale", [1e20, 1e-20, 1.0, 1e300, 1e-290])
def test_largest_element_off_the_diagonal(n, diag, scale):
    rng = np.random.default_rng(n)
    unit = rng.uniform(-1.0, 1.0, (n, n))
    unit = 0.5 * (unit + unit.T)
    if n == 2:
        unit[0, 1] = unit[1, 0] = 1.0
    np.fill_diagonal(unit, diag * rng.uniform(0.5, 1.0, n))
    st, got, v = _syev(unit * scale)
    assert st == 0
    w = np.linalg.eigvalsh(unit)[::-1]
    norm = np.max(np.abs(w))
    lim = 2 * n * (3e-14 + 4 * 2.0 ** -53) * norm
    got = got / scale
    assert np.max(np.abs(unit @ v - v * got)) <= lim
    assert np.max(np.abs(v.T @ v - np.eye(n))) <= 8 * n * 2.0 ** -53
    assert np.max(np.abs(got - w)) <= lim


@pytest.mark.parametrize("n", [2, 20, 100])
def test_infinite_diagonal_element_stands_alone(n):
    """No rotation touches it: the sweeps on the matrix itself leave it, the
    others and the unit vectors exactly."""
    A = np.eye(n)
    A[1, 1] = np.inf
    st, got, v = _syev(A)
    assert st == 0
    assert got[0] == np.inf and np.all(got[1:] == 1.0)
    assert np.array_equal(np.sort(np.abs(v), axis=None)[::-1][:n], np.ones(n)) and np.sum(np.abs(v)) == n


@pytest.mark.parametrize("n", [2, 50, 100])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_input_is_reported(n, bad):
    from dmrgpy_gb300 import _lib
    A = np.eye(n)
    A[0, 1] = A[1, 0] = bad
    assert _syev(A)[0] == _lib.DMRG_ERR_NAN
