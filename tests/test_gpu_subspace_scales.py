"""Split-TF32 truncation of a matrix times a power of two: its FP32 Ritz
values are those of the matrix times that power, bit for bit (every step of
the route scales exactly while FP32 holds the matrix)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("absorb", [0, 1])
@pytest.mark.parametrize("m,k", [(96, 40), (200, 128)])
def test_ritz_values_scale_with_the_matrix(m, k, absorb):
    import torch
    from dmrgpy_gb300 import Engine
    from dmrgpy_gb300 import mpo
    rng = np.random.default_rng(m)
    u, v = (np.linalg.qr(rng.standard_normal((m, m)))[0] for _ in range(2))
    M = (u * np.exp(-7.0 * np.sqrt(np.linspace(0.0, 1.0, m)))) @ v.T
    start = np.ascontiguousarray(v.T[:k] if absorb == 0 else u[:, :k])
    W, _ = mpo.build_mpo([2] * 4, [(1.0 + 0j, [("Sz", 1), ("Sz", 2)])])
    eng = Engine(W, real=True, precision="tf32x3")
    eng.want_spectra = True

    def values(scale):
        _, _, s, keep, _ = eng.subspace_split(torch.as_tensor(M * scale, device="cuda"), k,
                                              torch.as_tensor(start, device="cuda"), k, absorb, 0.0)
        assert keep == k
        return np.asarray(s)[:k]

    ref = values(1.0)
    # FP32 accuracy of the leading value, 1
    assert abs(ref[0] - 1.0) < 2e-6
    for p in (-80, -40, 40, 80):
        assert np.array_equal(values(2.0 ** p) / 2.0 ** p, ref), p
