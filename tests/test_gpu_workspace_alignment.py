"""FP64 entry points with a workspace 8 bytes off a 16-byte boundary, at sizes
whose products run as digit products otherwise: the calls keep to the FP64
pipe and agree with an aligned workspace.

Tolerance: chains of at most four FP64 contractions of K <= 3000, each side
within K 2^-53 of the factors' norms of the exact result: 1e-11 of the
result's norm leaves more than a decade (vectors of the Krylov loops: their
stop tolerance, 1e-8)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Shifted:
    """An engine's workspace, every pointer 8 bytes further on."""

    def __init__(self, ws):
        self.ws = ws

    def get(self, need):
        ptr, size = self.ws.get(need + 8)
        assert ptr % 16 == 0
        return ptr + 8, size - 8


def _two():
    from dmrgpy_gb300 import Engine
    from dmrgpy_gb300 import mpo
    terms = [(1.0 + 0j, [(op, i), (op, i + 1)]) for i in range(1, 6) for op in ("Sx", "Sy", "Sz")]
    W, _ = mpo.build_mpo([2] * 6, terms)
    out = [Engine(W, real=True, precision="fp64") for _ in range(2)]
    out[1].ws = _Shifted(out[1].ws)
    return out


def _close(a, b, tol=1e-11):
    a, b = a.cpu().numpy(), b.cpu().numpy()
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(a)


def _rand(*shape):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(shape))
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


def test_contractions():
    a, b = _two()
    chi = 300
    w = a.W[2].shape[0]
    L, R, x, A = _rand(chi, w, chi), _rand(chi, w, chi), _rand(chi, 2, 2, chi), _rand(chi, 2, chi)
    L, R = L + L.permute(2, 1, 0), R + R.permute(2, 1, 0)
    L, R = L.contiguous(), R.contiguous()
    y = [e.apply(e.heff2(L, e.W[2], e.W[3], R, x.shape), x) for e in (a, b)]
    _close(*y)
    _close(a.env_left(L, a.W[2], A), b.env_left(L, b.W[2], A))
    _close(a.env_right(R, a.W[2], A), b.env_right(R, b.W[2], A))
    _close(a.env_mixed(0, L, a.W[2], A, A), b.env_mixed(0, L, b.W[2], A, A))
    _close(a.merge(A, A), b.merge(A, A))


def test_krylov_loops():
    a, b = _two()
    chi = 300
    w = a.W[2].shape[0]
    L, R, x = _rand(chi, w, chi), _rand(chi, w, chi), _rand(chi, 2, 2, chi)
    L, R = (L + L.permute(2, 1, 0)).contiguous() / chi, (R + R.permute(2, 1, 0)).contiguous() / chi
    e, v = [], []
    for eng in (a, b):
        y = x.clone()
        e.append(eng.ground(eng.heff2(L, eng.W[2], eng.W[3], R, x.shape), y, 200)[0])
        z = x.clone() / x.norm()
        eng.expm(eng.heff2(L, eng.W[2], eng.W[3], R, x.shape), z, -0.01, 20)
        v.append(z)
    assert abs(e[0] - e[1]) <= 1e-11 * abs(e[0])
    _close(*v, tol=1e-8)


def test_prepared_matvec_and_status():
    import torch
    from dmrgpy_gb300 import _lib
    a, b = _two()
    chi = 300
    w = a.W[2].shape[0]
    L, R, x = _rand(chi, w, chi), _rand(chi, w, chi), _rand(chi, 2, 2, chi)
    ys = []
    for e in (a, b):
        h = e.heff2(L, e.W[2], e.W[3], R, x.shape)
        ptr, size = e.ws.get(e.lib.dmrg_heff_workspace_bytes(ctypes.byref(h)))
        y = torch.empty_like(x)
        r = ctypes.byref(h)
        _lib.check("dmrg_heff_prepare", e.lib.dmrg_heff_prepare(r, ptr, size, e.stream))
        _lib.check("dmrg_heff_apply_prepared",
                   e.lib.dmrg_heff_apply_prepared(r, x.data_ptr(), y.data_ptr(), ptr, size, e.stream))
        _lib.check("dmrg_heff_status", e.lib.dmrg_heff_status(r, ptr, size, e.stream))
        ys.append(y)
    _close(*ys)


def test_truncations():
    import torch
    a, b = _two()
    m = 520
    q = np.linalg.qr(np.random.default_rng(0).standard_normal((m, m)))[0]
    M = torch.as_tensor((q * np.exp(-10 * np.linspace(0.0, 1.0, m))) @ q[::-1].T.copy(), device="cuda")
    for absorb in (0, 1):
        o = [e.svd(M, 0.0, 300, 1, absorb) for e in (a, b)]
        assert o[0][3] == o[1][3] == 300
        assert np.max(np.abs(np.asarray(o[0][2])[:300] - np.asarray(o[1][2])[:300])) <= 1e-11
        _close(o[0][0] @ o[0][1], o[1][0] @ o[1][1])
        s = [e.subspace_split(M, 300, None, 0, absorb, 0.0) for e in (a, b)]
        assert s[0][3] == s[1][3] == 300
        lo = s[1][0] if absorb == 0 else s[1][1].T
        assert np.max(np.abs((lo.T @ lo).cpu().numpy() - np.eye(300))) <= 1e-12
