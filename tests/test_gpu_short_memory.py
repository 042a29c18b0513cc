"""FP64 engine calls where the device has no room for the operands of digit
products: they run in what the contractions themselves need, as they did
before there were such products, and give the same results to FP64 rounding
(1e-11 of the norm; chains of at most four contractions of K <= 1500)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Short:
    """A workspace on a device that grants `cap` bytes at most."""

    def __init__(self, ws, cap):
        self.ws, self.cap, self.refused = ws, cap, 0

    def get(self, need):
        import torch
        if need > self.cap:
            self.refused += 1
            raise torch.cuda.OutOfMemoryError("no room")
        return self.ws.get(need)[0], max(int(need), 256)


def test_calls_fall_back_to_the_intermediates():
    import torch
    from dmrgpy_gb300 import Engine
    from dmrgpy_gb300 import mpo
    terms = [(-1.0 + 0j, [("Sz", i), ("Sz", i + 1)]) for i in range(1, 6)] + [(0.7 + 0j, [("Sx", i)]) for i in range(1, 7)]
    W, _ = mpo.build_mpo([2] * 6, terms)
    full, short = (Engine(W, real=True, precision="fp64") for _ in range(2))
    chi, w = 300, full.W[2].shape[0]
    g = torch.Generator(device="cuda")
    g.manual_seed(5)

    def rnd(*s):
        return torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)

    L, x, A = rnd(chi, w, chi), rnd(chi, 2, 2, chi), rnd(chi, 2, chi)
    L = (L + L.permute(2, 1, 0)).contiguous() / chi
    inter = 2 * 8 * chi * w * 4 * chi          # both intermediates of the matvec

    def close(a, b, tol=1e-11):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(a)

    short.ws = _Short(short.ws, inter + 4096)
    for e in (full, short):
        e.h = e.heff2(L, e.W[2], e.W[3], L, x.shape)
    for _ in range(2):                          # the second time without asking again
        close(full.apply(full.h, x), short.apply(short.h, x))
    assert short.ws.refused == 1
    close(full.env_left(L, full.W[2], A), short.env_left(L, short.W[2], A))
    close(full.env_right(L, full.W[2], A), short.env_right(L, short.W[2], A))
    close(full.env_mixed(0, L, full.W[2], A, A), short.env_mixed(0, L, short.W[2], A, A))
    close(full.env_mixed(1, L, full.W[2], A, A), short.env_mixed(1, L, short.W[2], A, A))
    close(full.merge(A, A), short.merge(A, A))
    # Krylov loops: room for the basis and the intermediates, not for digits
    r = ctypes.byref(full.h)
    k = short._kcap(x.numel(), 200)
    lz = int(full.lib.dmrg_lanczos_workspace_bytes(r, k)) - int(full.lib.dmrg_heff_workspace_bytes(r))
    short.ws.cap, short.ws_limit = lz + inter + 4096, float("inf")
    out = []
    for e in (full, short):
        y, z = x.clone(), x / x.norm()
        out.append((e.ground(e.h, y, 200)[0], e.expm(e.h, z, -0.01, 20) and z))
    assert abs(out[0][0] - out[1][0]) <= 1e-11 * abs(out[0][0])
    close(out[0][1], out[1][1], 1e-8)
    # a split-TF32 call has no such form
    with pytest.raises(torch.cuda.OutOfMemoryError):
        t = Engine(W, real=True, precision="tf32x3")
        t.ws = _Short(t.ws, 4096)
        t.apply(t.heff2(L, t.W[2], t.W[3], L, x.shape), x)
