"""Batched Lanczos of a few long vectors, whose steps reorthogonalise over all
SMs from some step on, against the single-problem loop (same start, same
number of steps): energies to 1e-11 of their size and vectors to 1e-6, the
convergence of an unfinished loop's Ritz vector being limited by the start,
not by rounding (40 steps each)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one problem; unequal lengths; a breakdown (n below the number of steps) beside a long one
@pytest.mark.parametrize("cplx,chis", [(False, [150]), (False, [130, 1, 90]), (True, [100]), (True, [64, 80])])
def test_few_long_problems(cplx, chis):
    import torch
    from dmrgpy_gb300 import Engine, _lib
    from dmrgpy_gb300 import mpo
    # every MPO channel Hermitian by itself, as the environments' blocks are
    terms = [(-1.0 + 0j, [("Sz", i), ("Sz", i + 1)]) for i in range(1, 6)] + [(0.7 + 0j, [("Sx", i)]) for i in range(1, 7)]
    W, _ = mpo.build_mpo([2] * 6, terms)
    eng = Engine(W, real=not cplx, precision="fp64")
    lib, w, kmax = eng.lib, eng.W[2].shape[0], 40
    rng = np.random.default_rng(8)
    ops = (_lib.HeffDesc * len(chis))()
    keep, xs = [], []
    for p, chi in enumerate(chis):
        def rnd(*s):
            v = rng.standard_normal(s)
            return v + 1j * rng.standard_normal(s) if cplx else v
        L, x = rnd(chi, w, chi), rnd(chi, 2, 2, chi)
        L = torch.as_tensor(L + L.conj().transpose(2, 1, 0), device="cuda")
        xs.append(torch.as_tensor(x, device="cuda"))
        ops[p] = eng.heff2(L, eng.W[2], eng.W[3], L, x.shape)
        keep.append(L)
    ys = [x.clone() for x in xs]
    need = int(lib.dmrg_batch_lanczos_workspace_bytes(len(chis), ops, kmax))
    work = torch.empty(need, dtype=torch.uint8, device="cuda")
    e, it = (ctypes.c_double * len(chis))(), (ctypes.c_int * len(chis))()
    for graphs in (0, 1):
        for y, x in zip(ys, xs):
            y.copy_(x)
        ptrs = (ctypes.c_void_p * len(chis))(*[y.data_ptr() for y in ys])
        _lib.check("dmrg_batch_lanczos_ground", lib.dmrg_batch_lanczos_ground(
            len(chis), ops, ptrs, kmax, 1e-14, graphs, e, it, work.data_ptr(), need, eng.stream))
        for p, x in enumerate(xs):
            ref, e1, k1 = x.clone(), ctypes.c_double(), ctypes.c_int()
            r = ctypes.byref(ops[p])
            n1 = int(lib.dmrg_lanczos_workspace_bytes(r, kmax))
            w1 = torch.empty(n1, dtype=torch.uint8, device="cuda")
            _lib.check("dmrg_lanczos_ground", lib.dmrg_lanczos_ground(
                r, ref.data_ptr(), kmax, 1e-14, ctypes.byref(e1), ctypes.byref(k1), w1.data_ptr(), n1, eng.stream))
            assert it[p] == k1.value
            assert abs(e[p] - e1.value) <= 1e-11 * abs(e1.value)
            a, b = ys[p].flatten(), ref.flatten()
            assert abs(float(torch.linalg.vector_norm(a)) - 1.0) <= 1e-12
            assert abs(abs(complex(torch.vdot(a, b))) - 1.0) <= 1e-6
