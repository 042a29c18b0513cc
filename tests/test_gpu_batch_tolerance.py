"""Batched Lanczos with captured steps: a call after one with another tolerance
on the same workspace gives what it gives on a workspace of its own."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tolerance_of_an_earlier_call_is_not_replayed():
    import torch
    from dmrgpy_gb300 import Engine, _lib
    from dmrgpy_gb300 import mpo
    terms = [(1.0 + 0j, [(op, i), (op, i + 1)]) for i in range(1, 6) for op in ("Sx", "Sy", "Sz")]
    W, _ = mpo.build_mpo([2] * 6, terms)
    eng = Engine(W, real=True, precision="fp64")
    lib, w = eng.lib, eng.W[2].shape[0]
    rng = np.random.default_rng(4)
    ops = (_lib.HeffDesc * 2)()
    keep, starts = [], []
    for p, chi in enumerate((6, 9)):
        E = rng.standard_normal((chi, w, chi))
        E = torch.as_tensor(E + E.transpose(2, 1, 0), device="cuda")
        x = torch.as_tensor(rng.standard_normal((chi, 2, 2, chi)), device="cuda")
        ops[p] = eng.heff2(E, eng.W[2], eng.W[3], E, x.shape)
        keep.append(E)
        starts.append(x)
    kmax = 24
    need = int(lib.dmrg_batch_lanczos_workspace_bytes(2, ops, kmax))

    def call(tol, work):
        xs = [x.clone() for x in starts]
        e, it = (ctypes.c_double * 2)(), (ctypes.c_int * 2)()
        ptrs = (ctypes.c_void_p * 2)(*[x.data_ptr() for x in xs])
        _lib.check("dmrg_batch_lanczos_ground", lib.dmrg_batch_lanczos_ground(
            2, ops, ptrs, kmax, tol, 1, e, it, work.data_ptr(), work.numel(), eng.stream))
        return np.array(e[:]), list(it), xs

    def fresh():
        return torch.empty(need, dtype=torch.uint8, device="cuda")

    # every beta is below 1e6: one step; then the full loop, and one step again
    one, full = call(1e6, fresh()), call(1e-12, fresh())
    assert one[1] == [1, 1] and min(full[1]) > 8
    work = fresh()
    for tol, ref in ((1e6, one), (1e-12, full), (1e6, one), (1e-12, full)):
        e, it, xs = call(tol, work)
        assert it == ref[1] and np.array_equal(e, ref[0])
        assert all(torch.equal(a, b) for a, b in zip(xs, ref[2]))
