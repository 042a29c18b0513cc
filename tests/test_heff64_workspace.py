"""Sizes (host only): a bond operator with a wide MPO keeps lists of its two
site tensors, not of their product, which for dense tensors is the larger and
takes more multiplications than the two steps."""
import ctypes

import pytest


def _need(d, w, chi=4):
    from dmrgpy_gb300 import _lib
    lib = _lib.load()
    h = _lib.HeffDesc(kind=2, dtype=_lib.REAL64, precision=_lib.PREC_FP64, chil=chi, d1=d, d2=d, chir=chi,
                      wl=w, wm=w, wr=w, L=1, W1=1, W2=1, R=1)
    return int(lib.dmrg_heff_workspace_bytes(ctypes.byref(h)))


@pytest.mark.parametrize("d,w", [(4, 32), (3, 100), (8, 6)])
def test_no_list_of_the_product_of_wide_tensors(d, w):
    assert _need(d, w) < 16 * (d * d * w) ** 2


@pytest.mark.parametrize("d,w", [(2, 5), (3, 5), (4, 6), (2, 40)])
def test_narrow_or_two_level_bonds_take_one_pass(d, w):
    assert _need(d, w) >= 16 * (d * d * w) ** 2
