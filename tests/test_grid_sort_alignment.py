"""The grid-sort operators refuse arrays whose alignment their kernels' loads and stores do
not allow, before any device work (no GPU: the addresses are never read)."""
import ctypes as C

import pytest

from particles4all_b200 import _abi, _lib

NAMES = ["pos", "vel", "body", "rest", "pos_out", "vel_out", "pred_out", "body_out", "rest_out", "cell_start", "slot_out"]


def call(entry, shift, n=100, workspace=0):
    L = _lib.lib()
    g = _abi.Grid((C.c_float * 3)(0, 0, 0), 1.0, (C.c_int32 * 3)(4, 4, 4))
    ptrs = [0x10000000 + 0x10000 * k + shift.get(name, 0) for k, name in enumerate(NAMES)]
    if entry == "p4a_grid_sort":
        return L.p4a_grid_sort(C.byref(g), n, 1 / 240, 9.8, *ptrs, 0x20000000 + workspace, 1 << 20, None, None)
    return L.p4a_grid_sort_noalloc(C.byref(g), n, 1 / 240, 9.8, *ptrs, None, None)


@pytest.mark.parametrize("entry", ["p4a_grid_sort", "p4a_grid_sort_noalloc"])
@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("by", [1, 2, 4, 8])
def test_misaligned_arrays(built, entry, name, by):
    if name in ("cell_start", "slot_out") and by % 4 == 0:
        return  # allowed, and not to be run on these addresses
    assert call(entry, {name: by}) == _abi.P4A_ERR_ARG


@pytest.mark.parametrize("by", [1, 2, 4])
@pytest.mark.parametrize("n", [0, 100])
def test_misaligned_workspace(built, by, n):
    assert call("p4a_grid_sort", {}, n=n, workspace=by) == _abi.P4A_ERR_ARG
