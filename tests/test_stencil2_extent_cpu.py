"""A stencil2 call that its second pass cannot take is refused before the first pass, which would write the
output; no device is needed for that."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    import __graft_entry__ as ge
    path = ge._load_build().build()
    return ge.load_package().load(path)


@pytest.mark.parametrize("r", [(1, 1), (0, 1), (1, 0), (2, 2)])
@pytest.mark.parametrize("w", [3, 8])
def test_stencil2_refuses_extents_before_writing(lib, r, w):
    weights = (ctypes.c_float * 25)(*([1.0] * 25))
    some = ctypes.c_void_p(4096)  # never read: the call is refused by its extents
    h = 65535 * 64 + 1
    st = lib.acc_stencil2d_pair(3, r[0], r[1], weights, weights, 0, None, 0, None, some, h, w, some, h + 7, w, some, None)
    assert st == 8
