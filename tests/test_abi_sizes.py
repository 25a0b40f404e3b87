"""Sizes that the C entries refuse before they touch the device: addresses only, no GPU needed."""
import ctypes

import pytest


@pytest.mark.parametrize("b,t,c,nh", [(1 << 16, 1 << 21, 64, 1), (1 << 16, 1 << 21, 64, 3), (1, (1 << 31) - 64, 64, 64),
                                      ((1 << 31) - 1, (1 << 31) - 64, 1, (1 << 31) - 1), (25, 1 << 23, 1, 1)])
def test_more_chunk_states_than_a_grid_holds_are_refused(b, t, c, nh):
    from retention_integration_b200 import _lib

    lib = _lib.lib()
    ok = ctypes.c_void_p(1 << 20)
    rc = lib.pr_chunk_state(0, b, t, nh, 1, 64, c, ok, ok, ok, ok, ok, 1, 0, None)
    assert rc == -1 and b"grid limit" in lib.pr_last_error()
