"""The FP64 element kernel's bounded wait for its geometry: a warp whose lanes
see different things near the limit gives up as a whole."""
import ctypes as C

import pytest

from nimblesm_gb300 import engine as E


@pytest.mark.gpu
def test_a_warp_gives_up_as_a_whole():
    from nimblesm_gb300 import build as B
    B.build()
    lanes = C.c_int(-1)
    for limit_us in (100, 1000):
        assert E.library().nsm_warp_wait_selftest(limit_us, C.byref(lanes)) == 0
        assert lanes.value == 0
