"""The projection's waits for the sums of its cluster's other CTAs, made to run out
by a sum that is not sent: the call reports JC_DEVICE_TIMEOUT, no CTA whose sums
are not whole stores anything, and the context stays usable."""

import ctypes as C

import numpy as np
import pytest

from jacobi2000_gb300 import engine

pytestmark = pytest.mark.gpu


def _run(pass_, one_peer):
    L = engine.load_library()
    L.jc_selftest_projection_wait.argtypes = [C.c_int32, C.c_int32, C.c_uint32]
    L.jc_selftest_projection_wait.restype = C.c_int
    return engine.STATUS[L.jc_selftest_projection_wait(pass_, one_peer, 1000)], L.jc_last_error().decode()


@pytest.mark.parametrize("pass_", [0, 1, 2])
@pytest.mark.parametrize("one_peer", [0, 1])
def test_unsent_sum_times_out_and_stores_nothing(pass_, one_peer, pt_tiny):
    status, msg = _run(pass_, one_peer)
    assert status == "DEVICE_TIMEOUT", msg
    assert _run(-1, 0)[0] == "OK"  # everything sent
    with engine.Model.from_bytes(pt_tiny["st_bytes"], pt_tiny["config"]) as m:
        out = m.forward(pt_tiny["ref"]["state"], pt_tiny["ref"]["meta"])
    assert np.abs(out - pt_tiny["ref"]["forward_stencil"]).max() < 1e-5
