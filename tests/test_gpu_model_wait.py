"""A device-side wait that ran out in a call which reads nothing back (forward_device,
rollout_device) is reported by the model's next call with host results, whichever it
is, and once: eager and replayed forward and step calls, and rollouts."""

import ctypes as C

import numpy as np
import pytest

from jacobi2000_gb300 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calls_before", [0, 3])
@pytest.mark.parametrize("precision", [engine.FP32, engine.BF16])
@pytest.mark.parametrize("call", ["forward", "step", "rollout"])
def test_next_host_call_reports_an_unread_timeout(pt_tiny, call, precision, calls_before):
    L = engine.load_library()
    L.jc_selftest_model_wait.argtypes = [C.c_void_p, C.c_uint32]
    L.jc_selftest_model_wait.restype = C.c_int
    x, meta = pt_tiny["ref"]["state"], pt_tiny["ref"]["meta"]
    with engine.Model.from_bytes(pt_tiny["st_bytes"], pt_tiny["config"], precision) as m:
        run = (lambda: m.rollout(x, meta, 2)[0]) if call == "rollout" else (lambda: getattr(m, call)(x, meta))
        for _ in range(calls_before):
            run()
        assert L.jc_selftest_model_wait(m._h, 1000) == 0
        with pytest.raises(engine.JcError) as e:
            run()
        assert e.value.name == "DEVICE_TIMEOUT"
        again = run()
        assert np.isfinite(again).all() and np.array_equal(again, run())
