"""The solver by size, step count and alignment, which decide the kernels and passes
of a run: the oracle's bits at widths that end inside a strip of columns, heights of
several bands of rows, odd widths, after an odd and an even number of passes, and for
states that start 4 bytes off an 8-byte boundary."""

import ctypes as C

import numpy as np
import pytest

from jacobi2000_gb300 import engine
from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

STEPS = (1, 2, 3, 5, 6, 7)


def _states(p, count, seed):
    rng = np.random.default_rng(seed)
    few = engine.sw_flat(p, min(count, 5))
    for s in few:
        engine.sw_add_drop(p, s[0], rng.uniform(0, p.nx), rng.uniform(0, p.ny), 0.08, 2.5)
        s[1:] = (0.02 * rng.standard_normal((2, p.ny, p.nx))).astype(np.float32)
    return np.ascontiguousarray(few[np.arange(count) % len(few)])


# one state; bands and strips with odd widths; narrow states; launches that fill the
# SMs many times over; the most rows
@pytest.mark.parametrize("nx,ny,count", [(64, 64, 1), (129, 75, 3), (57, 300, 2), (121, 66, 40), (18, 70, 5), (3, 9, 7),
                                         (128, 128, 48), (64, 64, 1000), (63, 64, 1000), (1, 2_200_000, 1)])
@pytest.mark.parametrize("shift", [0, 1])
def test_solver_gives_the_oracles_bits(nx, ny, count, shift):
    p = engine.JcSwParams(nx, ny, 1.0, 0.0903, 9.81, 1.0, 1e-3)
    q = O._SwParams()
    q.nx, q.ny, q.dx, q.dt, q.g, q.depth, q.nu = p.nx, p.ny, p.dx, p.dt, p.g, p.depth, p.nu
    s0 = _states(p, count, nx + ny)
    L = engine.load_library()
    engine._declare_eval(L)
    buf = torch.empty(s0.size + 1, device="cuda")
    d = buf[shift:shift + s0.size]
    for steps in STEPS:
        d.copy_(torch.from_numpy(s0).reshape(-1))
        torch.cuda.synchronize()
        engine._check(L.jc_sw_run_device(C.byref(p), d.data_ptr(), count, steps, None))
        torch.cuda.synchronize()
        got = d.cpu().numpy().reshape(s0.shape)
        for k in range(min(count, 5)):
            want = s0[k].copy()
            O.sw_steps(q, want, steps)
            for j in (k, count - 1 - (count - 1 - k) % min(count, 5)):  # the first and the last with these inputs
                np.testing.assert_array_equal(got[j], want)
