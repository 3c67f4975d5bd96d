"""Forms that a call takes by what surrounds it give the same bits: the projection of a
small grid alone (warp-sized units in registers) and beside a grid of more than 16
segments (segments in shared memory), and host calls before and after the model has a
captured graph, for inputs that the graph has not seen."""

import numpy as np
import pytest

from jacobi2000_gb300 import engine
from jacobi2000_gb300.checkpoint import meta_of, parse_config, synthetic_family, write_safetensors_bytes
from jacobi2000_gb300.ic import random_drops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(60, 68), (100, 60), (64, 128), (256, 256)])
def test_projection_forms(nx, ny):
    fam = synthetic_family(128, 1, 3, [], rect=[(nx, ny), (256, 260)])
    made = [(parse_config(cj, t), write_safetensors_bytes(t), cj) for t, cj in fam.values()]
    cfg, meta = made[0][0], meta_of(made[0][0])
    x, big = random_drops(cfg, seed=nx), random_drops(made[1][0], seed=1)
    with engine.Model.from_bytes(made[0][1], made[0][2]) as m, engine.Model.from_bytes(made[1][1], made[1][2]) as w:
        final, energies = m.rollout(x, meta, 3)[:2]
        with engine.Batch([m, w], max_instances=2, max_cells=nx * ny + 256 * 260) as b:
            res = b.rollout([(0, x, meta, 3), (1, big, meta, 3)])
    assert np.array_equal(res[0][0], final)
    assert res[0][1] == energies[-1]


@pytest.mark.parametrize("precision", [engine.FP32, engine.BF16])
def test_replayed_host_calls_take_new_inputs(precision):
    t, cj = synthetic_family(128, 1, 3, [], rect=[(36, 20)])[(36, 20)]
    cfg, raw, meta = parse_config(cj, t), write_safetensors_bytes(t), meta_of(parse_config(cj, t))
    xs = [random_drops(cfg, seed=k) for k in range(4)]

    def fresh(call, k):  # a model's first call is launched kernel by kernel
        with engine.Model.from_bytes(raw, cj, precision) as m:
            return getattr(m, call)(xs[k], meta)

    want = {(call, k): fresh(call, k) for call in ("forward", "step") for k in range(4)}
    with engine.Model.from_bytes(raw, cj, precision) as m:
        for k in (0, 1, 2, 0, 3):
            for call in ("forward", "step"):
                assert np.array_equal(getattr(m, call)(xs[k], meta), want[call, k]), (call, k)
