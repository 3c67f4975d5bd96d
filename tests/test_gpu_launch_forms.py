"""The forms that a launch takes by its size: a model's instances alone (few
rows: two embed rows a warp, two CTAs a projection + MLP tile, one conv tile a
CTA) and in a batch of over 152 row tiles give the same bits, at grids that
leave ragged token, cell and row tiles; projections on both sides of the 16
segments that the unit form takes; host calls before and after their graph
exists."""

import numpy as np
import pytest

from helpers import field_errors
from jacobi2000_gb300 import engine
from jacobi2000_gb300.checkpoint import meta_of, parse_config, synthetic_family, write_safetensors_bytes
from jacobi2000_gb300.ic import random_drops
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu


def _family(dim, nx, ny, layers=1, seed=3):
    t, cj = synthetic_family(dim, layers, seed, [], rect=[(nx, ny)])[(nx, ny)]
    return parse_config(cj, t), t, cj, write_safetensors_bytes(t)


@pytest.mark.parametrize("dim,nx,ny,count", [(128, 64, 128, 40), (128, 100, 60, 28), (256, 68, 132, 20),
                                              (128, 36, 20, 160), (32, 36, 20, 440), (64, 132, 68, 36)])
def test_alone_equals_large_batch(dim, nx, ny, count):
    cfg, t, cj, raw = _family(dim, nx, ny)
    xs, meta = [random_drops(cfg, seed=k) for k in range(count)], meta_of(cfg)
    with engine.Model.from_bytes(raw, cj, engine.BF16) as m:
        with engine.Batch([m], max_instances=count, max_cells=count * nx * ny) as b:
            res = b.rollout([(0, x, meta, 2) for x in xs])
        for k in (0, count // 2, count - 1):
            assert np.array_equal(res[k][0], m.rollout(xs[k], meta, 2)[0]), k
        got = m.forward(xs[0], meta)
    # the BF16 form's bound on a field's error
    want = OracleModel(cfg, t).forward(xs[0].astype(np.float64), meta.astype(np.float64), f64=True)
    assert max(field_errors(got, want)) <= 1e-2


@pytest.mark.parametrize("nx,ny", [(4, 4), (60, 68), (64, 64), (64, 68), (252, 256), (256, 256), (256, 260)])
def test_projection_holds_its_bounds(nx, ny):
    """The rollout's bounds: channel 0's box mean to 1e-4, an energy violation of at most 1e-6."""
    cfg, t, cj, raw = _family(128, nx, ny)
    x, meta = random_drops(cfg, seed=nx), meta_of(cfg)
    with engine.Model.from_bytes(raw, cj, engine.FP32) as m:
        final, energies = m.rollout(x, meta, 3)[:2]
        with engine.Batch([m], max_instances=3, max_cells=3 * nx * ny) as b:
            for f in b.rollout([(0, x, meta, 3)] * 3):
                assert np.array_equal(f[0], final)
    assert abs(final[0].mean(dtype=np.float64) - x[0].mean(dtype=np.float64)) < 1e-4
    viol = np.max(np.maximum((energies[1:] - energies[:-1] * cfg.energy_r_max) / energies[:-1], 0))
    assert viol <= 1e-6


@pytest.mark.parametrize("precision", [engine.FP32, engine.BF16])
def test_host_calls_repeat(precision):
    cfg, t, cj, raw = _family(128, 36, 20)
    meta = meta_of(cfg)
    xs = [random_drops(cfg, seed=k) for k in range(3)]
    with engine.Model.from_bytes(raw, cj, precision) as m:
        first = {(f, k): (m.forward if f else m.step)(xs[k], meta) for f in (0, 1) for k in (0,)}
    with engine.Model.from_bytes(raw, cj, precision) as m:
        for k in (0, 1, 0, 2, 0):  # the first of each is eager, the others replay a graph
            f, s = m.forward(xs[k], meta), m.step(xs[k], meta)
            if k == 0:
                assert np.array_equal(f, first[1, 0]) and np.array_equal(s, first[0, 0])
            else:
                assert not np.array_equal(f, first[1, 0])
