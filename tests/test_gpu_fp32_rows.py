"""FP32 launches around the sizes where the GEMMs change tiles (row tiles of an SM, and
the most rows of tiles that a launch has): an instance's bits are those it has alone."""

import numpy as np
import pytest

from jacobi2000_gb300 import engine
from jacobi2000_gb300.checkpoint import meta_of, parse_config, synthetic_family, write_safetensors_bytes
from jacobi2000_gb300.ic import random_drops

pytestmark = pytest.mark.gpu


# 64 x 64: 256 rows and 4096 cells an instance; 512 instances are 65,536 tiles of 32 cells
@pytest.mark.parametrize("dim,count", [(128, 7), (128, 60), (32, 511), (32, 513)])
def test_rows_do_not_depend_on_the_launch(dim, count):
    t, cj = synthetic_family(dim, 1, 5, [64])[(64, 64)]
    cfg = parse_config(cj, t)
    meta = meta_of(cfg)
    xs = [random_drops(cfg, seed=k) for k in range(3)]
    with engine.Model.from_bytes(write_safetensors_bytes(t), cj) as m:
        with engine.Batch([m], max_instances=count, max_cells=count * 4096) as b:
            res = b.rollout([(0, xs[k % 3], meta, 1) for k in range(count)])
        for k in (0, 1, 2, count - 2, count - 1):
            assert np.array_equal(res[k][0], m.rollout(xs[k % 3], meta, 1)[0]), k
