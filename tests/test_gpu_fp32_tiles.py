"""FP32 forward at the edges of its kernels' tiles: grids of one token up to
past the switch to the large GEMM tiles, widths that fill no tile, head widths
with and without the four-features-a-lane attention, and a state that starts
on a 4-byte boundary. Tolerance: sums of at most 9 x 128 products in f32 through
a few layers, 1e-5 normwise per field (the reference's forward gate,
crates/engine/tests/parity.rs:43)."""

import numpy as np
import pytest

from helpers import field_errors
from jacobi2000_gb300 import engine
from jacobi2000_gb300.checkpoint import meta_of, parse_config, synthetic_family, write_safetensors_bytes
from jacobi2000_gb300.ic import random_drops
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,dim,heads", [(4, 4, 128, 4), (12, 8, 128, 4), (132, 124, 128, 4), (260, 132, 64, 4),
                                             (36, 44, 32, 4), (64, 40, 96, 3), (28, 20, 36, 3), (40, 24, 128, 2)])
def test_forward_at_tile_edges(nx, ny, dim, heads):
    t, cj = synthetic_family(dim, 2, 7, [], heads=heads, rect=[(nx, ny)])[(nx, ny)]
    cfg = parse_config(cj, t)
    x, meta = random_drops(cfg, seed=nx + ny), meta_of(cfg)
    with engine.Model.from_bytes(write_safetensors_bytes(t), cj) as m:
        got = m.forward(x, meta)
    want = OracleModel(cfg, t).forward(x, meta)
    assert max(field_errors(got, want)) <= 1e-5, field_errors(got, want)


def test_small_and_large_tiles_give_the_same_bits():
    t, cj = synthetic_family(128, 4, 0, [32])[(32, 32)]
    cfg = parse_config(cj, t)
    with engine.Model.from_bytes(write_safetensors_bytes(t), cj) as m:
        for count in (3, 12, 60):  # 192, 768 and 3840 rows a launch, 64 alone
            items = [(0, random_drops(cfg, seed=k), meta_of(cfg), 2) for k in range(count)]
            with engine.Batch([m], max_instances=count, max_cells=count * 1024) as b:
                res = b.rollout(items)
            for k in (0, count - 1):
                assert np.array_equal(res[k][0], m.rollout(items[k][1], items[k][2], 2)[0]), (count, k)


def test_state_on_a_word_boundary():
    torch = pytest.importorskip("torch")
    t, cj = synthetic_family(128, 4, 0, [32])[(32, 32)]
    cfg = parse_config(cj, t)
    x = random_drops(cfg, seed=1)
    buf = torch.zeros(x.size + 1, device="cuda")
    buf[1:] = torch.from_numpy(x).cuda().reshape(-1)
    meta, out = torch.from_numpy(meta_of(cfg)).cuda(), torch.empty(x.size, device="cuda")
    torch.cuda.synchronize()
    with engine.Model.from_bytes(write_safetensors_bytes(t), cj) as m:
        lib = engine.load_library()
        engine._check(lib.jc_forward_device(m._h, buf.data_ptr() + 4, meta.data_ptr(), out.data_ptr(), None))
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().reshape(x.shape), m.forward(x, meta_of(cfg)))
