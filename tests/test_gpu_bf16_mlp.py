"""The fused projection + MLP (dim 128) at the edges of its tiles and chunks:
hidden widths that end in a 64-column chunk, one to eight chunks, one token to
several tiles per CTA. The same bits as the separate projection and MLP kernels
(another MLP chunk width selects them), and within the BF16 form's 1e-2 of the
f64 oracle."""

import json

import numpy as np
import pytest

from helpers import field_errors
from jacobi2000_gb300 import engine
from jacobi2000_gb300.checkpoint import meta_of, parse_config, synthetic_family, write_safetensors_bytes
from jacobi2000_gb300.ic import random_drops
from oracle.oracle import OracleModel

pytestmark = pytest.mark.gpu


def _checkpoint(nx, ny, hidden, layers=2):
    t, cj = synthetic_family(128, layers, 11, [], rect=[(nx, ny)])[(nx, ny)]
    rng = np.random.default_rng(hidden)
    for i in range(layers):
        t[f"blocks.{i}.ff1.weight"] = rng.uniform(-0.1, 0.1, (128, hidden)).astype(np.float32)
        t[f"blocks.{i}.ff1.bias"] = rng.uniform(-0.1, 0.1, hidden).astype(np.float32)
        t[f"blocks.{i}.ff2.weight"] = rng.uniform(-0.05, 0.05, (hidden, 128)).astype(np.float32)
    return t, cj


@pytest.mark.parametrize("nx,ny,hidden", [(4, 4, 64), (44, 48, 128), (64, 32, 192), (44, 44, 256), (64, 64, 320),
                                          (100, 60, 448), (128, 128, 512), (36, 20, 1024)])
def test_fused_equals_separate_kernels(tmp_path, monkeypatch, nx, ny, hidden):
    t, cj = _checkpoint(nx, ny, hidden)
    cfg = parse_config(cj, t)
    x, meta = random_drops(cfg, seed=hidden), meta_of(cfg)
    prev = engine.autotune(False)
    try:
        with engine.Model.from_bytes(write_safetensors_bytes(t), cj, engine.BF16) as m:
            fused = m.forward(x, meta)
        cache = tmp_path / "tune.txt"
        key = f"d128_l2_f{hidden}_r1_k1_g1"
        cache.write_text("".join(json.dumps({"model": key, "rows": 1 << b, "nc": 32, "attn_threads": 0}) + "\n"
                                 for b in range(7, 25)))
        monkeypatch.setenv("JC_AUTOTUNE_CACHE", str(cache))
        engine.autotune(True)
        with engine.Model.from_bytes(write_safetensors_bytes(t), cj, engine.BF16) as m:
            assert np.array_equal(m.forward(x, meta), fused)
    finally:
        engine.autotune(prev)
    want = OracleModel(cfg, t).forward(x.astype(np.float64), meta.astype(np.float64), f64=True)
    assert max(field_errors(fused, want)) <= 1e-2


def test_many_tiles_per_cta_equal_alone():
    t, cj = _checkpoint(256, 256, 512)
    cfg = parse_config(cj, t)
    items = [(0, random_drops(cfg, seed=k), meta_of(cfg), 2) for k in range(17)]  # 544 tiles
    with engine.Model.from_bytes(write_safetensors_bytes(t), cj, engine.BF16) as m:
        with engine.Batch([m], max_instances=17, max_cells=17 * 65536) as b:
            res = b.rollout(items)
        for k in (0, 9, 16):
            assert np.array_equal(res[k][0], m.rollout(items[k][1], items[k][2], 2)[0]), k
