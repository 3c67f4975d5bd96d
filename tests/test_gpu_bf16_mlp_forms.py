"""The forms of the projection + MLP by size: the warp-specialised MLP of dims
above 128 (one to sixteen chunks, ragged row tiles) and, at dim 128, two CTAs a
tile up to half of the SMs (76 and 77 tiles of the 152). The same bits as the
chunk-after-chunk kernel, which another chunk width selects."""

import json

import numpy as np
import pytest

from jacobi2000_gb300 import engine
from jacobi2000_gb300.checkpoint import meta_of, parse_config, synthetic_family, write_safetensors_bytes
from jacobi2000_gb300.ic import random_drops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nx,ny,hidden", [(256, 4, 4, 64), (256, 44, 48, 192), (256, 60, 36, 320),
                                              (256, 100, 60, 1024), (256, 128, 128, 768), (128, 512, 304, 512),
                                              (128, 512, 308, 512)])
def test_forms_give_the_same_bits(tmp_path, monkeypatch, dim, nx, ny, hidden):
    t, cj = synthetic_family(dim, 2, 5, [], rect=[(nx, ny)])[(nx, ny)]
    rng = np.random.default_rng(hidden)
    for i in range(2):
        t[f"blocks.{i}.ff1.weight"] = rng.uniform(-0.1, 0.1, (dim, hidden)).astype(np.float32)
        t[f"blocks.{i}.ff1.bias"] = rng.uniform(-0.1, 0.1, hidden).astype(np.float32)
        t[f"blocks.{i}.ff2.weight"] = rng.uniform(-0.05, 0.05, (hidden, dim)).astype(np.float32)
    cfg = parse_config(cj, t)
    x, meta = random_drops(cfg, seed=hidden), meta_of(cfg)
    cache, out = tmp_path / "tune.txt", {}
    monkeypatch.setenv("JC_AUTOTUNE_CACHE", str(cache))
    prev = engine.autotune(True)
    try:
        for nc in (64, 32):
            cache.write_text("".join(json.dumps({"model": f"d{dim}_l2_f{hidden}_r1_k1_g1", "rows": 1 << b, "nc": nc,
                                                 "attn_threads": 0}) + "\n" for b in range(0, 25)))
            with engine.Model.from_bytes(write_safetensors_bytes(t), cj, engine.BF16) as m:
                out[nc] = m.forward(x, meta)
    finally:
        engine.autotune(prev)
    assert np.isfinite(out[64]).all()
    np.testing.assert_array_equal(out[64], out[32])
