"""Head widths that the BF16 path has no attention for are refused by every call, with
or without autotuning, before anything is launched."""

import numpy as np
import pytest

from jacobi2000_gb300 import engine
from jacobi2000_gb300.checkpoint import meta_of, parse_config, synthetic_family, write_safetensors_bytes
from jacobi2000_gb300.ic import random_drops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuning", [True, False])
@pytest.mark.parametrize("dim,heads", [(96, 4), (160, 4), (64, 16)])
def test_other_head_widths_are_refused(dim, heads, tuning, pt_tiny):
    t, cj = synthetic_family(dim, 1, 0, [32], heads=heads)[(32, 32)]
    cfg = parse_config(cj, t)
    x, meta = random_drops(cfg, seed=0), meta_of(cfg)
    before = engine.autotune(tuning)
    try:
        with engine.Model.from_bytes(write_safetensors_bytes(t), cj, engine.BF16) as m:
            for call in (lambda: m.forward(x, meta), lambda: m.step(x, meta), lambda: m.rollout(x, meta, 1)):
                with pytest.raises(engine.JcError) as e:
                    call()
                assert e.value.name == "LIMIT"
    finally:
        engine.autotune(before)
    with engine.Model.from_bytes(pt_tiny["st_bytes"], pt_tiny["config"], engine.BF16) as m:
        assert np.isfinite(m.forward(pt_tiny["ref"]["state"], pt_tiny["ref"]["meta"])).all()
