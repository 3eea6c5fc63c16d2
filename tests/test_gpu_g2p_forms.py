"""GPU: every compiled G2P form (threads per CTA, register budget, halo staged by bulk copies) launches and gives the oracle's
result, on the slab with damage and on a fibre slab. FP64: only the order of sums differs; FP32 within the schedule test's bounds."""
import numpy as np
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu
SCENES = {
    "borden": lambda: scenes.aniso_slab(size=(0.1, 0.05, 0.1), sigma_c=(20.0, 2.0), pull=1.0),
    "fibre": lambda: scenes.aniso_slab(size=(0.06, 0.03, 0.06), sigma_c=(20.0, 2.0), pull=1.0, model=zr.QR_STABLE_NEOHOOKEAN, fiber=10.0),
    "no damage": lambda: scenes.elastic_box(size=0.0625, ground=0.56, v0=(0.0, -1.0, 0.0)),
}


@pytest.mark.parametrize("name", SCENES)
@pytest.mark.parametrize("prec", [zr.F64, zr.F32])
def test_every_form_matches_the_oracle(name, prec):
    d = SCENES[name]()
    o = scenes.oracle_scene(d, 8)
    o.step(6)
    r = o.state()
    for threads in (64, 128, 256):
        for tight in (0, 1, 2, 3):
            s = scenes.gpu_scene(d, prec)
            s.set_schedule(0, 0, 2, threads, fused=2, g2p_tight=tight)
            s.step(6)
            e = scenes.errors(scenes.gpu_state(s), r)
            assert e["x"][0] < (1e-12 if prec == zr.F64 else 2e-6), (threads, tight, e)
            if d["damage"]:
                assert e["d"][0] < (1e-9 if prec == zr.F64 else 1e-3), (threads, tight, e)
