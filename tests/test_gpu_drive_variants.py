"""GPU: G2P's compiled forms by the damage a batch can have (none, on the Borden model only, any), over the mixes of scenes that
choose them. Each scene of each batch against the FP64 oracle: only the order of sums differs."""
import numpy as np
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu


def box():
    return scenes.elastic_box(size=0.0625, ground=0.56, v0=(0.0, -1.0, 0.0))


def slab(model=None, fiber=0.0, damage=True, implicit=False):
    d = scenes.aniso_slab(size=(0.06, 0.03, 0.06), sigma_c=(20.0, 2.0), pull=1.0, model=model, fiber=fiber, implicit=implicit)
    return d if damage else {**d, "damage": None, "implicit": False}


MIXES = {
    "no damage": lambda: [box()],
    "undamaged fibre slab": lambda: [slab(zr.QR_STABLE_NEOHOOKEAN, 10.0, damage=False)],
    "borden": lambda: [slab()],
    "borden beside a box": lambda: [box(), slab()],
    "borden beside an undamaged fibre slab": lambda: [slab(), slab(zr.QR_STABLE_NEOHOOKEAN, 10.0, damage=False)],
    "fibre beside borden": lambda: [slab(zr.QR_STABLE_NEOHOOKEAN, 10.0), slab()],
    "implicit borden beside a box": lambda: [slab(implicit=True), box()],
}


@pytest.mark.parametrize("mix", MIXES)
@pytest.mark.parametrize("prec", [zr.F64, zr.F32])
def test_each_scene_matches_the_oracle(mix, prec):
    descs = MIXES[mix]()
    b = zr.Batch(prec)
    for d in descs:
        b.add_scene(scenes.gpu_scene(d, prec))
    b.step(12)
    for slot, d in enumerate(descs):
        o = scenes.oracle_scene(d, 8)
        o.step(12)
        r = o.state()
        assert np.abs(b.get(slot, "x") - r["x"]).max() < (1e-12 if prec == zr.F64 else 2e-6), slot
        if d["damage"]:
            assert np.abs(b.get(slot, "d") - r["d"]).max() < (1e-9 if prec == zr.F64 else 1e-3), slot
