"""GPU, FP64: the P2G forms that read a payload from HBM are set, left and set again between steps, on a scene with the explicit
and with the implicit damage solve (whose scratch is in the same buffer); the run equals one that stays with the default
schedule (only the order of sums differs)."""
import numpy as np
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("implicit", [False, True])
def test_switching_payload_forms(implicit):
    d = scenes.aniso_slab(size=(0.1, 0.05, 0.1), sigma_c=(20.0, 2.0), pull=1.0, implicit=implicit)
    runs = []
    for forms in (None, ((3, 128, 2), (2, 256, 0), (0, 256, 1), (0, 128, 2))):
        s = scenes.gpu_scene(d, zr.F64)
        s.set_autotune(0)
        for q in range(5):
            if forms and q:
                fused, chunk, nbuf = forms[q - 1]
                s.set_schedule(chunk, nbuf, 2, 64, fused=fused, g2p_tight=0)
            s.step(3)
        runs.append(scenes.gpu_state(s))
    e = scenes.errors(runs[1], runs[0])
    assert e["x"][0] < 1e-12 and e["v"][0] < 1e-9 and e["d"][0] < 1e-9, e
