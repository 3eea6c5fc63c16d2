"""GPU: a state written into a scene that has already stepped. Where more than a quarter of the particles left the key
their storage slot was sorted by, the next substep sorts in full; otherwise the incremental sort takes over from the old base. Either way the run from the written state equals the oracle's (FP64: only the order of sums differs)."""
import numpy as np
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("speed, between", [(0.5, 4), (8.0, 12), (40.0, 12)], ids=["few movers", "some movers", "all moved"])
def test_written_state_after_motion(speed, between):
    """32,768 particles: 0.5 m/s for 4 substeps moves 1% of the particles to another cell, 8 m/s
    for 12 moves about half, 40 m/s for 12 all of them."""
    d = scenes.elastic_box(size=0.25, v0=(0.0, -speed, 0.0), gravity=(0.0, 0.0, 0.0), ground=-1.0, center=(0.5, 0.7, 0.5))
    s = scenes.gpu_scene(d, zr.F64)
    s.set_autotune(0)
    start = s.get_state(np.zeros((s.count, 25)))
    s.step(between)
    s.set_state(start)
    s.step(9)
    o = scenes.oracle_scene(d, 8)
    o.step(9)
    e = scenes.errors(scenes.gpu_state(s), o.state())
    assert e["x"][0] < 1e-12 and e["v"][0] < 1e-9 and e["F"][0] < 1e-9, e
