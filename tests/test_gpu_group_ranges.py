"""GPU: the incremental sort's group ranges at the edges of its tiles (512 storage indices, 2,048 in large scenes): particle counts around whole
tiles, groups longer than a tile, tiles whose particles all move, groups that start and end with a tile. FP64 against the
oracle: only the order of sums differs."""
import numpy as np
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu
DX = 1 / 64


def scene(x, v):
    n = len(x)
    rng = np.random.default_rng(n)
    F = np.tile(np.eye(3).reshape(9), (n, 1)) + 0.01 * rng.standard_normal((n, 9))
    return {"dx": DX, "dt": 1e-4, "gravity": (0.0, -9.8, 0.0), "apic": 1.0, "cfl": 0.6, "domain": 68, "x": x, "v": v, "m": np.full(n, 1e-3),
            "V0": np.full(n, DX**3 / 8), "F": F, "sigma_c": np.ones(n), "materials": [dict(model=zr.COROTATED, E=1e4, nu=0.3)], "damage": None,
            "objects": []}


@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 2047, 2048, 2049, 4096, 6145])
@pytest.mark.parametrize("spread", [0.5, 8.0], ids=["one or two long groups", "many groups"])
def test_ranges_at_tile_edges(n, spread):
    rng = np.random.default_rng(17 * n)
    x = 0.5 + DX * spread * rng.uniform(-1, 1, (n, 3))
    v = rng.uniform(-1, 1, (n, 3)) * 20.0 + np.array([25.0, 0.0, 0.0])  # up to 0.29 cells per substep
    d = scene(x, v)
    s = scenes.gpu_scene(d, zr.F64)
    s.set_autotune(0)
    s.step(6)
    o = scenes.oracle_scene(d, 8)
    o.step(6)
    e = scenes.errors(scenes.gpu_state(s), o.state())
    assert e["x"][0] < 1e-12 and e["v"][0] < 1e-9 * np.abs(v).max() and e["F"][0] < 1e-9, e
