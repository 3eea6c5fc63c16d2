"""GPU, FP64: the autotuner tries the split P2G form where it can win, in sparse scenes (P2G at 1 particle per cell 269 us split,
338 fused), and takes the fused form in dense ones (8 per cell 789 / 745, 27 per cell 1434 / 647); the payload buffer stays only
with a schedule that reads it, and the choice of a sparse scene is not taken for a dense one of the same size class."""
import numpy as np
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu


def lattice(side, per_cell):
    """side^3 cells with one particle per cell, or 27"""
    k = round(per_cell ** (1 / 3))
    dx = 1 / 96
    rng = np.random.default_rng(side)
    ax = np.arange(side * k)
    x = (np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), axis=-1).reshape(-1, 3) + rng.random((len(ax) ** 3, 3))) / k * dx + 0.2
    n = len(x)
    F = np.tile(np.eye(3).reshape(9), (n, 1)) + 0.01 * rng.standard_normal((n, 9))
    return {"dx": dx, "dt": 1e-4, "gravity": (0.0, -9.8, 0.0), "apic": 1.0, "cfl": 0.6, "domain": 100, "x": x, "v": 0.1 * rng.standard_normal((n, 3)),
            "m": np.full(n, 1000 * dx**3 / per_cell), "V0": np.full(n, dx**3 / per_cell), "F": F, "sigma_c": np.ones(n),
            "materials": [dict(model=zr.COROTATED, E=1e4, nu=0.3)], "damage": None, "objects": []}


def run(d, mode):
    s = scenes.gpu_scene(d, zr.F64)
    s.set_autotune(mode)
    s.step(8)
    return s


def payload_bytes(n):
    return 37 * 8 * ((n + n // 8 + 64 + 63) // 64 * 64)


@pytest.mark.parametrize("mode", [1, 2])
def test_the_form_follows_the_density(mode):
    sparse, dense = lattice(41, 1), lattice(14, 27)  # 68,921 and 74,088 particles: one size class (17 bits)
    a, b = run(sparse, mode), run(dense, mode)
    fixed_a, fixed_b = run(sparse, 0), run(dense, 0)
    assert a.schedule()["tuned"] and a.schedule()["fused"] == 0
    assert b.schedule()["tuned"] and b.schedule()["fused"] in (1, 2)
    for s, f in ((a, fixed_a), (b, fixed_b)):
        e = scenes.errors(scenes.gpu_state(s), scenes.gpu_state(f))
        assert e["x"][0] < 1e-12 and e["v"][0] < 1e-9, e
    held = lambda s, f: s.stats()["device_bytes"] - f.stats()["device_bytes"]
    assert payload_bytes(a.count) <= held(a, fixed_a) < payload_bytes(a.count) + 65536  # (the trials' copy of the scene parameters)
    assert 0 <= held(b, fixed_b) < 65536
    assert run(sparse, mode).schedule()["fused"] == 0  # mode 1: from the cache, with its payload
