"""GPU: a scene whose cells are so crowded that it has more work items than eight block slots per group: the grid is sized for them
when the scene is loaded, so the first substep neither aborts nor grows it (the device bytes stay what they were), and the result is
that of a grid with room to spare."""
import numpy as np
import pytest

import ziran2020_gb300 as zr

pytestmark = pytest.mark.gpu
N = 2_600_000
DX = 1 / 64


def scene(prec):
    """2.6 million particles in 8 x 8 x 8 cells: 5,079 pieces of 512 (FP32) or 10,157 of 256 (FP64), in at most 27 blocks"""
    rng = np.random.default_rng(9)
    x = (28 + 8 * rng.random((N, 3))) * DX
    s = zr.Scene(prec)
    s.set_params(DX, 5e-5, (0.0, -9.8, 0.0), 1.0, 0.6, 68)
    first = s.add_particles(x, np.full(N, 1e-6), np.full(N, DX**3 * 512 / N), v=np.zeros((N, 3)))
    s.add_corotated(first, N, 1e4, 0.3)
    return s, x


@pytest.mark.parametrize("prec", [zr.F32, zr.F64])
def test_first_substep_of_a_crowded_scene(prec):
    s, x = scene(prec)
    s.set_autotune(0)
    y = s.get("x")  # loads the scene
    assert np.abs(y - x).max() < (1e-12 if prec == zr.F64 else 1e-7)
    before = s.stats()["device_bytes"]
    s.step(1)
    assert s.stats()["device_bytes"] == before
    groups, blocks = s.last_grid()
    items = groups + N // (512 if prec == zr.F32 else 256)
    assert items > 4096 and items > 8 * groups
    # one substep from rest: every particle gains gravity's velocity, stress is zero at F = 1
    v = s.get("v")
    assert np.abs(v - np.array([0.0, -9.8 * 5e-5, 0.0])).max() < (1e-12 if prec == zr.F64 else 1e-8)
