"""GPU: the fused P2G where a chunk's cells are crowded and are cut into pieces over the threads of an x-offset: per-cell
counts around the threshold (16), chunks of one cell, crowded cells beside sparse ones, with and without damage. FP64 against
the oracle: only the order of sums differs (positions 1e-12, velocities and F 1e-9); FP32 within the 1e-6 of the domain that
the degenerate layouts are held to, as each node sums at most ~5e3 terms of one sign more or less."""
import numpy as np
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu
DX = 1 / 64


def scene(counts, damage):
    """counts[i] particles in cell i of a 4 x 2 x 4 box of cells that straddles a block face"""
    rng = np.random.default_rng(sum(counts) + damage)
    cells = [(i, j, k) for i in range(4) for j in range(2) for k in range(4)]
    x = np.concatenate([(np.array(c) + np.array([30, 31, 30]) + rng.uniform(0, 1, (n, 3))) * DX for c, n in zip(cells, counts)])
    n = len(x)
    F = np.tile(np.eye(3).reshape(9), (n, 1)) + 0.01 * rng.standard_normal((n, 9))
    mat = dict(model=zr.NEOHOOKEAN_BORDEN if damage else zr.COROTATED, E=1e4, nu=0.3)
    return {"dx": DX, "dt": 5e-5, "gravity": (0.0, -9.8, 0.0), "apic": 1.0, "cfl": 0.6, "domain": 68, "x": x, "v": rng.uniform(-1, 1, (n, 3)),
            "m": np.full(n, 1e-3), "V0": np.full(n, DX**3 / 8), "F": F, "sigma_c": np.full(n, 60.0), "materials": [mat],
            "damage": dict(alpha=-1.0, l0=0.5 * DX, eta=0.1, zeta=1.0, residual=0.01) if damage else None, "objects": []}


LAYOUTS = {"16 per cell": [16] * 32, "17 per cell": [17] * 32, "27 per cell": [27] * 32, "one full cell": [3000] + [0] * 31,
           "crowded among sparse": [300 if i % 5 == 0 else i % 3 for i in range(32)], "uneven": [(37 * i) % 101 for i in range(32)]}


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("damage", [0, 1])
@pytest.mark.parametrize("prec, fused", [(zr.F64, 1), (zr.F64, 2), (zr.F32, 1), (zr.F32, 2)])
def test_crowded_cells_match_the_oracle(layout, damage, prec, fused):
    d = scene(LAYOUTS[layout], damage)
    s = scenes.gpu_scene(d, prec)
    s.set_schedule(512, 0, 2, 128, fused=fused)
    s.step(4)
    o = scenes.oracle_scene(d, 8)
    o.step(4)
    e = scenes.errors(scenes.gpu_state(s), o.state())
    if prec == zr.F64:
        assert e["x"][0] < 1e-12 and e["v"][0] < 1e-9 and e["F"][0] < 1e-9 and e["d"][0] < 1e-9, e
    else:
        assert e["x"][0] < 1e-6, e
