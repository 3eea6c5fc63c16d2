"""CPU: the server's estimate of a request's device memory counts every array of a particle and of a grid block slot. A request whose estimate is one
byte above the budget is refused when it is submitted; no device is needed for that."""
import pytest

import ziran2020_gb300 as zr


def estimate(prec, n):
    s, nodes = (8, 32) if prec == zr.F64 else (4, 64)
    particle = 2 * (30 * s + 4) + 28 + (41 if prec == zr.F64 else 27) * s * 9 / 8 + 24  # pools, keys, largest payload, sort lists
    # node fields (6 accumulators, 4 velocities); two neighbour lists, item, block key; 8 hash entries: key, value, open range
    slot = 10 * nodes * s + 32 + 32 + 16 + 8 + 8 * (8 + 4 + 8)
    return n * particle + 8 * (n / (nodes * 4) + 64) * slot


@pytest.mark.parametrize("prec", [zr.F32, zr.F64])
def test_the_estimate_counts_every_array(prec):
    r = zr.recipe(zr.RECIPE_ELASTIC_BOX, size=(0.125, 0.125, 0.125))
    need = estimate(prec, zr.recipe_count(r))
    with pytest.raises(zr.ZrError) as e:
        zr.Server(prec, budget_bytes=need - 1).submit(r, 10)
    assert e.value.code == zr.ZR_ERR_BUDGET
    zr.Server(prec, budget_bytes=need + 1).submit(r, 10)
