"""GPU, FP64: the payload buffer of a split P2G form is made when the schedule is set (or with the scene), never inside a step,
so a step cannot be the call that finds the memory short."""
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused, chunk, nbuf", [(0, 256, 1), (3, 128, 2)])
@pytest.mark.parametrize("implicit", [False, True])
def test_steps_allocate_nothing(fused, chunk, nbuf, implicit):
    d = scenes.aniso_slab(size=(0.1, 0.05, 0.1), implicit=implicit)
    late = scenes.gpu_scene(d, zr.F64)  # the schedule set after the first substeps
    late.set_autotune(0)
    late.step(2)
    default = late.stats()["device_bytes"]
    late.set_schedule(chunk, nbuf, 2, 64, fused=fused)
    with_payload = late.stats()["device_bytes"]
    assert with_payload > default
    late.step(2)
    assert late.stats()["device_bytes"] == with_payload
    early = scenes.gpu_scene(d, zr.F64)  # before them
    early.set_schedule(chunk, nbuf, 2, 64, fused=fused)
    early.step(2)
    assert early.stats()["device_bytes"] == with_payload
