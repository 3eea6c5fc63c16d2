"""GPU: the device bytes a scene reports are those it holds: a buffer that is replaced by a larger one leaves the count."""
import numpy as np
import pytest

import ziran2020_gb300 as zr
import scenes

pytestmark = pytest.mark.gpu


def test_replaced_payload_buffer_leaves_the_count():
    """FP64 keeps 4 payload fields, and 41 once a split P2G form is asked for: the count grows by 37 of them"""
    s = scenes.gpu_scene(scenes.aniso_slab(size=(0.1, 0.05, 0.1)), zr.F64)
    s.set_autotune(0)
    s.step(1)
    before = s.stats()["device_bytes"]
    s.set_schedule(256, 1, 2, 64, fused=0)
    s.step(1)
    stride = (s.count + s.count // 8 + 64 + 63) // 64 * 64  # elements of a field: a gap after every 8 particles, room for a copy
    assert s.stats()["device_bytes"] - before == (41 - 4) * 8 * stride


def test_exchanged_staging_buffers_leave_the_count():
    """host transfers of growing sizes: one staging buffer, the largest"""
    s = scenes.gpu_scene(scenes.elastic_box(size=0.125), zr.F32)
    s.set_autotune(0)
    s.step(1)
    small, large = np.zeros(s.count * 3), np.zeros((s.count, 25))
    s.get("m")
    before = s.stats()["device_bytes"]
    s.set("x", s.get("x"))
    s.get_state(large)
    assert s.stats()["device_bytes"] - before == large.nbytes - small.nbytes // 3
