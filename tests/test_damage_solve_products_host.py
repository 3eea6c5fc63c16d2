"""CPU: the shares of p . A p that the implicit damage solve sums in FP64 (physics.cuh compiled as host C++), from FP32 values:
every product is an FP64 one. An FP32 product is off by 2^-25 and more of itself; an FP64 sum of a few terms by 2^-50 at most."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpu_physics", "precision_shim.cpp")


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("products") / "libprecision_shim.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", SRC, "-o", so])
    L = C.CDLL(so)
    for name, n in (("shim_gradient_share", 4), ("shim_diagonal_share", 2)):
        getattr(L, name).restype = C.c_double
        getattr(L, name).argtypes = [C.c_float] * n
    return L


@pytest.mark.parametrize("scale", [1e-12, 1.0, 1e6])
def test_products_are_taken_in_fp64(shim, scale):
    rng = np.random.default_rng(3)
    worst = 0.0
    for _ in range(200):
        s, g0, g1, g2 = (np.float32(v) for v in rng.normal(size=4) * scale)
        s64, g64 = float(s), np.array([g0, g1, g2], dtype=np.float64)
        want = s64 * float(g64 @ g64)
        assert abs(shim.shim_gradient_share(s, g0, g1, g2) - want) <= 2.0**-50 * abs(want)
        want = s64 * float(g0) * float(g0)
        assert abs(shim.shim_diagonal_share(s, g0) - want) <= 2.0**-50 * abs(want)
        in_fp32 = float(np.float32(s * g0)) * float(g0)
        worst = max(worst, abs(in_fp32 - want) / abs(want))
    assert worst > 2.0**-26  # what an FP32 product would show
