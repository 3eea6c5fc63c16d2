"""CPU: the scale of the FP64 polar iteration (physics.cuh compiled as host C++). It comes from an FP32 root, whose error
e leaves e^2 / 2 in the rotation of a step that is returned: near det X = 1, where the last step lies, the scale has to be exactly
one, also where the root is a unit off."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpu_physics", "precision_shim.cpp")
UNIT = 2.0**-23  # of an FP32 number just above one


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("scale") / "libphysics_shim.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", SRC, "-o", so])
    L = C.CDLL(so)
    L.shim_newton_scale.restype = C.c_double
    L.shim_newton_scale.argtypes = [C.c_double]
    return L


def step(X, g):
    return 0.5 * (g * X + np.linalg.inv(X).T / g)


def test_an_inexact_scale_shows_in_the_returned_rotation():
    """why: one step from the exact rotation with a scale one FP32 unit off leaves it tens of FP64 units off"""
    R, _ = np.linalg.qr(np.random.default_rng(0).normal(size=(3, 3)))
    off = np.abs(step(R, 1 + UNIT) @ step(R, 1 + UNIT).T - np.eye(3)).max()
    assert off > 1e-14
    assert np.abs(step(R, 1.0) @ step(R, 1.0).T - np.eye(3)).max() < 2e-15


def test_the_last_steps_are_unscaled(shim):
    """a root one unit off is what an exact root gives at det X one unit times three off: the scale is one there too"""
    for J in 1 + np.array([0.0, 1e-16, -1e-16, 3e-8, -3e-8, UNIT, -UNIT, 3 * UNIT, -3 * UNIT]):
        assert shim.shim_newton_scale(J) == 1.0, J


def test_earlier_steps_keep_the_scale(shim):
    for J in (1e-40, 1e-20, 0.01, 0.5, 0.999, 0.99999, 1.00001, 1.001, 2.0, 100.0, 1e20, 1e40):
        assert abs(shim.shim_newton_scale(J) * np.cbrt(J) - 1) < 2 * UNIT, J
