"""GPU: a device checkpoint taken before the implicit solve's damage drives were formed (after a load or a state write) gives the
same run again when it is restored: a frame restarted for its time step goes through it."""
import os
import subprocess

import pytest

import ziran2020_gb300 as zr

pytestmark = pytest.mark.gpu
SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "engine_flags.cpp")


@pytest.mark.parametrize("precision", [8, 4])
def test_restored_run_equals_the_first(tmp_path, precision):
    lib = zr.library_path()
    exe = str(tmp_path / "engine_flags")
    subprocess.check_call(["g++", "-std=c++17", "-O2", SRC, "-o", exe, lib, "-Wl,-rpath," + os.path.dirname(lib)])
    words = subprocess.check_output([exe, "restore", str(precision)], text=True, timeout=300).split()
    r = {k: float(v) for k, v in zip(words[::2], words[1::2])}
    assert r["damage"] > 1e-3  # there is damage to lose
    assert r["difference"] < (1e-12 if precision == 8 else 1e-5) * max(1.0, r["damage"])  # sums in another order
