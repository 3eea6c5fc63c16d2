"""GPU: the incremental sort where a tile's bucket has no room for its movers, through the engine interface (tests/cpp/engine_flags.cpp),
whose report says whether a substep overflowed and was repeated."""
import os
import subprocess

import pytest

import ziran2020_gb300 as zr

pytestmark = pytest.mark.gpu
SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "engine_flags.cpp")
TOL = {8: 1e-12, 4: 1e-5}  # a few substeps of sums of ~100 terms in another order, in units of each field


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    lib = zr.library_path()
    exe = str(tmp_path_factory.mktemp("flags") / "engine_flags")
    subprocess.check_call(["g++", "-std=c++17", "-O2", SRC, "-o", exe, lib, "-Wl,-rpath," + os.path.dirname(lib)])

    def call(mode, precision, *more):
        words = subprocess.check_output([exe, mode, str(precision)] + [str(m) for m in more], text=True, timeout=300).split()
        return {k: float(v) for k, v in zip(words[::2], words[1::2])}

    return call


@pytest.mark.parametrize("precision", [8, 4])
def test_a_written_state_that_would_overflow_one_bucket_is_sorted_in_full(run, precision):
    """a twelfth of the particles moved into one place: nothing aborts, the next substep sorts in full"""
    r = run("written", precision)
    assert r["particles"] == 32768 and r["overflow"] == 0
    assert r["difference"] < TOL[precision]


@pytest.mark.parametrize("precision", [8, 4])
def test_a_body_that_overflows_in_every_substep_launches_few_empty_ones(run, precision):
    """681,472 particles (tiles of 2,048 storage indices) that move 0.25 cells along each axis per substep: every incremental sort
    overflows. The substeps launched stay within four times those asked for (they were n (n + 1) / 2), and the run equals the
    one that sorts in full."""
    r = run("fast", precision)
    assert r["particles"] == 681472 and r["overflow"] == 1 and r["done"] == 40
    assert r["launched"] <= 4 * 40
    assert r["difference"] < TOL[precision]


@pytest.mark.parametrize("precision", [8, 4])
def test_pipelined_jobs_run_again_after_an_overflow(run, precision):
    """the pipeline does not count movers; the job whose sort overflows and those behind it run the safe way"""
    r = run("stream", precision)
    assert 0 < r["reruns"] <= 6
    assert r["difference"] < TOL[precision]


@pytest.mark.parametrize("n", [599_999, 600_000, 600_001, 614_399, 614_400, 614_401])
@pytest.mark.parametrize("precision", [8, 4])
def test_large_tiles_at_their_edges(run, precision, n):
    """512-index tiles up to 600,000 particles, 2,048 above (614,400 = 300 whole ones): incremental against full sort"""
    r = run("tiles", precision, n)
    assert r["particles"] == n and r["overflow"] == 0
    assert (r["groups"], r["blocks"]) == (r["full_groups"], r["full_blocks"])
    assert r["difference"] < TOL[precision]


@pytest.mark.parametrize("n", [2048 * 4096, 2048 * 4096 + 1])
def test_more_tiles_than_a_block_copies(run, n):
    """beyond 4,096 tiles the first keys are searched in global memory"""
    r = run("tiles", 4, n)
    assert r["particles"] == n and r["overflow"] == 0
    assert (r["groups"], r["blocks"]) == (r["full_groups"], r["full_blocks"])
    assert r["difference"] < TOL[4]
