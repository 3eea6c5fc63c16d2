"""CPU: how many substeps a run launches when substeps overflow the incremental sort (SortBackoff in engine.h, compiled here): every
pattern of overflows stays within a small multiple of the substeps asked for."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include "ziran2020_gb300/csrc/engine.h"
#include <algorithm>
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv)
{
    // substep i overflows when it sorts incrementally and i % period < width (the substeps a run does in full cannot)
    const int n = std::atoi(argv[1]), period = std::atoi(argv[2]), width = std::atoi(argv[3]);
    zr::SortBackoff b;
    long done = 0, launched = 0, rounds = 0;
    bool stale = true;
    while (done < n) {
        const int todo = std::min<long>(n - done, b.limit), full = std::min(todo, std::max(b.full, stale ? 1 : 0));
        launched += todo;
        rounds++;
        int k = full;
        while (k < todo && (done + k) % period >= width) k++;
        done += k;
        stale = k < todo;
        if (k < todo) b.overflowed(k);
        else b.finished();
    }
    std::printf("%ld %ld\n", launched, rounds);
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("backoff")
    src = d / "backoff.cpp"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", ROOT, str(src), "-o", str(d / "backoff")])
    return lambda *a: [int(w) for w in subprocess.check_output([str(d / "backoff")] + [str(v) for v in a], text=True).split()]


@pytest.mark.parametrize("n", [1, 2, 7, 40, 1000, 20000])
@pytest.mark.parametrize("period, width", [(1, 1), (2, 1), (3, 2), (5, 1), (17, 1), (64, 48), (1000, 1), (1000, 500), (7, 0)])
def test_launches_are_linear(run, n, period, width):
    launched, rounds = run(n, period, width)
    # the first launch takes the whole run; after it a round leaves at most its limit unfinished: 8, or twice what it finished
    assert launched <= n + 8 * n
    if width == 0:
        assert launched == n and rounds == 1
    if period == 1:
        assert launched <= 4 * n + 8 and rounds <= n.bit_length() + 2
