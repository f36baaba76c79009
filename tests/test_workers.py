"""
The packing threads of the host call (csrc/qpd_host.h) on the CPU: jobs of changing sizes one after the other, each
index run exactly once and every one of them before parallel() returns, whatever a thread of an earlier job still does.

A small C++ program around the header, under a time limit: a lost count shows as a wait that never ends.
"""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "q-pop-diffraction_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <memory>
#include "qpd_host.h"

int main(int argc, char** argv) {
    const int threads = std::atoi(argv[1]), rounds = std::atoi(argv[2]), nsizes = argc - 3;
    qpd::Workers w(threads - 1);
    for (long long r = 0; r < rounds; r++) {
        const int count = std::atoi(argv[3 + r % nsizes]);
        // the job's own counters, gone after it: a late index of an earlier job has nowhere to go unseen
        std::vector<std::atomic<int>> ran(count);
        w.parallel(count, [&](int i) {
            if (i < 0 || i >= count) std::_Exit(3);
            ran[i].fetch_add(1);
        });
        for (int i = 0; i < count; i++)
            if (ran[i].load() != 1) {
                std::printf("job %lld: index %d of %d ran %d times\n", r, i, count, ran[i].load());
                return 2;
            }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is needed to compile the header")
    where = tmp_path_factory.mktemp("workers")
    src = where / "jobs.cpp"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", "-I", str(CSRC), str(src), "-o", str(where / "jobs")], check=True)
    return where / "jobs"


# sizes as a host call makes them (packing, then the pieces of the result), alternating large and small, and no jobs
@pytest.mark.parametrize("threads,sizes", [(16, (16, 16, 16, 16, 9, 9, 9, 9, 9, 9, 9, 8)), (16, (16, 1)), (8, (8, 8, 8, 1, 5, 2)),
                                           (4, (64, 3, 1, 200, 0, 7)), (1, (5, 1))])
def test_every_index_runs_once(program, threads, sizes):
    got = subprocess.run([str(program), str(threads), "100000", *map(str, sizes)], capture_output=True, text=True, timeout=120)
    assert got.returncode == 0, got.stdout
