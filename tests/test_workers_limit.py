"""
The packing threads where the system gives fewer than were asked for (an address-space limit that the stacks of 64 threads
exceed): the ones there are, and the calling thread, run every job.
"""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "q-pop-diffraction_b200" / "csrc"

PROGRAM = r"""
#include <sys/resource.h>
#include <cstdio>
#include <cstring>
#include "qpd_host.h"

int main() {
    long pages = 0;
    std::FILE* f = std::fopen("/proc/self/statm", "r");
    if (!f || std::fscanf(f, "%ld", &pages) != 1) return 4;
    std::fclose(f);
    rlimit r{};
    r.rlim_cur = r.rlim_max = (rlim_t)pages * 4096 + (192u << 20);
    if (setrlimit(RLIMIT_AS, &r) != 0) return 4;
    qpd::Workers w(64);
    std::printf("%d threads\n", w.size());
    if (w.size() >= 64) return 4;  // the limit did not bite: nothing tested
    for (int k = 0; k < 1000; k++) {
        std::atomic<int> ran{0};
        w.parallel(100, [&](int) { ran.fetch_add(1); });
        if (ran.load() != 100) return 2;
    }
    return 0;
}
"""


def test_fewer_threads_than_asked(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is needed to compile the header")
    (tmp_path / "limit.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", "-I", str(CSRC), str(tmp_path / "limit.cpp"), "-o", str(tmp_path / "limit")], check=True)
    got = subprocess.run([str(tmp_path / "limit")], capture_output=True, text=True, timeout=60)
    if got.returncode == 4:
        pytest.skip(f"no limit on the address space here: {got.stdout}")
    assert got.returncode == 0, (got.returncode, got.stdout, got.stderr)
