"""
How the layers of a stack are shared out among blocks in the field preparation (csrc/qpd_fields_split.h), on the CPU:
every chunk of the crop in one group and no group empty; wide planes sum hardly any layer twice; films keep a block per chunk.
"""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "q-pop-diffraction_b200" / "csrc"
FILL = 12 * 148

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "qpd_fields_split.h"

int main(int argc, char** argv) {
    const long long blocks = std::atoll(argv[1]);
    for (long long cols : {1, 2, 13, 40, 128, 300, 625, 1500, 1776, 2048, 8192, 500000})
        for (long long z0 : {0, 1, 31, 32, 100, 500, 2000})
            for (long long nz : {1, 20, 32, 33, 64, 68, 104, 256, 400, 1024, 4096}) {
                const qpd::FieldsSplit s = qpd::fields_split(cols, z0, nz, blocks);
                const long long end = s.first + s.chunks;
                long long next = s.first, sums = 0;  // chunks summed by all groups of a column
                for (long long g = 0; g < s.groups; g++) {
                    const long long b = s.first + g * s.per, e = b + s.per < end ? b + s.per : end;
                    if (b != next || e <= b) return 1;
                    next = e;
                    sums += e;
                }
                if (next != end || s.first * 32 > z0 || (s.first + 1) * 32 <= z0 || end * 32 < z0 + nz || (end - 1) * 32 >= z0 + nz) return 2;
                // columns that fill the device by themselves: at most half the layers again
                if (cols >= blocks && 2 * sums > 3 * end) {
                    std::printf("%lld columns, layers %lld + %lld: %lld of %lld chunks summed\n", cols, z0, nz, sums, end);
                    return 3;
                }
                // few columns: a block for every chunk
                if (cols * s.chunks <= blocks && s.groups != s.chunks) return 4;
            }
    return 0;
}
"""


def test_split(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is needed to compile the header")
    (tmp_path / "split.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), str(tmp_path / "split.cpp"), "-o", str(tmp_path / "split")], check=True)
    got = subprocess.run([str(tmp_path / "split"), str(FILL)], capture_output=True, text=True, timeout=60)
    assert got.returncode == 0, (got.returncode, got.stdout)
