"""
The lines that the float32 z stage requests ahead (csrc/qpd_zprefetch.h) on the CPU: all of a tile's inputs, and no
address outside the arrays, which have nStruc planes of P and no more, whatever the tile and its place.
"""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "q-pop-diffraction_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <set>
#include <utility>
#include "qpd_zprefetch.h"

int main() {
    for (int nStruc = 0; nStruc <= 3; nStruc++)
        for (int cells : {16, 50, 128, 208, 272, 416, 450, 1088})
            for (long long tiles = 1; tiles <= 3; tiles++)
                for (long long t = 0; t < tiles; t++) {
                    const long long n = tiles * cells, g = t * cells, size[3] = {nStruc * n, 3 * n, n};
                    std::set<std::pair<int, long long>> lines;  // (array, 128-byte line counted from the tile's start in its plane)
                    for (int i = 0; i < qpd::prefetch_lines(cells, nStruc); i++) {
                        const qpd::PrefetchLine l = qpd::prefetch_line(i, cells, nStruc, n, g);
                        if (l.array < 0 || l.array > 2 || l.at < 0 || l.at >= size[l.array]) {
                            std::printf("nStruc %d, %d cells, tile %lld of %lld, line %d: array %d, value %lld\n", nStruc, cells, t, tiles, i, l.array, l.at);
                            return 1;
                        }
                        const long long plane = l.at / n, in = l.at % n - g;
                        if (in < 0 || in >= cells) return 2;
                        lines.insert({l.array, plane * 1000 + in * (l.array == 2 ? 1 : 4) / 128});
                    }
                    const int per = (cells * 4 + 127) / 128;
                    if ((int)lines.size() != (nStruc + 3) * per + (cells + 127) / 128) return 3;
                }
    return 0;
}
"""


def test_prefetch_stays_inside_the_inputs(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is needed to compile the header")
    (tmp_path / "lines.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), str(tmp_path / "lines.cpp"), "-o", str(tmp_path / "lines")], check=True)
    got = subprocess.run([str(tmp_path / "lines")], capture_output=True, text=True, timeout=60)
    assert got.returncode == 0, (got.returncode, got.stdout)
