// Which lines of a tile's inputs the z stage (qpd_zcol.cuh) requests ahead.  Plain C++, so that the addresses can be
// checked without a GPU.
#pragma once

#ifdef __CUDACC__
#define QPD_HD __host__ __device__ __forceinline__
#else
#define QPD_HD inline
#endif

namespace qpd {

// Line i of a tile of `cells` values per plane starting at value `g`, planes of `n` values: P has nStruc planes and no
// more, U three (4-byte values), the phase index one (bytes).
struct PrefetchLine {
    int array;            // 0: P, 1: U, 2: phase
    long long at;         // its first value in that array
};
constexpr int kLineBytes = 128;

QPD_HD int prefetch_lines(int cells, int nStruc) {
    return (nStruc + 3) * ((cells * 4 + kLineBytes - 1) / kLineBytes) + (cells + kLineBytes - 1) / kLineBytes;
}
QPD_HD PrefetchLine prefetch_line(int i, int cells, int nStruc, long long n, long long g) {
    const int lines = (cells * 4 + kLineBytes - 1) / kLineBytes, k = i / lines, l = i - k * lines;
    if (k < nStruc) return {0, k * n + g + l * (kLineBytes / 4)};
    if (k < nStruc + 3) return {1, (k - nStruc) * n + g + l * (kLineBytes / 4)};
    return {2, g + (i - (nStruc + 3) * lines) * kLineBytes};
}

}  // namespace qpd
