// Instantiations and launch of the float32 z stage (qpd_zcol.cuh).
#include <algorithm>

#include "qpd_smem.h"
#include "qpd_zcol.cuh"
#include "qpd_zcol.h"

namespace qpd {
namespace {

template <int N1, int N2, int M, int MINB, bool ISO>
cudaError_t go(const ZArgs<float>& a, int cta_tiles, int sms, size_t smem_max, cudaStream_t st, bool* done) {
    using L = ZCol<N1, N2, M>;
    const size_t smem = L::bytes(a.in.nPhase * a.nAtom, a.nAtom, ISO, a.in.weight != nullptr);
    *done = smem <= smem_max;
    if (!*done) return cudaSuccess;
    auto k = zcol<N1, N2, M, MINB, ISO>;
    cudaError_t e = allow_smem<zcol<N1, N2, M, MINB, ISO>>(smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, L::NT, smem);
    if (e != cudaSuccess) return e;
    const long long ntiles = (a.ncols + M - 1) / M;
    long long grid = (long long)std::max(per_sm, 1) * sms;
    if (cta_tiles > 0) grid = std::max(grid, (ntiles + cta_tiles - 1) / cta_tiles);
    grid = std::min(grid, ntiles);
    k<<<(unsigned)grid, L::NT, smem, st>>>(a);
    return cudaGetLastError();
}

template <int N1, int N2, int M, int MINB>
cudaError_t pick(const ZArgs<float>& a, int cta_tiles, int sms, size_t smem_max, cudaStream_t st, bool* done) {
    if (a.isok) return go<N1, N2, M, MINB, true>(a, cta_tiles, sms, smem_max, st, done);
    return go<N1, N2, M, MINB, false>(a, cta_tiles, sms, smem_max, st, done);
}

}  // namespace

// The lengths from 16 to 136 that are N1 N2 with N1 = 4 .. 8 and N2 = 4 .. 17, each with its cheapest factors (butterflies,
// a twiddle unless they are coprime).
#define QPD_ZCOL_LENGTHS(X) \
    X(4, 4) X(4, 5) X(4, 6) X(4, 7) X(4, 8) X(4, 9) X(4, 11) X(4, 12) X(4, 13) X(4, 15) X(4, 16) X(4, 17) \
    X(5, 5) X(5, 6) X(5, 7) X(5, 8) X(5, 9) X(5, 10) X(5, 11) X(5, 13) X(5, 14) X(5, 15) X(5, 16) X(5, 17) \
    X(6, 7) X(6, 9) X(6, 11) X(6, 13) X(6, 15) X(6, 17) \
    X(7, 7) X(7, 8) X(7, 9) X(7, 11) X(7, 12) X(7, 13) X(7, 14) X(7, 15) X(7, 16) X(7, 17) \
    X(8, 9) X(8, 11) X(8, 12) X(8, 13) X(8, 15) X(8, 16) X(8, 17)

// Columns per tile: about 128 rows of phase B (four CTAs of four warps per SM), an even number of cells.
constexpr int zcol_columns(int N1, int N2) {
    const int a = N1 == 8 ? 2 * N2 : N2, b = 4 * N1;
    int m = 128 / (a > b ? a : b);
    if (m < 1) m = 1;
    return N1 * N2 * m % 2 ? (m > 1 ? m - 1 : 2) : m;
}

cudaError_t launch_zcol(const ZArgs<float>& a, int cta_tiles, int sms, size_t smem_max, cudaStream_t st, bool* done) {
    *done = false;
    if (a.in.wdense || a.yfast) return cudaSuccess;
    switch (a.nz) {
#define QPD_ZCOL_CASE(A, B)                                                                            \
    case A * B:                                                                                        \
        return pick<A, B, zcol_columns(A, B), ZCol<A, B, zcol_columns(A, B)>::NT <= 128 ? 4 : 3>(a, cta_tiles, sms, smem_max, \
                                                                                                 st, done);
        QPD_ZCOL_LENGTHS(QPD_ZCOL_CASE)
#undef QPD_ZCOL_CASE
    }
    return cudaSuccess;
}

}  // namespace qpd
