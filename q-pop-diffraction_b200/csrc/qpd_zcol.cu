// Instantiations and launch of the float32 z stage (qpd_zcol.cuh).
#include <algorithm>

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
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
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

cudaError_t launch_zcol(const ZArgs<float>& a, int cta_tiles, int sms, size_t smem_max, cudaStream_t st, bool* done) {
    *done = false;
    if (a.in.wdense || a.yfast) return cudaSuccess;
    switch (a.nz) {
        case 32: return pick<4, 8, 16, 3>(a, cta_tiles, sms, smem_max, st, done);
        case 64: return pick<4, 16, 4, 9>(a, cta_tiles, sms, smem_max, st, done);
        case 68: return pick<4, 17, 7, 4>(a, cta_tiles, sms, smem_max, st, done);
        case 104: return pick<8, 13, 4, 4>(a, cta_tiles, sms, smem_max, st, done);
        case 128: return pick<8, 16, 4, 4>(a, cta_tiles, sms, smem_max, st, done);
    }
    return cudaSuccess;
}

}  // namespace qpd
