// Instantiations and launch of the compile-time y and x passes (qpd_axisct.cuh).
#include "qpd_axisct.cuh"
#include "qpd_axisct.h"

namespace qpd {
namespace {

template <int N, int CZ, int NT, int R1, int R2, int R3, int MINB, AnyMode MODE, bool XPASS>
cudaError_t go(const CUtensorMap& map, AxisArgs<float> a, const AnyFold& f, const float2* tw, long long nouter,
               cudaStream_t st) {
    using L = AxisCt<N, CZ, NT, R1, R2, R3>;
    auto k = axis_ct<N, CZ, NT, R1, R2, R3, MINB, MODE, XPASS>;
    a.Cz = CZ;
    a.nzc = (a.nz + CZ - 1) / CZ;
    const long long grid = nouter * a.nzc;
    if (grid < 1 || grid > 0x7fffffffLL || f.n < 1) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM);
    if (e != cudaSuccess) return e;
    k<<<(unsigned)grid, NT, L::SMEM, st>>>(map, a, f, tw);
    return cudaGetLastError();
}

template <int N, int CZ, int NT, int R1, int R2, int R3, int MINB>
cudaError_t pick(const CUtensorMap& map, const AxisArgs<float>& a, const AnyFold& f, const float2* tw, AnyMode mode,
                 bool xpass, long long nouter, cudaStream_t st) {
    switch (mode) {
        case AnyMode::Store:
            if (xpass) return cudaErrorInvalidValue;
            return go<N, CZ, NT, R1, R2, R3, MINB, AnyMode::Store, false>(map, a, f, tw, nouter, st);
        case AnyMode::Intensity: return go<N, CZ, NT, R1, R2, R3, MINB, AnyMode::Intensity, true>(map, a, f, tw, nouter, st);
        case AnyMode::Seed: return go<N, CZ, NT, R1, R2, R3, MINB, AnyMode::Seed, true>(map, a, f, tw, nouter, st);
        case AnyMode::Pre:
            return xpass ? go<N, CZ, NT, R1, R2, R3, MINB, AnyMode::Pre, true>(map, a, f, tw, nouter, st)
                         : go<N, CZ, NT, R1, R2, R3, MINB, AnyMode::Pre, false>(map, a, f, tw, nouter, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

// length, z values and threads of a tile, radices, CTAs per SM that the registers leave room for
#define QPD_AXIS_CT(X)               \
    X(64, 8, 64, 8, 8, 1, 12)        \
    X(128, 8, 64, 8, 16, 1, 8)       \
    X(256, 8, 128, 16, 16, 1, 4)     \
    X(512, 8, 512, 8, 8, 8, 2)       \
    X(1024, 4, 256, 8, 8, 16, 2)

AxisCtShape axis_ct_shape(int64_t N) {
    AxisCtShape s;
#define QPD_SHAPE(LEN, CZ, NT, RA, RB, RC, MINB)                        \
    if (N == LEN) {                                                     \
        s.cz = CZ;                                                    \
        s.box = tma_rows(LEN, CZ * 8);                                  \
        s.stages.N = LEN;                                               \
        s.stages.n = RC > 1 ? 3 : 2;                                  \
        s.stages.R[0] = RA;                                           \
        s.stages.R[1] = RB;                                           \
        s.stages.R[2] = RC;                                           \
        s.stages.ntw = AxisCt<LEN, CZ, NT, RA, RB, RC>::TW;             \
    }
    QPD_AXIS_CT(QPD_SHAPE)
#undef QPD_SHAPE
    return s;
}

cudaError_t launch_axis_ct(const CUtensorMap& map, const AxisArgs<float>& a, const AnyFold& f, const float2* tw,
                           AnyMode mode, bool xpass, long long nouter, cudaStream_t st) {
#define QPD_GO(LEN, CZ, NT, RA, RB, RC, MINB) \
    if (a.N == LEN) return pick<LEN, CZ, NT, RA, RB, RC, MINB>(map, a, f, tw, mode, xpass, nouter, st);
    QPD_AXIS_CT(QPD_GO)
#undef QPD_GO
    return cudaErrorInvalidValue;
}

}  // namespace qpd
