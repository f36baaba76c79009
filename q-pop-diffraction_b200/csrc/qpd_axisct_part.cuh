// Launches of the compile-time y and x passes, instantiated by part (qpd_axisct_1.cu .. qpd_axisct_4.cu).
#pragma once

#include "qpd_axisct.cuh"
#include "qpd_axisct.h"
#include "qpd_axisct_lengths.h"
#include "qpd_smem.h"

namespace qpd {
namespace {

template <int N, int CZ, int NT, int R1, int R2, int R3, int MINB, AnyMode MODE, bool XPASS>
cudaError_t go(const CUtensorMap* map, AxisArgs<float> a, const AnyFold& f, const float2* tw, long long nouter,
               cudaStream_t st) {
    using L = AxisCt<N, CZ, NT, R1, R2, R3>;
    auto k = axis_ct<N, CZ, NT, R1, R2, R3, MINB, MODE, XPASS>;
    a.Cz = CZ;
    a.nzc = (a.nz + CZ - 1) / CZ;
    const long long grid = nouter * a.nzc;
    if ((!map && !ct_odd_nz(N)) || grid < 1 || grid > 0x7fffffffLL || f.n < 1) return cudaErrorInvalidValue;
    cudaError_t e = allow_smem<axis_ct<N, CZ, NT, R1, R2, R3, MINB, MODE, XPASS>>(L::SMEM);
    if (e != cudaSuccess) return e;
    k<<<(unsigned)grid, NT, L::SMEM, st>>>(map ? *map : CUtensorMap{}, a, f, tw, map != nullptr);
    return cudaGetLastError();
}

template <int N, int CZ, int NT, int R1, int R2, int R3, int MINB>
cudaError_t pick(const CUtensorMap* map, const AxisArgs<float>& a, const AnyFold& f, const float2* tw, AnyMode mode,
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

#define QPD_GO(LEN, CZ, NT, RA, RB, RC, MINB) \
    case LEN: return pick<LEN, CZ, NT, RA, RB, RC, MINB>(map, a, f, tw, mode, xpass, nouter, st);
#define QPD_AXIS_CT_PART(NAME, LIST)                                                                               \
    cudaError_t NAME(const CUtensorMap* map, const AxisArgs<float>& a, const AnyFold& f, const float2* tw,        \
                     AnyMode mode, bool xpass, long long nouter, cudaStream_t st) {                                \
        switch (a.N) { LIST(QPD_GO) }                                                                              \
        return cudaErrorInvalidValue;                                                                              \
    }

}  // namespace qpd
