// Compile-time y and x passes: which lengths are covered, and the dispatch to their parts (qpd_axisct_part.cuh).
#include "qpd_axisct.h"

#include "qpd_axisct_lengths.h"

namespace qpd {

AxisCtShape axis_ct_shape(int64_t N) {
    AxisCtShape s;
    switch (N) {
#define QPD_SHAPE(LEN, CZ, NT, RA, RB, RC, MINB)                                      \
    case LEN:                                                                         \
        s.cz = CZ;                                                                    \
        s.odd_nz = ct_odd_nz(LEN);                                                    \
        s.box = ct_rows(LEN, CZ * 8);                                                \
        s.stages.N = LEN;                                                             \
        s.stages.n = RC > 1 ? 3 : 2;                                                  \
        s.stages.R[0] = RA;                                                           \
        s.stages.R[1] = RB;                                                           \
        s.stages.R[2] = RC;                                                           \
        s.stages.ntw = RA * any_tw_row(RB) + (RC > 1 ? RA * RB * any_tw_row(RC) : 0); \
        break;
        QPD_AXIS_CT(QPD_SHAPE)
#undef QPD_SHAPE
    }
    return s;
}

cudaError_t launch_axis_ct(const CUtensorMap* map, const AxisArgs<float>& a, const AnyFold& f, const float2* tw,
                           AnyMode mode, bool xpass, long long nouter, cudaStream_t st) {
    switch (a.N) {
#define QPD_GO(LEN, CZ, NT, RA, RB, RC, MINB) case LEN:
        QPD_AXIS_CT_1(QPD_GO) return launch_axis_ct_1(map, a, f, tw, mode, xpass, nouter, st);
        QPD_AXIS_CT_2(QPD_GO) return launch_axis_ct_2(map, a, f, tw, mode, xpass, nouter, st);
        QPD_AXIS_CT_3(QPD_GO) return launch_axis_ct_3(map, a, f, tw, mode, xpass, nouter, st);
        QPD_AXIS_CT_4(QPD_GO) return launch_axis_ct_4(map, a, f, tw, mode, xpass, nouter, st);
#undef QPD_GO
    }
    return cudaErrorInvalidValue;
}

}  // namespace qpd
