// Compile-time y and x passes (qpd_axisct.cuh): the lengths covered, their tiles, and their launch.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "qpd_any.h"

namespace qpd {

// Rows per tensor box: the whole tile up to 256 rows (a box dimension's limit), else the largest divisor whose box of
// `row_bytes`-byte rows is a multiple of 128 bytes, since a box lands at a 128-byte aligned address.
__host__ __device__ constexpr int ct_rows(int N, int row_bytes) {
    if (N <= 256) return N;
    for (int b = 256; b > 0; b--)
        if (N % b == 0 && b * row_bytes % 128 == 0) return b;
    return 0;
}

// Whether a length's kernels also hold the loads for odd nz, where no tensor map has the row strides.  Powers of two
// do not, since axis_fast has odd nz for them and the second path costs the first (y pass 12.8 -> 14.4 us at
// 64x64x32), nor do lengths from 512 on (745 -> 756 us at 512x512x104).
__host__ __device__ constexpr bool ct_odd_nz(int N) { return N < 512 && (N & (N - 1)) != 0; }

// Tile of a covered length: z values per tile, rows per tensor box, and the stages whose twiddle rows the pass
// reads (cz = 0: not covered).
struct AxisCtShape {
    int cz = 0, box = 0;
    bool odd_nz = false;  // loads its tiles by threads too
    AnyStages stages;
};
AxisCtShape axis_ct_shape(int64_t N);

// y pass (xpass false, nouter = nx) or x pass (nouter = ny) over (x, y, z) fields; map: the field array in boxes of
// (2 cz, box, 1) or (2 cz, 1, box), or null (odd nz) for tiles loaded by the threads; tw: the twiddle rows of
// axis_ct_shape(N).stages.
cudaError_t launch_axis_ct(const CUtensorMap* map, const AxisArgs<float>& a, const AnyFold& f, const float2* tw,
                           AnyMode mode, bool xpass, long long nouter, cudaStream_t st);

// The same for the lengths of one part (qpd_axisct_lengths.h).
#define QPD_AXIS_CT_DECL(NAME)                                                                              \
    cudaError_t NAME(const CUtensorMap* map, const AxisArgs<float>& a, const AnyFold& f, const float2* tw, \
                     AnyMode mode, bool xpass, long long nouter, cudaStream_t st);
QPD_AXIS_CT_DECL(launch_axis_ct_1)
QPD_AXIS_CT_DECL(launch_axis_ct_2)
QPD_AXIS_CT_DECL(launch_axis_ct_3)
QPD_AXIS_CT_DECL(launch_axis_ct_4)
#undef QPD_AXIS_CT_DECL

}  // namespace qpd
