// Compile-time y and x passes (qpd_axisct.cuh): the lengths covered, their tiles, and their launch.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "qpd_any.h"

namespace qpd {

// Tile of a covered length: z values per tile, rows per tensor box, and the stages whose twiddle rows the pass
// reads (cz = 0: not covered).
struct AxisCtShape {
    int cz = 0, box = 0;
    AnyStages stages;
};
AxisCtShape axis_ct_shape(int64_t N);

// y pass (xpass false, nouter = nx) or x pass (nouter = ny) over (x, y, z) fields with even nz; map: the field array
// in boxes of (2 cz, box, 1) or (2 cz, 1, box); tw: the twiddle rows of axis_ct_shape(N).stages.
cudaError_t launch_axis_ct(const CUtensorMap& map, const AxisArgs<float>& a, const AnyFold& f, const float2* tw,
                           AnyMode mode, bool xpass, long long nouter, cudaStream_t st);

}  // namespace qpd
