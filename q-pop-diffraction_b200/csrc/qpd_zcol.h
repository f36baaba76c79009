// The float32 z stage of qpd_zcol.cuh: which lengths it covers, and its launch.
#pragma once

#include <cuda_runtime.h>

#include "qpd_kernels.cuh"

namespace qpd {

// *done is false, and nothing launched, when nz has no instantiation, the inputs carry dense weights or the tables
// do not fit.  cta_tiles > 0: at most that many tiles per CTA (qpd_set_cta_tiles).
cudaError_t launch_zcol(const ZArgs<float>& a, int cta_tiles, int sms, size_t smem_max, cudaStream_t st, bool* done);

}  // namespace qpd
