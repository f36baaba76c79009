// Runtime-length passes (qpd_any.cuh) behind the fused schedule and its adjoint: any axis whose length is a product
// of factors up to 17 and whose tile fits shared memory.  (The plain schedule runs the general kernels.)
#pragma once

#include <cuda_runtime.h>

#include "qpd_kernels.cuh"

namespace qpd {

// Inputs of one pass: the size of the list that travels as a kernel parameter.  A crystal of more than 21 distinct
// (R_x, R_y) has more in its y pass, which the kernels of qpd_fast.cuh and qpd_kernels.cuh run then.
constexpr int kAnyInputs = 64;
constexpr int kAnyStages = 8;
// The longest axes that their tiles hold: one pencil of 8192 values (y and x), one column of 512 threads x 4 cells (z).
constexpr int kAnyTile = 8192, kAnyColumn = 2048;

// Stages of one axis, radices up to 17, and its twiddles on the device in the order the stages read them: for
// each stage after the first and each k < Ns the row exp(-2 pi i r k / (Ns R)), r = 1 .. R - 1, padded to an
// even number of values (any_twiddles), so that a butterfly reads its row with 16-byte loads.
struct AnyStages {
    int N = 0, n = 0;
    int R[kAnyStages] = {};
    int ntw = 0;              // complex values of the table
    const void* tw = nullptr;
};
__host__ __device__ constexpr int any_tw_row(int R) { return R / 2 * 2; }

// Fill p for length N; false when N has a prime factor above 17 or needs too many stages.
bool any_stages(long long N, AnyStages* p);
void any_twiddles(const AnyStages& p, double2* tw);  // ntw values

// The inputs of one pass in segment order: input i is field[i] times coef[i][k], and closes the output out[i]
// when last[i]; n = 0: not a pass that these kernels take.
struct AnyFold {
    int n = 0;
    short field[kAnyInputs];
    short out[kAnyInputs];
    signed char last[kAnyInputs];
    const void* coef[kAnyInputs];  // complex values in the pass's precision
};

enum class AnyMode { Store, Intensity, Seed, Pre };

// y or x pass of nouter * nin pencils: pencil P is element (P / nin) * ostride + P % nin of a field, its values
// a.stride apart.  Store / Intensity / Seed fold after the transform (axis_kernel's EPI 0, 1, 2); Pre multiplies
// before it (adj_axis_kernel).  *done is false, and nothing launched, when the length or the tile is not covered.
template <typename T>
cudaError_t launch_axis_any(const AxisArgs<T>& a, const AnyFold& f, const AnyStages& st, AnyMode mode,
                            long long nouter, long long nin, int sms, size_t smem_max, cudaStream_t stream, bool* done);

// Fused z stage, and the adjoint's z stage with the source transpose.
template <typename T>
cudaError_t launch_z_any(const ZArgs<T>& a, const AnyStages& st, int sms, size_t smem_max, cudaStream_t stream,
                         bool* done);
template <typename T>
cudaError_t launch_adjz_any(const AdjZArgs<T>& a, const AnyStages& st, int sms, size_t smem_max, cudaStream_t stream,
                            bool* done);

}  // namespace qpd
