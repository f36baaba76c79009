// Kernel and launch of the boundary-input preparation (qpd_fields.h).
#include "qpd_fields.h"

#include "qpd_fields_split.h"
#include "qpd_smem.h"

namespace qpd {

// Dynamic shared memory: ramp (double) + phase index (char) + one float tile per input plane.
inline size_t fields_smem_bytes(int planes) {
    return sizeof(double) * kFT * kFPitch + sizeof(float) * (size_t)planes * kFT * kFPitch + kFT * kFPitch;
}

// LOOP: the block walks more than one chunk.  A kernel of its own for one, since the loop's registers cost it (256x256x64:
// 92 us as a loop of one, 82 us); four blocks per SM either way.
template <typename T, bool LOOP>
__global__ void __launch_bounds__(kFT * kFRows, LOOP ? 4 : 0) fields_kernel(const __grid_constant__ FieldsArgs<T> a,
                                                                            long long first, long long per) {
    extern __shared__ __align__(128) unsigned char fsm[];
    double* ramp = reinterpret_cast<double*>(fsm);                        // [z][column]
    float* tiles = reinterpret_cast<float*>(ramp + kFT * kFPitch);        // [plane][z][column]
    __shared__ double sdc[kMaxMaterials + 1];      // one more entry for layers outside the stack or the tables
    __shared__ signed char spo[kMaxMaterials + 1];
    const int nU = a.u[0] ? 3 : 0, nW = a.phase ? a.nPhase : 0, nR = a.region ? 1 : 0;
    const int planes = a.nStruc + nU + nW + nR;
    signed char* pidx = reinterpret_cast<signed char*>(tiles + (size_t)planes * kFT * kFPitch);

    const int tx = threadIdx.x, ty = threadIdx.y;
    const long long plane_xy = a.nx * a.ny, c0 = (long long)blockIdx.x * kFT, c = c0 + tx;
    const long long n = plane_xy * a.nz;
    // the layers of this block's chunks: zbeg and the one past them
    const long long zbeg = (first + blockIdx.y * (LOOP ? per : 1)) * kFT, ztop = a.z0 + a.nz;
    const long long zmine = zbeg + (LOOP ? per : 1) * kFT, zend = zmine < ztop ? zmine : ztop;
    unsigned int f = 0;
    for (int i = ty * kFT + tx; i < a.nMat; i += kFT * kFRows) {
        sdc[i] = a.dc[i];
        spo[i] = a.phase_of[i];
    }
    if (tx == 0 && ty == 0) {
        sdc[kMaxMaterials] = 0.0;
        spo[kMaxMaterials] = -1;
    }
    __syncthreads();

    double run = 0.0;  // column sum of the layers so far (warp 0)
    for (long long zc = zbeg;;) {
        if (ty == 0) {
            // 1. ramp: one lane per column, layers in order (numpy.cumsum's summation order), the first chunk's from layer 0
            // on; the materials of the next 32 layers are on their way while the sum runs over the current ones
            const signed char* mat = a.mat + c;
            const long long zlast = c < plane_xy ? zend : 0;
            int next[kFT], m[kFT];
            auto fetch = [&](long long z) {
#pragma unroll
                for (int i = 0; i < kFT; i++) next[i] = z + i < zlast ? (int)mat[(z + i) * plane_xy] : 256;
            };
            auto take = [&]() {  // table entries of the 32 layers; 256 marks a layer that is not summed
#pragma unroll
                for (int i = 0; i < kFT; i++) {
                    m[i] = next[i];
                    if (m[i] < 0 || m[i] >= a.nMat) {
                        f |= m[i] != 256 ? kFlagBadMaterial : 0u;
                        m[i] = kMaxMaterials;
                    }
                }
            };
            long long z = LOOP && zc != zbeg ? zc : 0;
            fetch(z);
#pragma unroll 1
            for (; z < zc; z += kFT) {
                take();
                fetch(z + kFT);
                double d[kFT];
#pragma unroll
                for (int i = 0; i < kFT; i++) d[i] = sdc[m[i]];
#pragma unroll
                for (int i = 0; i < kFT; i++) run = __dadd_rn(run, d[i]);
            }
            take();
#pragma unroll
            for (int i = 0; i < kFT; i++) {
                const double d = sdc[m[i]];
                run = __dadd_rn(run, d);
                ramp[i * kFPitch + tx] = __dmul_rn(__dadd_rn(run, -0.5 * d), a.dz);
                pidx[i * kFPitch + tx] = spo[m[i]];
            }
        } else {
            // 2. the chunk's cropped input planes, columns fastest; a layer's planes are all in flight before the first
            // is stored
            for (int zz = ty - 1; zz < kFT; zz += kFRows - 1) {
                const long long zl = zc + zz - a.z0;
                const bool in = zl >= 0 && zl < a.nz && c < plane_xy;
                const long long off = zl * plane_xy + c;
                float v[7 + kMaxPhases];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    v[k] = in && k < a.nStruc ? a.P[k][off] : 0.f;
                    v[3 + k] = in && nU ? a.u[k][off] : 0.f;
                }
                v[6] = in && nR ? a.region[off] : 0.f;
#pragma unroll
                for (int k = 0; k < kMaxPhases; k++) v[7 + k] = in && k < nW ? a.phase[k * n + off] : 0.f;
                float* row = tiles + zz * kFPitch + tx;
                constexpr int plane = kFT * kFPitch;
                int q = 0;
#pragma unroll
                for (int k = 0; k < 3; k++)
                    if (k < a.nStruc) row[q++ * plane] = v[k];
#pragma unroll
                for (int k = 0; k < 3; k++)
                    if (nU) row[q++ * plane] = v[3 + k];
#pragma unroll
                for (int k = 0; k < kMaxPhases; k++)
                    if (k < nW) row[q++ * plane] = v[7 + k];
                if (nR) row[q * plane] = v[6];
            }
        }
        __syncthreads();
        // 3. cropped layers, z fastest: lane = layer, rows = columns
        const int zz = tx;
        const long long zl = zc + zz - a.z0;
        for (int xx = ty; xx < kFT; xx += kFRows) {
            const long long col = c0 + xx;
            if (zl < 0 || zl >= a.nz || col >= plane_xy) continue;
            const long long y = col / a.nx;
            const long long g = ((col - y * a.nx) * a.ny + y) * a.nz + zl;
            const int t = zz * kFPitch + xx;
            int q = 0;
            for (int k = 0; k < 3; k++)
                a.Pout[k * n + g] = k < a.nStruc ? T(__dmul_rn(a.p_scale, (double)tiles[(q + k) * kFT * kFPitch + t])) : T(0);
            q += a.nStruc;
            for (int k = 0; k < 3; k++) {  // rounded products and sums, no contraction: as numpy
                double v = nU ? __dmul_rn((double)tiles[(q + k) * kFT * kFPitch + t], a.u_scale) : 0.0;
                if (k == 2) v = __dadd_rn(v, ramp[t]);
                a.Uout[k * n + g] = T(v);
            }
            q += nU;
            const int p = pidx[t];
            const double r = p >= 0 ? (nR ? (double)tiles[(q + nW) * kFT * kFPitch + t] : 1.0) : 0.0;
            if (a.wdense) {
                for (int k = 0; k < a.nPhase; k++) {
                    const double o = nW ? (double)tiles[(q + k) * kFT * kFPitch + t] : (k == p ? 1.0 : 0.0);
                    a.wdense[k * n + g] = T(o * r);
                }
            } else {
                int which = -1;
                double w = 0.0;
                for (int k = 0; k < a.nPhase; k++) {
                    const double o = nW ? (double)tiles[(q + k) * kFT * kFPitch + t] : (k == p ? 1.0 : 0.0);
                    const double wp = o * r;
                    if (wp != 0.0) {
                        if (which >= 0) f |= 1u;
                        else {
                            which = k;
                            w = wp;
                        }
                    }
                }
                if (which >= 0 && w != 1.0) f |= 2u;
                a.phase_idx[g] = (signed char)which;
                a.weight[g] = T(w);
            }
        }
        zc += kFT;
        if (!LOOP || zc >= zend) break;
        __syncthreads();
    }
    if (f) atomicOr(a.flags, f);
}

template <typename T> cudaError_t launch_fields(const FieldsArgs<T>& a, cudaStream_t st) {
    const int planes = a.nStruc + (a.u[0] ? 3 : 0) + (a.phase ? a.nPhase : 0) + (a.region ? 1 : 0);
    const size_t smem = fields_smem_bytes(planes);
    const long long cols = (a.nx * a.ny + kFT - 1) / kFT;
    const FieldsSplit l = fields_split(cols, a.z0, a.nz, kFieldsBlocks);
    if (cols > 0x7fffffffLL || l.groups > 65535) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)cols, (unsigned)l.groups), block(kFT, kFRows);
    const cudaError_t e = l.per > 1 ? allow_smem<fields_kernel<T, true>>(smem) : allow_smem<fields_kernel<T, false>>(smem);
    if (e != cudaSuccess) return e;
    if (l.per > 1) fields_kernel<T, true><<<grid, block, smem, st>>>(a, l.first, l.per);
    else fields_kernel<T, false><<<grid, block, smem, st>>>(a, l.first, l.per);
    return cudaGetLastError();
}

template cudaError_t launch_fields<float>(const FieldsArgs<float>&, cudaStream_t);
template cudaError_t launch_fields<double>(const FieldsArgs<double>&, cudaStream_t);

}  // namespace qpd
