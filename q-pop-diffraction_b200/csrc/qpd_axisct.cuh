// Compile-time y and x passes of the float32 fused schedule, the adjoint's included.
//
// A CTA owns a tile of N rows along the axis by CZ neighbouring z values and walks the pass's input fields; the
// next field's tile arrives by TMA while the current one is transformed in two or three Stockham stages of radix
// R1, R2 (, R3).  Stage 1 reads the tile as it landed, the last stage leaves its outputs in registers, and the
// thread that holds them folds them into its accumulators: a value crosses shared memory once per stage, and a
// field costs one barrier per stage after the first.  (axis_tma writes the last stage back, reads it again to fold
// and needs two barriers more.)
//
// Rows hold CZ values, so 16 / CZ rows share the banks of a half-warp; the first stage's outputs of neighbouring
// threads are R1 rows apart, which would be the same banks: row i of the exchange buffer sits at
// i ^ ((i / R1) mod (16 / CZ)) (odd R1 need none of it).  Later stages write neighbouring rows from neighbouring threads.
#pragma once

#include "qpd_any.h"
#include "qpd_axisct.h"
#include "qpd_fast.cuh"
#include "qpd_radix.cuh"
#include "qpd_tma.cuh"

namespace qpd {

template <int N, int CZ, int NT, int R1, int R2, int R3> struct AxisCt {
    static constexpr int RL = R3 > 1 ? R3 : R2;          // radix of the last stage
    static constexpr int JT = NT / CZ;                   // butterflies (rows of a stage) done at once
    static constexpr int Q1 = cdiv(N / R1, JT), Q2 = cdiv(N / R2, JT), QL = cdiv(N / RL, JT);  // per thread and stage
    static constexpr int EPT = QL * RL;                  // outputs per thread
    static constexpr int TILE = (N * CZ + 15) / 16 * 16;
    static constexpr int TW = R1 * any_tw_row(R2) + (R3 > 1 ? R1 * R2 * any_tw_row(R3) : 0);
    static constexpr size_t SMEM = sizeof(float2) * (3 * TILE + TW) + 128;
    static_assert(R1 * R2 * R3 == N && NT % CZ == 0, "tile");
};

// v[r] times the twiddle row w (16-byte aligned, values r = 1 ..)
template <int R> __device__ __forceinline__ void tw_row(float2 (&v)[R], const float2* w) {
#pragma unroll
    for (int r = 1; r < R; r += 2) {
        const float4 q = *reinterpret_cast<const float4*>(w + r - 1);
        v[r] = tw_mul(make_float2(q.x, q.y), v[r]);
        if (r + 1 < R) v[r + 1] = tw_mul(make_float2(q.z, q.w), v[r + 1]);
    }
}

template <int N, int CZ, int NT, int R1, int R2, int R3, int MINB, AnyMode MODE, bool XPASS>
__global__ void __launch_bounds__(NT, MINB) axis_ct(const __grid_constant__ CUtensorMap map,
                                                    const __grid_constant__ AxisArgs<float> a,
                                                    const __grid_constant__ AnyFold f, const float2* __restrict__ twg,
                                                    int tensor) {
    using L = AxisCt<N, CZ, NT, R1, R2, R3>;
    using C = float2;
    const bool tma = !ct_odd_nz(N) || tensor;
    constexpr int EPT = L::EPT, JT = L::JT, TILE = L::TILE, RL = L::RL, QL = L::QL;
    // rows that share the banks of a half-warp; stage 1's outputs of neighbouring threads meet only when R1 is even
    constexpr int SW = 16 / CZ > 1 && R1 % (16 / CZ) == 0 ? 16 / CZ - 1 : 0;
    static_assert(SW == 0 || (JT % (SW + 1) == 0 && N / R2 % R1 == 0 && N / R2 % (SW + 1) == 0), "one swizzle per thread");
    static_assert(SW == 0 || JT % (R1 * (SW + 1)) == 0 || L::Q2 == 1, "one swizzle per thread");
    constexpr int BOX = ct_rows(N, CZ * (int)sizeof(C));
    constexpr uint32_t BYTES = N * CZ * sizeof(C);
    static_assert(BOX > 0, "a tile is one box, or whole boxes of 128-byte multiples");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // Three tiles.  Three stages: inputs alternate between tiles 0 and 1, stage 1 writes tile 2, stage 2 writes back
    // into the input's.  Two stages: input i lands in tile i mod 3 and stage 1 writes tile (i + 2) mod 3, since the
    // tile that the previous input's stage 1 wrote may still be read by its stage 2.
    C* const tiles = reinterpret_cast<C*>(smem_raw);
    C* const tw = tiles + 3 * TILE;
    constexpr int RING = R3 > 1 ? 2 : 3;
    __shared__ __align__(8) uint64_t bar[2];
    const int tid = threadIdx.x;
    const int c = tid % CZ, j0 = tid / CZ;
    const int outer = blockIdx.x / a.nzc;
    const int z0 = (int)(blockIdx.x - outer * a.nzc) * CZ;
    const bool live = z0 + c < a.nz;
    if (smem_u32(smem_raw) % 128 != 0) {  // TMA destinations must be 128-byte aligned: refuse, do not load
        if (tid == 0) atomicExch(a.status, QPD_DEVERR_ALIGN);
        return;
    }
    const int nfx = (int)a.nx;
    // Input i's tile: one thread's tensor copies, or (odd nz: no tensor map has its row strides) every thread's 8-byte
    // ones; either completes bar[i & 1].
    auto issue_threads = [&](int i) {
        const C* src = a.in + (long long)f.field[i] * a.fstride + (long long)outer * a.ostride + z0 + c;
        C* dst = tiles + (i % RING) * TILE;
        if (live)
            for (int k = j0; k < N; k += JT) cp_async<sizeof(C)>(dst + k * CZ + c, src + k * a.stride);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bar[i & 1])) : "memory");
    };
    auto issue = [&](int i) {
        const int b = i & 1, fl = f.field[i];
        C* dst = tiles + (i % RING) * TILE;
        mbar_expect_tx(&bar[b], BYTES);
#pragma unroll
        for (int k = 0; k < N / BOX; k++) {
            if (XPASS) tma_load_3d(dst + k * BOX * CZ, &map, &bar[b], 2 * z0, outer, fl * nfx + k * BOX);
            else tma_load_3d(dst + k * BOX * CZ, &map, &bar[b], 2 * z0, k * BOX, fl * nfx + outer);
        }
    };
    if (tid == 0) {
        mbar_init(&bar[0], tma ? 1 : NT);
        mbar_init(&bar[1], tma ? 1 : NT);
        fence_barrier_init();
        if (tma) issue(0);
    }
    for (int i = tid; i < L::TW; i += NT) tw[i] = twg[i];
    __syncthreads();
    if (!tma) issue_threads(0);

    // row offsets of the swizzled stage-1 outputs: s and s ^ (j mod (SW + 1)) differ in the low bits only
    int wofs[SW + 1];
#pragma unroll
    for (int s = 0; s <= SW; s++) wofs[s] = (s ^ (j0 & SW)) * CZ;
    const int p2 = (j0 / R1) & SW;
    C acc[EPT];
#pragma unroll
    for (int e = 0; e < EPT; e++) acc[e] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int i = 0; i < f.n; i++) {
        C* const cur = tiles + (i % RING) * TILE;
        C* const W = tiles + (R3 > 1 ? 2 : (i + 2) % 3) * TILE;
        const C* const cf = static_cast<const C*>(f.coef[i]);
        // first output row of the thread's butterfly q (row 0 where it has none)
        auto row_of = [&](int q) { return N / RL % JT == 0 || j0 + q * JT < N / RL ? j0 + q * JT : 0; };
        // with 16 values per thread the fold's coefficients are requested before the input's tile is awaited (1024
        // points: y pass 2850 -> 2290 us at 1024x1024x68); with 8, at 64 registers, they would spill
        constexpr bool EARLY = EPT > 8 && MODE != AnyMode::Pre;
        C cfr[EARLY ? EPT : 1];
        if constexpr (EARLY) {
#pragma unroll
            for (int q = 0; q < QL; q++)
#pragma unroll
                for (int s = 0; s < RL; s++) cfr[q * RL + s] = __ldg(cf + row_of(q) + s * (N / RL));
        }
        const bool ok = mbar_wait(&bar[i & 1], (i >> 1) & 1, a.status);
        // ---- stage 1
        {
            constexpr int LR = N / R1;
#pragma unroll
            for (int q = 0; q < L::Q1; q++) {
                const int j = j0 + q * JT;  // j mod (SW + 1) = j0 mod (SW + 1)
                if (LR % JT != 0 && j >= LR) break;
                C v[R1];
#pragma unroll
                for (int r = 0; r < R1; r++) v[r] = cur[(j + r * LR) * CZ + c];
                if constexpr (MODE == AnyMode::Pre) {
#pragma unroll
                    for (int r = 0; r < R1; r++) v[r] = tw_mul(__ldg(cf + j + r * LR), v[r]);
                }
                Bfly<R1, C>::run(v);
                C* const o = W + j * R1 * CZ + c;
#pragma unroll
                for (int s = 0; s < R1; s++) o[(s & ~SW) * CZ + wofs[s & SW]] = v[s];
            }
        }
        if (!__syncthreads_and(ok)) return;  // a load never landed; no other is in flight
        // the next input's tile: its last readers (three stages: stage 3, two: stage 2 of the input before) are past
        // this barrier
        if (!tma) {
            if (i + 1 < f.n) issue_threads(i + 1);
        } else if (tid == 0 && i + 1 < f.n) {
            fence_proxy_async();
            issue(i + 1);
        }
        // ---- stage 2
        C x[EPT];
        if constexpr (L::QL * JT != N / RL) {
#pragma unroll
            for (int e = 0; e < EPT; e++) x[e] = make_float2(0.f, 0.f);
        }
        {
            constexpr int LR = N / R2;
#pragma unroll
            for (int q = 0; q < L::Q2; q++) {
                const int j = j0 + q * JT;
                if (LR % JT != 0 && j >= LR) break;
                C v[R2];
#pragma unroll
                for (int r = 0; r < R2; r++) {
                    const int turn = (r * (LR / R1)) & SW;  // LR is a multiple of R1: (j + r LR) / R1 = j / R1 + r LR / R1
                    // low bits: p2 + turn without a carry into higher bits, as both are taken mod SW + 1
                    const int sw = (p2 + turn) & SW;
                    v[r] = W[((j ^ sw) + r * LR) * CZ + c];  // LR is a multiple of SW + 1
                }
                const int k = j % R1, blk = j / R1;
                tw_row<R2>(v, tw + k * any_tw_row(R2));
                Bfly<R2, C>::run(v);
                if constexpr (R3 > 1) {
                    C* const o = cur + (blk * R1 * R2 + k) * CZ + c;
#pragma unroll
                    for (int s = 0; s < R2; s++) o[s * R1 * CZ] = v[s];
                } else {
#pragma unroll
                    for (int s = 0; s < R2; s++) x[q * R2 + s] = v[s];
                }
            }
        }
        if constexpr (R3 > 1) {
            __syncthreads();
            constexpr int LR = N / R3;
#pragma unroll
            for (int q = 0; q < QL; q++) {
                const int j = j0 + q * JT;
                if (LR % JT != 0 && j >= LR) break;
                C v[R3];
#pragma unroll
                for (int r = 0; r < R3; r++) v[r] = cur[(j + r * LR) * CZ + c];
                tw_row<R3>(v, tw + R1 * any_tw_row(R2) + j * any_tw_row(R3));
                Bfly<R3, C>::run(v);
#pragma unroll
                for (int s = 0; s < R3; s++) x[q * R3 + s] = v[s];
            }
        }
        // a thread without a butterfly at q folds zeros with the coefficients of row 0
        constexpr int LL = N / RL;
        auto has = [&](int q) { return LL % JT == 0 || j0 + q * JT < LL; };
        // ---- fold: x[q RL + s] is output row k = j0 + q JT + s N / RL
#pragma unroll
        for (int q = 0; q < QL; q++)
#pragma unroll
            for (int s = 0; s < RL; s++) {
                const int e = q * RL + s;
                if constexpr (MODE == AnyMode::Pre) acc[e] = x[e];
                else fold_fma(acc[e], EARLY ? cfr[EARLY ? e : 0] : __ldg(cf + row_of(q) + s * (N / RL)), x[e]);
            }
        if (!f.last[i]) continue;
        if (live) {
            const long long base = (long long)outer * a.ostride + z0 + c;
            if constexpr (MODE == AnyMode::Store || MODE == AnyMode::Pre) {
                C* const dst = a.out + (long long)f.out[i] * a.fstride + base;
#pragma unroll
                for (int q = 0; q < QL; q++)
#pragma unroll
                    for (int s = 0; s < RL; s++)
                        if (has(q)) dst[(j0 + q * JT + s * (N / RL)) * a.stride] = acc[q * RL + s];
            } else {
                const int ky = outer, kz = z0 + c, ny = (int)a.ny;
                const int sy = fftshift_at(ky, ny), sz = fftshift_at(kz, a.nz);
                const double syz = a.S[1][ky] * a.S[2][kz];
                C* const dst = a.out + (long long)f.out[i] * a.fstride + base;
                double gi[MODE == AnyMode::Seed ? EPT : 1];
                if constexpr (MODE == AnyMode::Seed) {  // all in flight before the first is needed
#pragma unroll
                    for (int q = 0; q < QL; q++)
#pragma unroll
                        for (int s = 0; s < RL; s++) {
                            const int k = j0 + q * JT + s * (N / RL);
                            gi[q * RL + s] = has(q) ? __ldg(a.gI + ((long long)fftshift_at(k, N) * ny + sy) * a.nz + sz) : 0.0;
                        }
                }
#pragma unroll
                for (int q = 0; q < QL; q++)
#pragma unroll
                    for (int s = 0; s < RL; s++) {
                        const int k = j0 + q * JT + s * (N / RL), e = q * RL + s;
                        if (!has(q)) continue;
                        const double S = a.S[0][k] * syz;
                        const double re = (double)acc[e].x, im = (double)acc[e].y;
                        const long long at = ((long long)fftshift_at(k, N) * ny + sy) * a.nz + sz;
                        if constexpr (MODE == AnyMode::Intensity) {
                            a.I[at] = floor_1e50(S * S * (re * re + im * im) * a.scale2);
                        } else {
                            const double S2 = S * S * a.scale2;
                            const double g = S2 * (re * re + im * im) > 1e-50 ? gi[MODE == AnyMode::Seed ? e : 0] * S2 : 0.0;
                            dst[k * a.stride] = make_float2((float)(g * re), (float)(-g * im));
                        }
                    }
            }
        }
#pragma unroll
        for (int e = 0; e < EPT; e++) acc[e] = make_float2(0.f, 0.f);
    }
}

}  // namespace qpd
