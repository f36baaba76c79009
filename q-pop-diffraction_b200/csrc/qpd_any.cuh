// Passes for axes of any length that is a product of factors up to 17, the length known at run time.
//
// A tile is a power of two of neighbouring pencils (PC of them, value k of pencil p at k PC + p in shared
// memory), so a stage finds a butterfly's pencil with a mask, its row with a shift and its Stockham block
// with one multiplication by a reciprocal; the radix is the only thing a stage switches on, and one stage of
// radix up to 17 does the work of up to four stages of 2, 3 and 5.  Stages run out of place (one barrier and
// one butterfly in registers at a time).
//
// They are bound by instruction issue and by the latency of the stages' barriers (issue slots 55% busy, 13 warps
// per SM at 128 registers; caps of 80 and 64 registers measured slower), not by memory: 91 instructions per
// transformed value against 430 of the general kernels (150x135x75, whose lengths qpd_zcol.cuh and qpd_axisct.cuh take
// now).  One B200, float32, us, general kernels (qpd_kernels.cuh) -> here, at sizes that these take:
//   240x200x60 z stage, dense weights    889 -> 345
//   1x400x400 z stage                    87 -> 40
//   120x100x50 adjoint z stage           244 -> 82
//   x pass of Nx64x32    1080: 300 -> 105, 1536: 354 -> 134, 2000: 431 -> 207, 3000: 637 -> 297, 4096: 816 -> 480,
//                        6000: 1379 -> 959 (8192: 1801, on the general kernels: the tile exceeds 8192 values)
//   y pass of 64xNx32    1080: 907 -> 240, 2000: 1263 -> 516, 3000: 1993 -> 762, 4096: 2316 -> 1275, 5000: 3044 -> 1749
//
// The pass over y or x (axis_any) walks its input fields with the next one's tile arriving by cp.async in a
// second buffer while the current one is transformed; every thread owns one pencil and rows k0, k0 + K, ...
// of it in the copies, the fold and the stores alike, so those need no barrier of their own.
#pragma once

#include "qpd_any.h"
#include "qpd_radix.cuh"
#include "qpd_smem.h"
#include "qpd_tma.cuh"

namespace qpd {

struct AnyStageDev {
    int R, L, Ns;             // radix, N / R, product of the earlier radices
    int tw;                   // first value of the stage's twiddle rows
    unsigned magic;           // j / Ns = umulhi(j, magic) (Ns > 1)
};
struct AnyDev {
    int N, n, lp;             // length, stages, log2 of the pencils per tile
    int ntw;
    const void* tw;           // twiddle rows (AnyStages)
    AnyStageDev s[kAnyStages];
};

// One radix-R stage of every pencil of the tile, src -> dst (Stockham order).  Pencil p's row k is at
// k pitch + p.
template <typename T, int R>
__device__ __forceinline__ void any_stage(const C_t<T>* __restrict__ src, C_t<T>* __restrict__ dst,
                                          const C_t<T>* __restrict__ tw, const AnyStageDev& s, int lp, int pitch,
                                          int tid, int nt) {
    using C = C_t<T>;
    const int nb = s.L << lp;
    const int istep = s.L * pitch, ostep = s.Ns * pitch;
    for (int b = tid; b < nb; b += nt) {
        const int j = b >> lp;
        const int at = j * pitch + (b - (j << lp));
        C v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = src[at + r * istep];
        int q = j;
        if (s.Ns > 1) {
            q = (int)__umulhi((unsigned)j, s.magic);
            const C* w = tw + s.tw + (j - q * s.Ns) * any_tw_row(R);
#pragma unroll
            for (int r = 1; r < R; r += 2) {
                if constexpr (sizeof(C) == 8) {
                    const float4 ww = *reinterpret_cast<const float4*>(w + r - 1);
                    v[r] = tw_mul(cmake<C>(ww.x, ww.y), v[r]);
                    if (r + 1 < R) v[r + 1] = tw_mul(cmake<C>(ww.z, ww.w), v[r + 1]);
                } else {
                    v[r] = tw_mul(w[r - 1], v[r]);
                    if (r + 1 < R) v[r + 1] = tw_mul(w[r], v[r + 1]);
                }
            }
        }
        Bfly<R, C>::run(v);
        C* o = dst + at + q * (R - 1) * ostep;
#pragma unroll
        for (int r = 0; r < R; r++) o[r * ostep] = v[r];
    }
}

// All stages; returns the buffer that holds the result.  Ends with a barrier when there is a stage.
template <typename T>
__device__ __forceinline__ C_t<T>* any_fft(C_t<T>* a, C_t<T>* b, const C_t<T>* tw, const AnyDev& d, int lp, int pitch,
                                           int tid, int nt) {
    for (int i = 0; i < d.n; i++) {
        const AnyStageDev& s = d.s[i];
        switch (s.R) {
            case 2: any_stage<T, 2>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 3: any_stage<T, 3>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 4: any_stage<T, 4>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 5: any_stage<T, 5>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 6: any_stage<T, 6>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 7: any_stage<T, 7>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 8: any_stage<T, 8>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 9: any_stage<T, 9>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 10: any_stage<T, 10>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 11: any_stage<T, 11>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 12: any_stage<T, 12>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 13: any_stage<T, 13>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 14: any_stage<T, 14>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 15: any_stage<T, 15>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 16: any_stage<T, 16>(a, b, tw, s, lp, pitch, tid, nt); break;
            case 17: any_stage<T, 17>(a, b, tw, s, lp, pitch, tid, nt); break;
        }
        __syncthreads();
        C_t<T>* t = a;
        a = b;
        b = t;
    }
    return a;
}

template <typename T> struct AxisAny {
    AxisArgs<T> a;
    AnyFold f;
    AnyDev d;
    long long npen, nin;      // pencils; neighbouring ones before the outer index moves on
};

template <typename T, int EPT, AnyMode MODE>
__global__ void __launch_bounds__(512) axis_any(const __grid_constant__ AxisAny<T> g) {
    using C = C_t<T>;
    extern __shared__ __align__(16) unsigned char any_smem[];
    const AxisArgs<T>& a = g.a;
    const int N = g.d.N, lp = g.d.lp, PC = 1 << lp;
    C* const tw = reinterpret_cast<C*>(any_smem);
    C* const in0 = tw + g.d.ntw;
    C* const in1 = in0 + (N << lp);
    C* const work = in1 + (N << lp);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int p = tid & (PC - 1), k0 = tid >> lp, K = nt >> lp;  // nt is a multiple of PC
    const long long P = (long long)blockIdx.x * PC + p;
    const bool live = P < g.npen;
    const long long outer = live ? P / g.nin : 0;
    const long long base = live ? outer * a.ostride + (P - outer * g.nin) + k0 * a.stride : 0;  // row k0 of the pencil
    const int rows = (N - k0 + K - 1) / K;   // rows k0 + q K this thread owns, at tid + q nt of a tile
    const int nq = live ? rows : 0;
    const long long kstep = K * a.stride;
    const uint32_t ld0 = smem_u32(in0 + tid), ld1 = smem_u32(in1 + tid);
    auto load = [&](int i) {
        const C* src = a.in + (long long)g.f.field[i] * a.fstride + base;
        uint32_t d = (i & 1) ? ld1 : ld0;
#pragma unroll
        for (int q = 0; q < EPT; q++) {
            if (q < nq)
                asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"((int)sizeof(C)) : "memory");
            src += kstep;
            d += nt * sizeof(C);
        }
        cp_async_commit();
    };
    load(0);
    for (int i = tid; i < g.d.ntw; i += nt) tw[i] = static_cast<const C*>(g.d.tw)[i];

    C acc[EPT];
#pragma unroll
    for (int q = 0; q < EPT; q++) acc[q] = cmake<C>(0, 0);
    for (int i = 0; i < g.f.n; i++) {
        C* const cur = (i & 1) ? in1 : in0;
        // the other buffer's last readers passed the barrier that ended the previous input's stages, and each
        // thread overwrites only the elements that it folded itself
        if (i + 1 < g.f.n) load(i + 1);
        else cp_async_commit();
        const C* cf = static_cast<const C*>(g.f.coef[i]);
        C cfr[EPT];
#pragma unroll
        for (int q = 0; q < EPT; q++)
            if (q < rows) cfr[q] = __ldg(cf + k0 + q * K);
        cp_async_wait<1>();
        if constexpr (MODE == AnyMode::Pre) {
#pragma unroll
            for (int q = 0; q < EPT; q++)
                if (q < nq) cur[tid + q * nt] = tw_mul(cfr[q], cur[tid + q * nt]);
        }
        __syncthreads();
        const C* res = any_fft<T>(cur, work, tw, g.d, lp, PC, tid, nt) + tid;
#pragma unroll
        for (int q = 0; q < EPT; q++) {
            if (q < rows) {
                const C v = res[q * nt];
                if (MODE == AnyMode::Pre) acc[q] = cadd(acc[q], v);
                else fold_fma(acc[q], cfr[q], v);
            }
        }
        if (!g.f.last[i]) continue;
        if (live) {
            if constexpr (MODE == AnyMode::Store || MODE == AnyMode::Pre) {
                C* dst = a.out + (long long)g.f.out[i] * a.fstride + base;
#pragma unroll
                for (int q = 0; q < EPT; q++) {
                    if (q < nq) *dst = acc[q];
                    dst += kstep;
                }
            } else {  // the x pass: pencil P is (k_y, k_z) = (P / nz, P % nz)
                const int ky = (int)(P / a.nz), kz = (int)(P - (long long)ky * a.nz);
                const int nx = (int)a.nx, ny = (int)a.ny;
                const int sy = ky + ny / 2 >= ny ? ky + ny / 2 - ny : ky + ny / 2;
                const int sz = kz + a.nz / 2 >= a.nz ? kz + a.nz / 2 - a.nz : kz + a.nz / 2;
                const double syz = a.S[1][ky] * a.S[2][kz];
                C* dst = a.out + (long long)g.f.out[i] * a.fstride + base;
#pragma unroll
                for (int q = 0; q < EPT; q++) {
                    const int k = k0 + q * K;
                    if (q >= nq) continue;
                    const double S = a.S[0][k] * syz;
                    const double re = (double)acc[q].x, im = (double)acc[q].y;
                    const int sx = k + nx / 2 >= nx ? k + nx / 2 - nx : k + nx / 2;
                    const long long at = ((long long)sx * ny + sy) * a.nz + sz;
                    if constexpr (MODE == AnyMode::Intensity) {
                        a.I[at] = floor_1e50(S * S * (re * re + im * im) * a.scale2);
                    } else {
                        const double S2 = S * S * a.scale2;
                        const double f = S2 * (re * re + im * im) > 1e-50 ? a.gI[at] * S2 : 0.0;
                        dst[q * kstep] = cmake<C>(T(f * re), T(-f * im));
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < EPT; q++) acc[q] = cmake<C>(0, 0);
    }
    cp_async_wait<0>();
}

// An axis of length 1 (a film one cell thick): no transform, so a thread folds its pencil's inputs as they arrive.
template <typename T, AnyMode MODE> __global__ void __launch_bounds__(256) axis_one(const __grid_constant__ AxisAny<T> g) {
    using C = C_t<T>;
    const AxisArgs<T>& a = g.a;
    const long long P = (long long)blockIdx.x * 256 + threadIdx.x;
    if (P >= g.npen) return;
    const long long outer = P / g.nin;
    const long long base = outer * a.ostride + (P - outer * g.nin);
    C acc = cmake<C>(0, 0);
    for (int i = 0; i < g.f.n; i++) {
        const C v = a.in[(long long)g.f.field[i] * a.fstride + base];
        fold_fma(acc, __ldg(static_cast<const C*>(g.f.coef[i])), v);
        if (!g.f.last[i]) continue;
        C* dst = a.out + (long long)g.f.out[i] * a.fstride + base;
        if constexpr (MODE == AnyMode::Store || MODE == AnyMode::Pre) {
            *dst = acc;
        } else {
            const int ky = (int)(P / a.nz), kz = (int)(P - (long long)ky * a.nz), ny = (int)a.ny;
            const int sy = ky + ny / 2 >= ny ? ky + ny / 2 - ny : ky + ny / 2;
            const int sz = kz + a.nz / 2 >= a.nz ? kz + a.nz / 2 - a.nz : kz + a.nz / 2;
            const double S = a.S[0][0] * a.S[1][ky] * a.S[2][kz];
            const double re = (double)acc.x, im = (double)acc.y;
            const long long at = (long long)sy * a.nz + sz;
            if constexpr (MODE == AnyMode::Intensity) {
                a.I[at] = floor_1e50(S * S * (re * re + im * im) * a.scale2);
            } else {
                const double S2 = S * S * a.scale2;
                const double f = S2 * (re * re + im * im) > 1e-50 ? a.gI[at] * S2 : 0.0;
                *dst = cmake<C>(T(f * re), T(-f * im));
            }
        }
        acc = cmake<C>(0, 0);
    }
}

// ---------------------------------------------------------------------------------------
// z stage and its adjoint: M columns (a power of two), the 4 components of a column's cell at z pitch +
// {0, M, 2 M, 3 M} + m with pitch = 4 M + 1, odd so that the source's and the fold's accesses along z fall on
// different banks.  A thread evaluates and folds the same CPT cells (neighbouring threads take neighbouring z,
// as the fields lie in memory).
// ---------------------------------------------------------------------------------------
template <typename T, int CPT>
__global__ void __launch_bounds__(512) zstage_any(const __grid_constant__ ZArgs<T> a, const __grid_constant__ AnyDev d,
                                                  unsigned magic_nz) {
    using C = C_t<T>;
    extern __shared__ __align__(16) unsigned char any_smem[];
    const int M = 1 << (d.lp - 2), pitch = 4 * M + 1, nz = a.nz;
    AtomPhase<T>* apc = reinterpret_cast<AtomPhase<T>*>(any_smem);
    C* const tw = reinterpret_cast<C*>(apc + a.in.nPhase * a.nAtom);
    C* const b0 = tw + d.ntw;
    C* const b1 = b0 + nz * pitch;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int nap = a.in.nPhase * a.nAtom;
    for (int i = tid; i < nap; i += nt) apc[i] = a.apc[i];
    for (int i = tid; i < d.ntw; i += nt) tw[i] = static_cast<const C*>(d.tw)[i];

    const long long c0 = (long long)blockIdx.x * M;
    const int ncell = (int)min((long long)M, a.ncols - c0) * nz;
    const long long g0 = c0 * nz;
    CellIn<T> cell[CPT];
    int ph[CPT], zc[CPT], so[CPT];
    T wt[CPT];
    C accE[CPT], accX[CPT], accY[CPT];
#pragma unroll
    for (int q = 0; q < CPT; q++) {
        const int e = tid + q * nt;
        accE[q] = accX[q] = accY[q] = cmake<C>(0, 0);
        ph[q] = -1;
        wt[q] = T(0);
        zc[q] = -1;
        so[q] = 0;
        if (e < ncell) {
            const int m = nz > 1 ? (int)__umulhi((unsigned)e, magic_nz) : e;
            zc[q] = e - m * nz;
            so[q] = zc[q] * pitch + m;
            load_cell<T>(a.in, g0 + e, a.tq, cell[q]);
            if (!a.in.wdense) {
                ph[q] = a.in.phase[g0 + e];
                wt[q] = a.in.weight ? a.in.weight[g0 + e] : T(1);
            }
        }
    }
    __syncthreads();
    for (int at = 0; at < a.nAtom; at++) {
#pragma unroll
        for (int q = 0; q < CPT; q++) {
            if (zc[q] >= 0) {
                C E, X, Y, Z;
                cell_source<T>(a.in, g0 + tid + q * nt, cell[q], ph[q], wt[q], apc, a.nAtom, at, E, X, Y, Z);
                b0[so[q]] = E;
                b0[so[q] + M] = X;
                b0[so[q] + 2 * M] = Y;
                b0[so[q] + 3 * M] = Z;
            }
        }
        C e1[CPT], u1[CPT];  // fetched ahead of the stages' barriers
#pragma unroll
        for (int q = 0; q < CPT; q++) {
            const long long i = (long long)at * nz + (zc[q] >= 0 ? zc[q] : 0);
            e1[q] = __ldg(a.coefE + i);
            u1[q] = __ldg(a.coefUz + i);
        }
        __syncthreads();
        const C* res = any_fft<T>(b0, b1, tw, d, d.lp, pitch, tid, nt);
        // a thread folds the elements that it wrote, so the next atom's sources need no barrier after this
#pragma unroll
        for (int q = 0; q < CPT; q++) {
            if (zc[q] >= 0) {
                const C* s = res + so[q];
                fold_fma(accE[q], e1[q], s[0]);
                fold_fma(accE[q], u1[q], s[3 * M]);
                fold_fma(accX[q], e1[q], s[M]);
                fold_fma(accY[q], e1[q], s[2 * M]);
            }
        }
        const int gr = a.grp[at];
        if (at == a.nAtom - 1 || a.grp[at + 1] != gr) {
            C* o = a.out + 3LL * gr * a.fstride + g0 + tid;
#pragma unroll
            for (int q = 0; q < CPT; q++) {
                if (zc[q] >= 0) {
                    o[q * nt] = accE[q];
                    o[a.fstride + q * nt] = accX[q];
                    o[2 * a.fstride + q * nt] = accY[q];
                }
                accE[q] = accX[q] = accY[q] = cmake<C>(0, 0);
            }
        }
    }
}

template <typename T, int CPT>
__global__ void __launch_bounds__(512) adj_zstage_any(const __grid_constant__ AdjZArgs<T> a,
                                                      const __grid_constant__ AnyDev d, unsigned magic_nz) {
    using C = C_t<T>;
    extern __shared__ __align__(16) unsigned char any_smem[];
    const ZArgs<T>& z = a.z;
    const int M = 1 << (d.lp - 2), pitch = 4 * M + 1, nz = z.nz;
    AtomPhase<T>* apc = reinterpret_cast<AtomPhase<T>*>(any_smem);
    C* const tw = reinterpret_cast<C*>(apc + z.in.nPhase * z.nAtom);
    C* const b0 = tw + d.ntw;
    C* const b1 = b0 + nz * pitch;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int nap = z.in.nPhase * z.nAtom;
    for (int i = tid; i < nap; i += nt) apc[i] = z.apc[i];
    for (int i = tid; i < d.ntw; i += nt) tw[i] = static_cast<const C*>(d.tw)[i];

    const long long c0 = (long long)blockIdx.x * M, n = z.in.n;
    const int ncell = (int)min((long long)M, z.ncols - c0) * nz;
    const long long g0 = c0 * nz;
    CellIn<T> cell[CPT];
    int ph[CPT], zc[CPT], so[CPT];
    T wt[CPT], dU[CPT][3], dP[CPT][3];
    C A[CPT], X[CPT], Y[CPT];
#pragma unroll
    for (int q = 0; q < CPT; q++) {
        const int e = tid + q * nt;
        ph[q] = -1;
        wt[q] = T(0);
        zc[q] = -1;
        so[q] = 0;
        A[q] = X[q] = Y[q] = cmake<C>(0, 0);
#pragma unroll
        for (int c = 0; c < 3; c++) dU[q][c] = dP[q][c] = T(0);
        if (e < ncell) {
            const int m = nz > 1 ? (int)__umulhi((unsigned)e, magic_nz) : e;
            zc[q] = e - m * nz;
            so[q] = zc[q] * pitch + m;
            load_cell<T>(z.in, g0 + e, z.tq, cell[q]);
            if (!z.in.wdense) {
                ph[q] = z.in.phase[g0 + e];
                wt[q] = z.in.weight ? z.in.weight[g0 + e] : T(1);
            }
        }
    }
    // the 3 conjugate fields of a group at this thread's cells
    auto fetch = [&](int gr) {
        const C* f = a.fin + 3LL * gr * z.fstride + g0 + tid;
#pragma unroll
        for (int q = 0; q < CPT; q++)
            if (zc[q] >= 0) {
                A[q] = f[q * nt];
                X[q] = f[z.fstride + q * nt];
                Y[q] = f[2 * z.fstride + q * nt];
            }
    };
    fetch(z.grp[0]);
    __syncthreads();
    for (int at = 0; at < z.nAtom; at++) {
#pragma unroll
        for (int q = 0; q < CPT; q++) {
            if (zc[q] >= 0) {
                const C e1 = __ldg(z.coefE + (long long)at * nz + zc[q]), u1 = __ldg(z.coefUz + (long long)at * nz + zc[q]);
                b0[so[q]] = tw_mul(e1, A[q]);
                b0[so[q] + M] = tw_mul(e1, X[q]);
                b0[so[q] + 2 * M] = tw_mul(e1, Y[q]);
                b0[so[q] + 3 * M] = tw_mul(u1, A[q]);
            }
        }
        if (at + 1 < z.nAtom && z.grp[at + 1] != z.grp[at]) fetch(z.grp[at + 1]);  // lands during the stages
        __syncthreads();
        const C* res = any_fft<T>(b0, b1, tw, d, d.lp, pitch, tid, nt);
#pragma unroll
        for (int q = 0; q < CPT; q++) {
            if (zc[q] >= 0) {
                const C* s = res + so[q];
                const C gE = s[0], gX = s[M], gY = s[2 * M], gZ = s[3 * M];
                if (z.in.wdense) {
                    for (int p = 0; p < z.in.nPhase; p++) {
                        const T w = z.in.wdense[p * n + g0 + tid + q * nt];
                        if (w != T(0)) add_adjoint<T>(cell[q], apc[p * z.nAtom + at], w, a.qc, gE, gX, gY, gZ, dU[q], dP[q]);
                    }
                } else if (ph[q] >= 0 && ph[q] < z.in.nPhase) {
                    add_adjoint<T>(cell[q], apc[ph[q] * z.nAtom + at], wt[q], a.qc, gE, gX, gY, gZ, dU[q], dP[q]);
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < CPT; q++) {
        if (zc[q] >= 0) {
            const long long i = g0 + tid + q * nt;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                a.dU[c * n + i] = dU[q][c];
                a.dP[c * n + i] = c < z.in.nStruc ? dP[q][c] : T(0);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
inline AnyDev any_dev(const AnyStages& st, int lp) {
    AnyDev d = {};
    d.N = st.N;
    d.n = st.n;
    d.lp = lp;
    d.ntw = st.ntw;
    d.tw = st.tw;
    int Ns = 1, tw = 0;
    for (int i = 0; i < st.n; i++) {
        d.s[i].R = st.R[i];
        d.s[i].L = st.N / st.R[i];
        d.s[i].Ns = Ns;
        d.s[i].tw = tw;
        if (i) tw += Ns * any_tw_row(st.R[i]);
        d.s[i].magic = (unsigned)((1ull << 32) / (unsigned)Ns + 1);
        Ns *= st.R[i];
    }
    return d;
}

template <typename T, AnyMode MODE>
cudaError_t launch_axis_mode(const AxisAny<T>& g, int ept, unsigned grid, int nt, size_t smem, cudaStream_t st) {
    cudaError_t e = ept == 8 ? allow_smem<axis_any<T, 8, MODE>>(smem) : allow_smem<axis_any<T, 16, MODE>>(smem);
    if (e != cudaSuccess) return e;
    if (ept == 8) axis_any<T, 8, MODE><<<grid, nt, smem, st>>>(g);
    else axis_any<T, 16, MODE><<<grid, nt, smem, st>>>(g);
    return cudaGetLastError();
}

// Tile: 8 neighbouring pencils (64-byte rows of complex64), more while it holds under 1024 values, fewer while
// it exceeds 8192 values or shared memory, and down to 4 (a whole 32-byte sector) while there are not two tiles
// per SM.
template <typename T>
cudaError_t launch_axis_any(const AxisArgs<T>& a, const AnyFold& f, const AnyStages& st, AnyMode mode,
                            long long nouter, long long nin, int sms, size_t smem_max, cudaStream_t stream, bool* done) {
    using C = C_t<T>;
    *done = false;
    if (f.n < 1 || a.accumulate || st.N != a.N) return cudaSuccess;
    const long long npen = nouter * nin;
    if (a.N == 1 && (npen + 255) / 256 <= 0x7fffffffLL) {
        AxisAny<T> g;
        g.a = a;
        g.f = f;
        g.d = any_dev(st, 0);
        g.npen = npen;
        g.nin = nin;
        *done = true;
        const unsigned grid = (unsigned)((npen + 255) / 256);
        switch (mode) {  // 1x400x400 x pass: 17 us as a tile pass, 9 us here
            case AnyMode::Store: axis_one<T, AnyMode::Store><<<grid, 256, 0, stream>>>(g); break;
            case AnyMode::Intensity: axis_one<T, AnyMode::Intensity><<<grid, 256, 0, stream>>>(g); break;
            case AnyMode::Seed: axis_one<T, AnyMode::Seed><<<grid, 256, 0, stream>>>(g); break;
            case AnyMode::Pre: axis_one<T, AnyMode::Pre><<<grid, 256, 0, stream>>>(g); break;
        }
        return cudaGetLastError();
    }
    auto smem = [&](int lp) { return sizeof(C) * ((size_t)3 * (st.N << lp) + st.ntw); };
    int lp = sizeof(T) == 4 ? 3 : 2;
    while ((st.N << lp) < 1024 && lp < 8 && (1LL << lp) < npen) lp++;
    while (lp > 0 && ((st.N << lp) > kAnyTile || smem(lp) > smem_max)) lp--;
    if ((st.N << lp) > kAnyTile || smem(lp) > smem_max) return cudaSuccess;
    const int least = sizeof(T) == 4 ? 2 : 1;
    while (lp > least && (npen >> lp) < 2LL * sms) lp--;
    const int elems = st.N << lp;
    const int ept = elems > 4096 ? 16 : 8;
    const int unit = 1 << (lp > 5 ? lp : 5);
    const int nt = ((elems + ept - 1) / ept + unit - 1) / unit * unit;
    const long long grid = (npen + (1LL << lp) - 1) >> lp;
    if (nt > 512 || grid > 0x7fffffffLL) return cudaSuccess;
    AxisAny<T> g;
    g.a = a;
    g.f = f;
    g.d = any_dev(st, lp);
    g.npen = npen;
    g.nin = nin;
    *done = true;
    switch (mode) {
        case AnyMode::Store: return launch_axis_mode<T, AnyMode::Store>(g, ept, (unsigned)grid, nt, smem(lp), stream);
        case AnyMode::Intensity: return launch_axis_mode<T, AnyMode::Intensity>(g, ept, (unsigned)grid, nt, smem(lp), stream);
        case AnyMode::Seed: return launch_axis_mode<T, AnyMode::Seed>(g, ept, (unsigned)grid, nt, smem(lp), stream);
        case AnyMode::Pre: return launch_axis_mode<T, AnyMode::Pre>(g, ept, (unsigned)grid, nt, smem(lp), stream);
    }
    return cudaErrorInvalidValue;
}

// Columns per z tile: up to 512 cells (2 per thread), fewer while there are not two tiles per SM.
struct ZTile {
    int lm = 0, cpt = 0, nt = 0;
    size_t smem = 0;
    long long grid = 0;
};
template <typename T> bool z_tile(const ZArgs<T>& z, const AnyStages& st, int sms, size_t smem_max, ZTile* t) {
    using C = C_t<T>;
    if (st.N != z.nz) return false;
    auto smem = [&](int lm) {
        return sizeof(AtomPhase<T>) * z.in.nPhase * z.nAtom + sizeof(C) * ((size_t)st.ntw + 2 * (size_t)z.nz * ((4 << lm) + 1));
    };
    int lm = 0;
    while (((long long)z.nz << (lm + 1)) <= 512 && lm < 5 && (1LL << lm) < z.ncols) lm++;
    while (lm > 0 && (z.ncols >> lm) < 2LL * sms) lm--;
    const int cells = z.nz << lm;
    t->lm = lm;
    t->cpt = cells > 1024 ? 4 : 2;
    t->nt = ((cells + t->cpt - 1) / t->cpt + 31) / 32 * 32;
    t->smem = smem(lm);
    t->grid = (z.ncols + (1LL << lm) - 1) >> lm;
    return t->nt <= 512 && t->smem <= smem_max && t->grid <= 0x7fffffffLL;
}
inline unsigned z_magic(int nz) { return (unsigned)((1ull << 32) / (unsigned)nz + 1); }

template <typename T>
cudaError_t launch_z_any(const ZArgs<T>& a, const AnyStages& st, int sms, size_t smem_max, cudaStream_t stream,
                         bool* done) {
    ZTile t;
    *done = z_tile(a, st, sms, smem_max, &t);
    if (!*done) return cudaSuccess;
    const AnyDev d = any_dev(st, t.lm + 2);
    cudaError_t e = t.cpt == 2 ? allow_smem<zstage_any<T, 2>>(t.smem) : allow_smem<zstage_any<T, 4>>(t.smem);
    if (e != cudaSuccess) return e;
    if (t.cpt == 2) zstage_any<T, 2><<<(unsigned)t.grid, t.nt, t.smem, stream>>>(a, d, z_magic(a.nz));
    else zstage_any<T, 4><<<(unsigned)t.grid, t.nt, t.smem, stream>>>(a, d, z_magic(a.nz));
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_adjz_any(const AdjZArgs<T>& a, const AnyStages& st, int sms, size_t smem_max, cudaStream_t stream,
                            bool* done) {
    ZTile t;
    *done = z_tile(a.z, st, sms, smem_max, &t);
    if (!*done) return cudaSuccess;
    const AnyDev d = any_dev(st, t.lm + 2);
    cudaError_t e = t.cpt == 2 ? allow_smem<adj_zstage_any<T, 2>>(t.smem) : allow_smem<adj_zstage_any<T, 4>>(t.smem);
    if (e != cudaSuccess) return e;
    if (t.cpt == 2) adj_zstage_any<T, 2><<<(unsigned)t.grid, t.nt, t.smem, stream>>>(a, d, z_magic(a.z.nz));
    else adj_zstage_any<T, 4><<<(unsigned)t.grid, t.nt, t.smem, stream>>>(a, d, z_magic(a.z.nz));
    return cudaGetLastError();
}

#define QPD_ANY_INSTANTIATE(T)                                                                                        \
    template cudaError_t launch_axis_any<T>(const AxisArgs<T>&, const AnyFold&, const AnyStages&, AnyMode,         \
                                            long long, long long, int, size_t, cudaStream_t, bool*);                  \
    template cudaError_t launch_z_any<T>(const ZArgs<T>&, const AnyStages&, int, size_t, cudaStream_t, bool*);        \
    template cudaError_t launch_adjz_any<T>(const AdjZArgs<T>&, const AnyStages&, int, size_t, cudaStream_t, bool*);

}  // namespace qpd
