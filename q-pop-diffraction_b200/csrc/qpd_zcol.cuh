// Fused z stage of the float32 schedule for nz = N1 N2 (N1 = 4 .. 7, or 8 on lane pairs; N2 up to 17) and single-phase
// inputs: source, z transform and fold.
//
// A column is an N1 x N2 array of cells.  Phase A transforms over the N1 cells of one b in registers, straight
// from the sources; phase B transforms the N2 values of one row (column, component, a) in place; the fold gives
// every thread a pair of neighbouring k_z of some columns, combines the components with exp(-i (k_z + G_z) R_z) and
// -i k_z times it, and stores whole 16-byte units of the fields.  Coprime factors use the Good-Thomas maps and need no
// twiddles, others a twiddle after phase A.
//
// What bounds it is the shared-memory data pipe (87% busy at 512x512x104), then instruction issue (54%), so the
// layout is chosen for few wavefronts:
//   - a tile's inputs wait in shared memory in phase-A order and are re-read for every atom (16-byte loads);
//   - rows are an odd number of 16-byte units apart, so phase B reads and writes two values at a time without bank
//     conflicts, and every address is a per-thread base plus a literal;
//   - for N1 = 8 a pair of lanes evaluates the sources of four cells each, exchanges them (E and two factors per
//     cell instead of four components) and each lane transforms two of the four components whole;
//   - cells that do not scatter have a record of zeros, so the sources have no branches;
//   - with isotropic ionic shifts (su = k delta, ISO) the phase is one fma on qC.P and the shifts are three.
// Without pairs (N1 = 4 .. 7) a thread holds the N1 cells of its b alone.  Four CTAs of four warps at up to 128
// registers beat three of eight at 80, which spill (1.53 against 1.92 ms at 512x512x104, 3.98 against 4.97 at
// 1024x1024x68).  Folding in phase B's registers and storing from there halves the exchanges but not the wavefronts
// (1.59 and 4.67 ms).  One B200, us per z stage, before (qpd_fast.cuh, for nz = 68 qpd_zpfa.cuh) -> now: 512x512x104
// 1826 -> 1528, 1024x1024x68 4457 -> 3977, 256x256x64 238 -> 187, 128^3 144 -> 117, 64x64x32 18 -> 15; against the
// runtime-length stage (qpd_any.cuh) 150x135x75 159 -> 98, 120x100x50 74 -> 48.
#pragma once

#include "qpd_kernels.cuh"
#include "qpd_radix.cuh"
#include "qpd_zprefetch.h"

namespace qpd {

__host__ __device__ constexpr int zcol_gcd(int a, int b) { return b == 0 ? a : zcol_gcd(b, a % b); }

// Per (phase, atom) constants with isotropic shifts.
struct alignas(16) IsoAtom {
    double k;       // nm per C/m^2
    float fr, fi;
    float kf, pad[3];
};

template <int N1, int N2, int M> struct ZCol {
    static constexpr int N = N1 * N2, CELLS = M * N;
    static_assert(CELLS % 2 == 0, "16-byte tables behind the inputs");
    static constexpr int SPLIT = N1 == 8 ? 2 : 1;
    static constexpr bool PFA = zcol_gcd(N1, N2) == 1;
    static constexpr int H = (N2 + 1) / 2;                     // 16-byte units of a row
    static constexpr int RP = 2 * (H % 2 ? H : H + 1);         // row pitch, complex values
    static constexpr int CP0 = N1 * RP;
    // component pitch: the lanes of a pair store components two apart, half the banks away
    static constexpr int CP = SPLIT == 2 ? (CP0 + 7) / 8 * 8 + 4 : CP0;
    static constexpr int XB = 4 * M * CP;
    static constexpr int IA = SPLIT * M * N2, IB = 4 * M * N1;  // items of the two phases
    static constexpr int NT = ((IA > IB ? IA : IB) + 31) / 32 * 32;
    static constexpr int TWP = 10;                             // twiddle row pitch (N1 = 8)
    // position of cell z in the inputs, a N2 + b
    __host__ __device__ static constexpr int in_pos(int z) {
        if (!PFA) return z;
        for (int a = 0; a < N1; a++)
            for (int b = 0; b < N2; b++)
                if ((N2 * a + N1 * b) % N == z) return a * N2 + b;
        return 0;
    }
    // position of output k in its column's component, a RP + r
    __host__ __device__ static constexpr int out_pos(int k) { return (k % N1) * RP + (PFA ? k % N2 : k / N1); }
    static constexpr int NQ = (N + 7) / 8 * 8;
    static constexpr int CELLS16 = (CELLS + 15) / 16 * 16;
    static size_t bytes(int nap, int nAtom, bool iso, bool weights) {
        return (size_t)CELLS * (32 + (iso ? 8 : 0)) + CELLS16 * (weights ? 5 : 1) + sizeof(float2) * XB +
               (!PFA && SPLIT == 2 ? sizeof(float2) * N2 * TWP : 0) +
               (iso ? sizeof(IsoAtom) : sizeof(AtomPhase<float>)) * (nap + nAtom) + sizeof(short) * NQ;
    }
};

template <int N1, int N2, int M, int MINB, bool ISO>
__global__ void __launch_bounds__(ZCol<N1, N2, M>::NT, MINB) zcol(const __grid_constant__ ZArgs<float> a) {
    using L = ZCol<N1, N2, M>;
    using C = float2;
    constexpr int N = L::N, NT = L::NT, RP = L::RP, CP = L::CP, CELLS = L::CELLS, SPLIT = L::SPLIT;
    static_assert(N1 >= 4 && N1 <= 8, "phase A holds 4 to 7 cells per thread");
    constexpr int CA = SPLIT == 2 ? 4 : N1;  // cells of a phase-A item
    extern __shared__ __align__(16) unsigned char zsm[];
    float4* const inA = reinterpret_cast<float4*>(zsm);          // P, u_x
    float4* const inB = inA + CELLS;                             // u_y, u_z, qC.u / 2 pi (double)
    C* const xb = reinterpret_cast<C*>(inB + CELLS);             // exchange rows [m][component][a][RP]
    C* const twr = xb + L::XB;                                   // [b][TWP], N1 = 8 with twiddles
    constexpr int NTW = !L::PFA && SPLIT == 2 ? N2 * L::TWP : 0;
    double* const inT = reinterpret_cast<double*>(twr + NTW);    // ISO: qC.P / 2 pi
    unsigned char* const tab = reinterpret_cast<unsigned char*>(inT + (ISO ? CELLS : 0));
    const int nap = a.in.nPhase * a.nAtom;  // and nAtom more for cells that do not scatter
    IsoAtom* const iap = reinterpret_cast<IsoAtom*>(tab);
    AtomPhase<float>* const apc = reinterpret_cast<AtomPhase<float>*>(tab);
    short* const pin = reinterpret_cast<short*>(tab + (ISO ? sizeof(IsoAtom) : sizeof(AtomPhase<float>)) * (nap + a.nAtom));
    unsigned char* const inP = reinterpret_cast<unsigned char*>(pin + L::NQ);  // phase
    float* const inW = reinterpret_cast<float*>(inP + L::CELLS16);               // weight, when there is one
    const bool weights = a.in.weight != nullptr;
    const int tid = threadIdx.x;

    for (int i = tid; i < nap + a.nAtom; i += NT) {  // phase nPhase: does not scatter
        if (i >= nap) {
            if constexpr (ISO) iap[i] = IsoAtom{};
            else apc[i] = AtomPhase<float>{};
        } else if constexpr (ISO) {
            IsoAtom t;
            t.k = a.isok[i];
            t.kf = a.apc[i].su[0];
            t.fr = a.apc[i].fr;
            t.fi = a.apc[i].fi;
            iap[i] = t;
        } else {
            apc[i] = a.apc[i];
        }
    }
    for (int z = tid; z < N; z += NT) {
        int pi = z;
        if constexpr (L::PFA) {  // z = (N2 a + N1 b) mod N
            for (int i = 0; i < N1; i++) {
                const int w = (z - N2 * i % N + N) % N;
                if (w % N1 == 0) pi = i * N2 + w / N1;
            }
        }
        pin[z] = (short)pi;
    }
    if constexpr (NTW > 0)
        for (int i = tid; i < N1 * N2; i += NT) {
            const int b = i / N1, k = i - b * N1;
            twr[b * L::TWP + k] = static_cast<const C*>(a.zp.tw)[b * k];
        }

    // phase-A item: column am, b = ab, lane half ah; its cells are (4 ah + j, ab)
    const int ah = SPLIT == 2 ? tid & 1 : 0;
    const int am = (tid / SPLIT) / N2, ab = (tid / SPLIT) - am * N2;
    const bool actA = tid < L::IA;
    const int cell0 = actA ? am * N + 4 * ah * N2 + ab : 0;
    C* const st0 = xb + (actA ? (am * 4 + (SPLIT == 2 ? 2 * ah : 0)) * CP + ab : 0);
    C twa[N1 - 1] = {};  // without pairs: exp(-2 pi i b k / N), k = 1 .. N1 - 1
    if constexpr (!L::PFA && SPLIT == 1) {
#pragma unroll
        for (int k = 1; k < N1; k++) twa[k - 1] = static_cast<const C*>(a.zp.tw)[(actA ? ab : 0) * k];
    }
    // phase-B row
    const int ba = tid % N1, bc = (tid / N1) & 3, bm = tid / (4 * N1);
    const bool actB = tid < L::IB;
    float4* const row = reinterpret_cast<float4*>(xb + (bm * 4 + bc) * CP + ba * RP);
    // fold: this thread's V neighbouring k_z of columns om, om + OM, ...
    constexpr int V = N % 2 ? 1 : 2, KV = N / V, OM = NT / KV < M ? NT / KV : M, OI = (M + OM - 1) / OM;
    static_assert(KV <= NT, "a thread for every pair of a column");
    const int om = tid / KV, ok = (tid - om * KV) * V;
    const bool actO = om < OM;

    __syncthreads();
    const C* const os0 = xb + (actO ? om * 4 * CP + L::out_pos(ok) : 0);
    const C* const os1 = xb + (actO ? om * 4 * CP + L::out_pos(ok + V - 1) : 0);
    const long long ntiles = (a.ncols + M - 1) / M;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int mcols = (int)min((long long)M, a.ncols - t * M);
        const int ncell = mcols * N;
        const long long g0 = t * CELLS;
        // the next tile's inputs come closer while this one is computed
        const long long gn = (t + gridDim.x) * CELLS;
        if (gn + CELLS <= a.ncols * N) {
            const int nl = prefetch_lines(CELLS, a.in.nStruc);
            for (int i = tid; i < nl; i += NT) {
                const PrefetchLine l = prefetch_line(i, CELLS, a.in.nStruc, a.in.n, gn);
                const void* q = l.array == 0 ? (const void*)(a.in.P + l.at)
                              : l.array == 1 ? (const void*)(a.in.U + l.at)
                                             : (const void*)(a.in.phase + l.at);
                asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
            }
        }
        // ---- inputs, neighbouring threads on neighbouring z
        // (all loads of a batch of cells in flight together; a cell that does not scatter becomes zeros)
        constexpr int PER = (CELLS + NT - 1) / NT, BATCH = PER < 2 ? PER : 2;
        for (int e0 = tid; e0 < CELLS; e0 += BATCH * NT) {
            float in[BATCH][6], w[BATCH];
            int ph[BATCH];
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                const int e = e0 + i * NT;
                ph[i] = -1;
                w[i] = 1.f;
                if (e < ncell) {
                    ph[i] = a.in.phase[g0 + e];
                    if (a.in.weight) w[i] = a.in.weight[g0 + e];
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        in[i][k] = k < a.in.nStruc ? a.in.P[k * a.in.n + g0 + e] : 0.f;
                        in[i][3 + k] = a.in.U[k * a.in.n + g0 + e];
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                const int e = e0 + i * NT;
                if (CELLS % (BATCH * NT) == 0 || e < CELLS) {
                    const bool scat = ph[i] >= 0 && ph[i] < a.in.nPhase;
#pragma unroll
                    for (int k = 0; k < 6; k++) in[i][k] = scat ? in[i][k] : 0.f;
                    const int m = e / N;
                    const int at = m * N + pin[e - m * N];
                    const double tu = a.tq[0] * (double)in[i][3] + a.tq[1] * (double)in[i][4] + a.tq[2] * (double)in[i][5];
                    inA[at] = make_float4(in[i][0], in[i][1], in[i][2], in[i][3]);
                    inB[at] = make_float4(in[i][4], in[i][5], __int_as_float(__double2loint(tu)), __int_as_float(__double2hiint(tu)));
                    inP[at] = (unsigned char)(scat ? ph[i] : a.in.nPhase);
                    if (weights) inW[at] = scat ? w[i] : 0.f;
                    if constexpr (ISO)
                        inT[at] = a.tq[0] * (double)in[i][0] + a.tq[1] * (double)in[i][1] + a.tq[2] * (double)in[i][2];
                }
            }
        }
        C acc[OI][3][V];
#pragma unroll
        for (int i = 0; i < OI; i++)
#pragma unroll
            for (int v = 0; v < V; v++) acc[i][0][v] = acc[i][1][v] = acc[i][2][v] = make_float2(0.f, 0.f);
        __syncthreads();

        for (int at = 0; at < a.nAtom; at++) {
            // ---- phase A
            if ((tid & ~31) < L::IA) {
                C E[CA];
                float ua[3][CA];
#pragma unroll
                for (int j = 0; j < CA; j++) {
                    const float4 ca = inA[cell0 + j * N2], cb = inB[cell0 + j * N2];
                    const double tu = __hiloint2double(__float_as_int(cb.w), __float_as_int(cb.z));
                    const int ip = inP[cell0 + j * N2] * a.nAtom + at;
                    double ph;
                    float fr, fi;
                    if constexpr (ISO) {
                        const IsoAtom& k = iap[ip];
                        ph = tu + k.k * inT[cell0 + j * N2];
                        fr = k.fr;
                        fi = k.fi;
                        ua[0][j] = ca.w + k.kf * ca.x;
                        ua[1][j] = cb.x + k.kf * ca.y;
                        ua[2][j] = cb.y + k.kf * ca.z;
                    } else {
                        const AtomPhase<float>& k = apc[ip];
                        ph = tu + k.bq[0] * (double)ca.x + k.bq[1] * (double)ca.y + k.bq[2] * (double)ca.z;
                        fr = k.fr;
                        fi = k.fi;
                        ua[0][j] = ca.w + k.su[0] * ca.x + k.su[1] * ca.y + k.su[2] * ca.z;
                        ua[1][j] = cb.x + k.su[3] * ca.x + k.su[4] * ca.y + k.su[5] * ca.z;
                        ua[2][j] = cb.y + k.su[6] * ca.x + k.su[7] * ca.y + k.su[8] * ca.z;
                    }
                    ph -= rint(ph);  // reduced in double: the phase in turns, |ph| <= 1/2
                    float sn, cs;
                    expm2pi(ph, &sn, &cs);
                    E[j] = make_float2(fr * cs + fi * sn, fi * cs - fr * sn);
                    if (weights) {
                        const float w = inW[cell0 + j * N2];
                        E[j] = make_float2(w * E[j].x, w * E[j].y);
                    }
                }
                if constexpr (SPLIT == 1) {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        C v[CA];
#pragma unroll
                        for (int j = 0; j < CA; j++) {
                            const float u = ua[(q + 2) % 3][j];
                            v[j] = q == 0 ? E[j] : make_float2(E[j].x * u, E[j].y * u);
                        }
                        Bfly<CA, C>::run(v);
                        if constexpr (!L::PFA) {
#pragma unroll
                            for (int k = 1; k < CA; k++) v[k] = tw_mul(twa[k - 1], v[k]);
                        }
                        if (actA) {
#pragma unroll
                            for (int k = 0; k < CA; k++) st0[q * CP + k * RP] = v[k];
                        }
                    }
                } else {
                    // lane 0 transforms E and X = E u_x, lane 1 Y and Z: each needs the other's E and its two factors
                    C Eo[4];
                    float f0[4], f1[4], g0_[4], g1_[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        f0[j] = ah ? ua[1][j] : 1.f;
                        f1[j] = ah ? ua[2][j] : ua[0][j];
                        g0_[j] = ah ? 1.f : ua[1][j];
                        g1_[j] = ah ? ua[0][j] : ua[2][j];
                        Eo[j].x = __shfl_xor_sync(0xffffffffu, E[j].x, 1);
                        Eo[j].y = __shfl_xor_sync(0xffffffffu, E[j].y, 1);
                        g0_[j] = __shfl_xor_sync(0xffffffffu, g0_[j], 1);
                        g1_[j] = __shfl_xor_sync(0xffffffffu, g1_[j], 1);
                    }
                    // lane 1 holds its cells 4 places early: its outputs of odd k carry a factor -1, undone on the
                    // way out, in the fold
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        C v[8];
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const float fo = q ? f1[j] : f0[j], go = q ? g1_[j] : g0_[j];
                            v[j] = make_float2(E[j].x * fo, E[j].y * fo);
                            v[4 + j] = make_float2(Eo[j].x * go, Eo[j].y * go);
                        }
                        Bfly<8, C>::run(v);
                        if constexpr (!L::PFA) {
                            const C* w = twr + ab * L::TWP;
#pragma unroll
                            for (int k = 1; k < 8; k++) v[k] = tw_mul(w[k], v[k]);
                        }
                        if (actA) {
#pragma unroll
                            for (int k = 0; k < 8; k++) st0[q * CP + k * RP] = v[k];
                        }
                    }
                }
            }
            __syncthreads();
            C e1[V], u1[V];  // the fold's coefficients, on their way during phase B
            if (actO) {
                const C* ce = a.coefE + at * N + ok;
                const C* cu = a.coefUz + at * N + ok;
                if constexpr (V == 2) {
                    const float4 q = __ldg(reinterpret_cast<const float4*>(ce)), p = __ldg(reinterpret_cast<const float4*>(cu));
                    e1[0] = make_float2(q.x, q.y);
                    e1[V - 1] = make_float2(q.z, q.w);
                    u1[0] = make_float2(p.x, p.y);
                    u1[V - 1] = make_float2(p.z, p.w);
                } else {
                    e1[0] = __ldg(ce);
                    u1[0] = __ldg(cu);
                }
            }
            // ---- phase B, in place: only this thread reads the row
            if (actB) {
                C v[(N2 + 1) / 2 * 2];
#pragma unroll
                for (int i = 0; i < (N2 + 1) / 2; i++) {
                    const float4 q = row[i];
                    v[2 * i] = make_float2(q.x, q.y);
                    v[2 * i + 1] = make_float2(q.z, q.w);
                }
                C x[N2];
#pragma unroll
                for (int r = 0; r < N2; r++) x[r] = v[r];
                Bfly<N2, C>::run(x);
#pragma unroll
                for (int r = 0; r < N2; r++) v[r] = x[r];
#pragma unroll
                for (int i = 0; i < (N2 + 1) / 2; i++)
                    row[i] = make_float4(v[2 * i].x, v[2 * i].y, v[2 * i + 1].x, v[2 * i + 1].y);
            }
            __syncthreads();
            // ---- fold into the group's fields
            const int gr = a.grp[at];
            const bool last = at == a.nAtom - 1 || a.grp[at + 1] != gr;
            if (actO) {
                C* const o = a.out + 3LL * gr * a.fstride + g0 + om * N + ok;
#pragma unroll
                for (int i = 0; i < OI; i++) {
                    if (om + i * OM < mcols) {
#pragma unroll
                        for (int w = 0; w < V; w++) {
                            const C* s = (w ? os1 : os0) + i * OM * 4 * CP;
                            C E = s[0], X = s[CP], Y = s[2 * CP], Z = s[3 * CP];
                            if (SPLIT == 2 && (w & 1)) {  // odd a = k mod N1: lane 1's components carry a factor -1
                                Y = make_float2(-Y.x, -Y.y);
                                Z = make_float2(-Z.x, -Z.y);
                            }
                            fold_fma(acc[i][0][w], e1[w], E);
                            fold_fma(acc[i][0][w], u1[w], Z);
                            fold_fma(acc[i][1][w], e1[w], X);
                            fold_fma(acc[i][2][w], e1[w], Y);
                        }
                        if (last) {
#pragma unroll
                            for (int c = 0; c < 3; c++) {
                                C* d = o + c * a.fstride + i * OM * N;
                                if constexpr (V == 2)
                                    *reinterpret_cast<float4*>(d) =
                                        make_float4(acc[i][c][0].x, acc[i][c][0].y, acc[i][c][V - 1].x, acc[i][c][V - 1].y);
                                else *d = acc[i][c][0];
#pragma unroll
                                for (int w = 0; w < V; w++) acc[i][c][w] = make_float2(0.f, 0.f);
                            }
                        }
                    }
                }
            }
            __syncthreads();
        }
    }
}

}  // namespace qpd
