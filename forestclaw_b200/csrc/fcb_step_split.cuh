// Pipelined step kernel of the systems (shallow-water and Euler Roe solvers,
// GeoClaw f-waves): step2 + flux2 + conservative update with the two sweeps of a
// column on two threads.
//
// A patch column is worked on by one thread of the CTA's X half (x-Riemann
// problems, x limiter and corrections, their transverse parts, the cell update)
// and one of its Y half (loads, per-cell quantities, y-Riemann problems, y
// limiter and corrections, their transverse parts).  Rows stream top to bottom;
// everything the two halves and neighbouring columns exchange goes through rings
// of rows in shared memory whose consumers run at least one iteration after
// their producer, so one CTA barrier per row separates them.  Iteration s:
//   Y  row s loaded, its cell quantities -> rings Q, CELL (stored aux -> AX)
//      y-interface s-1 raw, y-interface s-2 final -> rings FYM, FYP; GY(row s-3)
//   X  x-row s-3: transverse parts of the right neighbour (ring GL) -> GX
//      cell row s-4: conservative update (rings FX, GY, FYM, FYP; own GX)
//      x-row s-2: limiter with the neighbours' waves (ring XW), second-order and
//      transverse corrections -> rings FX, GL
//      x-row s-1: Riemann problems (rings Q, CELL) -> ring XW
//
// What bounds it and why this split: a Riemann problem is a chain of dependent
// FP64 operations, and with both sweeps in one thread (the four-barrier form of
// fcb_step.cu, 248 registers) an SM holds eight warps, which cannot hide it.  Half a
// column per thread fits 128 registers, so sixteen warps are resident on the same
// shared memory.  What a thread needs of an interface in the next iteration is kept
// small (Roe averages and wave strengths, from which the waves are formed again),
// states arrive by cp.async in the ring the Riemann problems read, and the loop
// counters are uniform.  Shallow water, mx = 32, 1,024 patches, one level update on
// B200: 0.395 ms in the four-barrier form, 0.139 ms here (FP64 pipe 46 %, issue slots
// 60 %; stalls: fixed latencies and the barrier); Euler, mx = 16, 4,096 patches: 0.856
// and 0.320 ms; GeoClaw, mx = 32, 1,024 patches: 0.157 ms (pipelined form of one thread
// per column: 0.57 ms).  Those are of states with a front's tail in many patches; after 20
// steps from the dam break and the lake (CFL 0.4) and the quadrants (0.2): 0.119, 0.131 and
// 0.309 ms (0.121, 0.133 and 0.339 before the operators' path took the cells' quantities and
// the range checks of dividends became one comparison).
//
// Arithmetic, operation order and loop bounds are those of the reference
// (src/solvers/fc2d_clawpack4.6/fortran_source/clawpack46_step2.f, clawpack46_flux2.f,
// clawpack46_flux2fw.f, clawpack46_step2_wrap.f; clawpack5_step2.f90, clawpack5_flux2.f,
// clawpack5_step2_wrap.f), apart from products with wave components that are
// zero by construction (SOL::nz), which are left out: they add a zero.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "fcb_device.h"
#include "fcb_launch.hpp"
#include "fcb_solvers.cuh"
#include "fcb_strip.cuh"

namespace fcb {

namespace {

// LIM > 0: order (2, 2) and limiter LIM on every wave, fixed at compile time;
// LIM == 0: order and limiters read from the launch arguments.
template <int LIM>
struct SplitMethod {
    const StepArgs& a;
    __device__ __forceinline__ bool second_order() const { return LIM > 0 || a.order0 == 2; }
    __device__ __forceinline__ bool transverse() const { return LIM > 0 || a.order1 > 0; }
    __device__ __forceinline__ bool transverse2() const { return LIM > 0 || (a.order0 > 1 && a.order1 == 2); }
    __device__ __forceinline__ int lim(int mw) const { return LIM > 0 ? LIM : a.mthlim[mw]; }
};

// The f-wave solver's hydrostatic part reads FP64 states and bathymetry, so its
// state and aux rings are FP64 in the mixed form too.
template <class SOL>
constexpr bool split_qdbl = SOL::FWAVE && !std::is_same_v<typename SOL::Real, double>;
template <class SOL>
using split_qt = std::conditional_t<SOL::FWAVE, double, typename SOL::Real>;

// Component of a wave in the sweep's own order (0, normal, transverse, energy).
__host__ __device__ constexpr int wave_rel(int ixy, int m) { return (ixy == 2 && (m == 1 || m == 2)) ? 3 - m : m; }

// Rings [slot][component][column]: offsets in elements of their region, columns
// of all patches of the CTA side by side (PNX).
template <class SOL, int PNX, int NAUX>
struct SplitSmem {
    using R = typename SOL::Real;
    static constexpr int M = SOL::M, W = SOL::W, NC = SOL::NC;
    static constexpr bool TR = !SOL::FWAVE;  // no transverse parts in the f-wave solver
    static constexpr bool QD = split_qdbl<SOL>;
    // FP64 states: rows s+1 .. s-4, copied in by cp.async; FP32 ones: s .. s-2
    static constexpr int NQ = std::is_same_v<split_qt<SOL>, double> ? 6 : 3;
    // FP64 region
    static constexpr int GY = 0;                                  // 2 slots x 2M
    static constexpr int DQ = GY + (TR ? 2 * 2 * M * PNX : 0);    // NQ slots x M (QD)
    static constexpr int DAX = DQ + (QD ? NQ * M * PNX : 0);      // 3 slots x NAUX (QD)
    static constexpr int ND = DAX + (QD ? 3 * NAUX * PNX : 0);
    // region of the compute type
    static constexpr int XW = 0;                                  // 2 slots x W*M
    static constexpr int GL = XW + 2 * SOL::NWV * PNX;            // 2 slots x 2M
    static constexpr int FX = GL + (TR ? 2 * 2 * M * PNX : 0);    // 3 slots x 2M
    static constexpr int FYM = FX + 3 * 2 * M * PNX;              // 2 slots x M
    static constexpr int FYP = FYM + 2 * M * PNX;                 // 3 slots x M
    static constexpr int CELL = FYP + 3 * M * PNX;                // 3 slots x NC
    static constexpr int Q = CELL + 3 * NC * PNX;                 // NQ slots x M
    static constexpr int AX = Q + (QD ? 0 : NQ * M * PNX);        // 3 slots x NAUX
    // transverse parts a thread keeps for its next row: in registers, or here where
    // the FP64 Roe solvers would spill them and the shared memory has room
    static constexpr bool KEEPX = TR && sizeof(R) == 8 && M == 3, KEEPY = TR && sizeof(R) == 8;
    static constexpr int KX = AX + (QD ? 0 : 3 * NAUX * PNX);     // 2M
    static constexpr int KY = KX + (KEEPX ? 2 * M * PNX : 0);     // 2M
    // the f-waves of the y-interface that is final next
    static constexpr int KW = KY + (KEEPY ? 2 * M * PNX : 0);     // W*M
    static constexpr int NR = KW + (SOL::FWAVE ? SOL::NWV * PNX : 0);
    static constexpr int BYTES = ND * 8 + ((NR * (int)sizeof(R) + 15) / 16) * 16;
};

// 8 bytes of global memory into shared memory, without passing through registers.
__device__ __forceinline__ void copy_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The barrier of a row.  The two halves of the CTA meet at it from different places, which
// __syncthreads() is not made for (one call, reached by the whole CTA); a barrier with its
// number and count of threads is.  Both halves pass it NY + 3 times.
template <int THREADS>
__device__ __forceinline__ void row_barrier() {
    asm volatile("barrier.sync 1, %0;" ::"n"(THREADS) : "memory");
}

// The time-sync registers are accumulated for the shallow-water Roe solver in
// FP64, the one whose conservative flux the flux store has.
template <class SOL>
__host__ __device__ constexpr bool split_time_sync() {
    return std::is_same_v<SOL, SweRoeT<double, SOL::V5>>;
}

}  // namespace

// HALF: threads of each half of the CTA.  MXP > 0: patches of MXP x MXP cells,
// HALF / (MXP + 4) of them at most, a.ppc of them used; MXP == 0: one strip of at
// most HALF columns (a.strip, fcb_strip.cuh).
// TSYNC: accumulate the time-sync registers.
template <class SOL, int MXP, int NAUX, int HALF, int LIM, bool TSYNC>
__global__ void __launch_bounds__(2 * HALF) step_kernel_split(const StepArgs a) {
    using R = typename SOL::Real;
    using QT = split_qt<SOL>;
    constexpr int M = SOL::M, W = SOL::W, NC = SOL::NC, MBC = 2;
    constexpr bool STRIP = MXP == 0;
    constexpr int NXC = STRIP ? HALF : MXP + 2 * MBC;  // columns of a patch in the rings
    constexpr int PNX = STRIP ? HALF : HALF / NXC * NXC;
    const int x0 = STRIP ? blockIdx.x % a.strip.nsx * a.strip.w : 0, y0 = STRIP ? blockIdx.x / a.strip.nsx * a.strip.h : 0;
    const int MX = STRIP ? min(a.strip.w, a.strip.n - x0) : MXP;  // interior columns and rows
    const int MY = STRIP ? min(a.strip.h, a.strip.n - y0) : MXP;
    const int NX = MX + 2 * MBC, NY = MY + 2 * MBC;
    constexpr bool V5 = SOL::V5, FWAVE = SOL::FWAVE;
    constexpr bool R15 = V5 || FWAVE;  // fluxes on interfaces MBC..MBC+MX only
    constexpr bool TR = !FWAVE;
    using L = SplitSmem<SOL, PNX, NAUX>;
    const SplitMethod<LIM> meth{a};
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* const dsm = reinterpret_cast<double*>(smem_raw);
    R* const rsm = reinterpret_cast<R*>(smem_raw + L::ND * 8);

    // broadcast from lane 0: the compiler then knows each half's branch to be uniform in
    // a warp and keeps its loop counters and ring slots in uniform registers
    const bool yrole = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0) >= HALF / 32;
    const int t = yrole ? threadIdx.x - HALF : threadIdx.x;
    const int pl = t / NXC;
    const int c = t - pl * NXC;
    const int pg = blockIdx.x * a.ppc + pl;
    const int s1 = NY + 2;  // iteration s updates row s - 4, the last of them NY - 2

    const bool active = STRIP ? c < NX : pl < a.ppc && pg < a.npatches;
    const int col = active ? t : 0;  // threads without a patch read (never write) column 0
    const PatchDesc* D = (a.desc && active) ? a.desc + pg : nullptr;
    int slot = 0;
    if constexpr (STRIP) slot = __ldg(a.strip.grid);  // every patch has the same cell size
    else if (active && !a.desc) slot = a.slots[pg];
    const int req = D ? D->req : -1;
    SOL sol{R(a.grav), R(a.gamma), R(a.gamma1), R(a.drytol)};
    if constexpr (FWAVE) {
        sol.gdbl = a.grav;
        sol.drytol_d = a.drytol;
        sol.ctol2 = sqrt(dmax(a.drytol * a.grav, 1e-6));
    }
    double pdt, pdx, pdy;
    bool save_last;
    {
        const PatchMeta* mt = D ? &D->meta : a.meta + slot;
        pdx = active ? mt->dx : 1.0;
        pdy = active ? mt->dy : 1.0;
        save_last = !STRIP && active && (mt->flags & PATCH_SAVE_LAST);
        pdt = D ? D->dt : step_dt(a, active ? mt->level : 0);
    }
    double* const q = (D ? D->q : a.q + (int64_t)slot * a.q_stride) + c;
    const double* const qin = (D ? D->q : a.q + (int64_t)slot * a.q_stride) + c;
    // strip: the mesh column the values come from, whether a wall mirrors it, the
    // distance between components
    bool wallx = false;
    const int xs = STRIP ? strip_inside(x0 - MBC + c, a.strip.n, a.strip.bc[0], a.strip.bc[1], wallx) : 0;
    const int plane = STRIP ? a.strip.nxp * a.strip.nxp : NXC * NXC;
    int pslot = 0;  // strip: slot of the patch read (Y half) or written (X half) now
    const double dtdx = pdt / pdx, dtdy = pdt / pdy;
    R smax = R(0);     // largest |s| over the CFL interfaces of this thread's sweep
    bool bad = false;  // a Riemann problem the reference would stop on (reported as a NaN CFL)

    R* const rb = rsm + col;
    double* const db = dsm + col;
    QT* qb;  // state and aux rings
    int QO, AO;
    if constexpr (L::QD) { qb = db; QO = L::DQ; AO = L::DAX; }
    else { qb = rb; QO = L::Q; AO = L::AX; }
    auto abs_sign = [](R sv) -> R {
        if constexpr (FWAVE) return copysign(R(1), sv);
        else return fabs(sv);
    };
    // ring slots of rows s, s-1, s-2 (three-slot rings) and of row s in the state ring
    constexpr int NQ = L::NQ;
    constexpr bool ASYNC = NQ == 6;
    int a0 = 0, a1 = 2, a2 = 1, qs = 0;
    auto qslot = [&](int d) -> int { const int k = qs - d; return k < 0 ? k + NQ : k; };  // of row s-d, d >= 0

    if (yrole) {
        const double* const aux = (NAUX > 0 && active) ? (D ? D->aux : a.aux + (int64_t)slot * a.aux_stride) + c : nullptr;
        double* const qlast = (D ? D->qlast : a.qlast + (int64_t)slot * a.q_stride) + c;
        const R rdtdy = R(dtdy), rhdtdy = R(0.5 * dtdy);
        const bool ycol = active && c >= 1 && c <= NX - 2;
        // interface f (final next): Roe averages and wave strengths, fluctuations, dot
        // products of its waves with those of f-1
        typename SOL::Roe yR{};
        R yam[M], yap[M], ydotl[W], gRm_prev[M], gRp_prev[M];  // gR: transverse parts into row f-1 (KEEPY: in shared memory)
#pragma unroll
        for (int m = 0; m < M; ++m) yam[m] = yap[m] = gRm_prev[m] = gRp_prev[m] = R(0);
#pragma unroll
        for (int mw = 0; mw < W; ++mw) ydotl[mw] = R(0);
        if constexpr (FWAVE) {
            if (active) {
#pragma unroll
                for (int k = 0; k < SOL::NWV; ++k) rb[L::KW + k * PNX] = R(0);
            }
        }
        // address of row `row`, component 0, and the components a wall negates; strip:
        // rows come in order, the slot is looked up again at patch edges and outside
        // the domain
        auto row_at = [&](int row, unsigned& neg) -> const double* {
            neg = 0u;
            if constexpr (!STRIP) return qin + row * NXC;
            const int ym = y0 - MBC + row;
            bool wally;
            const int y = strip_inside(ym, a.strip.n, a.strip.bc[2], a.strip.bc[3], wally);
            if (row == 0 || ym <= 0 || ym >= a.strip.n || (y & ((1 << a.strip.lg) - 1)) == 0)
                pslot = strip_slot(a.strip, xs, y);
            neg = (wallx ? 2u : 0u) ^ (wally ? 4u : 0u);
            return a.qsrc + ((int64_t)pslot * a.q_stride + strip_cell(a.strip, xs, y));
        };
        if constexpr (L::KEEPY) {
            if (active) {
#pragma unroll
                for (int m = 0; m < 2 * M; ++m) rb[L::KY + m * PNX] = R(0);
            }
        }
        unsigned neg = 0u;  // of row s
        if constexpr (ASYNC) {
            if (active) {
                const double* p = row_at(0, neg);
#pragma unroll
                for (int m = 0; m < M; ++m) copy_async8(&qb[QO + (qs * M + m) * PNX], p + m * plane);
            }
        }
        for (int s = 0; s <= s1; ++s) {
            const int b0 = s & 1;
            double qn[M], an[NAUX > 0 ? NAUX : 1];
            const bool ld = active && s < NY;
            unsigned neg1 = 0u;
            if constexpr (ASYNC) {
                copy_async_wait();  // row s, asked for an iteration ago
                if (active && s + 1 < NY) {
                    const double* p = row_at(s + 1, neg1);
                    const int k = qs + 1 == NQ ? 0 : qs + 1;
#pragma unroll
                    for (int m = 0; m < M; ++m) copy_async8(&qb[QO + (k * M + m) * PNX], p + m * plane);
                }
            } else if (ld) {
                const double* p = row_at(s, neg);
#pragma unroll
                for (int m = 0; m < M; ++m) qn[m] = p[m * plane];
            }
            if constexpr (NAUX > 0) {
                if (ld) {
#pragma unroll
                    for (int k = 0; k < NAUX; ++k) {
                        if constexpr (STRIP) an[k] = strip_aux(a, x0 - MBC + c, y0 - MBC + s, k);
                        else an[k] = aux[(k * NXC + s) * NXC];
                    }
                }
            }
            // ---- y-interface i = s-1 (between rows s-2 and s-1): averages, wave strengths,
            // dot products of its waves with those of f = i-1 ----
            const int i = s - 1;
            const bool yraw = ycol && i >= 1 && i < NY;
            typename SOL::Roe yRn{};
            R wn[FWAVE ? W : 1][M], amn[M], apn[M], ydotr[W], w[W][M], ysp[W];
            QT qD[M], qU[M];
            typename SOL::Cell cD, cU;
            auto load_pair = [&]() {
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    qD[m] = qb[QO + (qslot(2) * M + m) * PNX];
                    qU[m] = qb[QO + (qslot(1) * M + m) * PNX];
                }
                R* kd = reinterpret_cast<R*>(&cD);
                R* ku = reinterpret_cast<R*>(&cU);
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    kd[k] = rb[L::CELL + (a2 * NC + k) * PNX];
                    ku[k] = rb[L::CELL + (a1 * NC + k) * PNX];
                }
            };
#pragma unroll
            for (int mw = 0; mw < W; ++mw) ydotr[mw] = R(0);
            if constexpr (FWAVE) {
                sol.speeds(yR, ysp);
                int w0 = 0;
#pragma unroll
                for (int mw = 0; mw < W; ++mw)
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        if (SOL::nz(mw, wave_rel(2, m))) w[mw][m] = rb[L::KW + (w0++) * PNX];
                        wn[mw][m] = R(0);
                    }
            } else {
                sol.waves(2, yR, w, ysp);
            }
            if (yraw) {
                load_pair();
                R(*wi)[M];
                R we[W][M], se[W];
                if constexpr (FWAVE) {
                    bool bd = false;
                    sol.rpn2b(2, qD, qU, qb[AO + a2 * NAUX * PNX], qb[AO + a1 * NAUX * PNX], wn, yRn.s, amn, apn, bd);
                    bad = bad || bd;
                    wi = wn;
                } else {
                    sol.roe(2, qD, qU, cD, cU, yRn);
                    sol.waves(2, yRn, we, se);
                    wi = we;
                }
#pragma unroll
                for (int mw = 0; mw < W; ++mw) {
                    R d = R(0);
                    bool first = true;
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        if (!SOL::nz(mw, wave_rel(2, m))) continue;
                        const R p = w[mw][m] * wi[mw][m];
                        d = first ? p : d + p;
                        first = false;
                    }
                    ydotr[mw] = d;  // dot(w(i-1), w(i))
                }
            }
            // ---- final y-interface f = s-2 ----
            const int f = s - 2;
            R FYm[M], FYp[M];
            double GYd[M], GYu[M];
#pragma unroll
            for (int m = 0; m < M; ++m) {
                FYm[m] = FYp[m] = R(0);
                GYd[m] = GYu[m] = 0.0;
            }
            // clawpack 5: interfaces MBC..MBC+MX carry fluxes; f = MBC+MX+1 only
            // closes the transverse sum of cell row MBC+MX
            const bool yblk = ycol && (R15 ? (f >= MBC && f <= MBC + MY + 1) : f >= 1 && f <= NY - 1);
            if (yblk) {
                const bool fact = !R15 || f <= MBC + MY;
                const bool inner = R15 ? fact : (f >= MBC && f <= MBC + MY);
                const bool god = R15 ? fact : f <= NY - 2;
                if (inner) {
#pragma unroll
                    for (int mw = 0; mw < W; ++mw) smax = absmax(smax, ysp[mw]);
                }
                R cq[M];
#pragma unroll
                for (int m = 0; m < M; ++m) cq[m] = R(0);
                if (meth.second_order() && fact) {
                    if (inner) {
                        R num[W], wn2[W], phi[W];
#pragma unroll
                        for (int mw = 0; mw < W; ++mw) {
                            wn2[mw] = R(0);
                            bool first = true;
#pragma unroll
                            for (int m = 0; m < M; ++m) {
                                if (!SOL::nz(mw, wave_rel(2, m))) continue;
                                const R p = w[mw][m] * w[mw][m];
                                wn2[mw] = first ? p : wn2[mw] + p;
                                first = false;
                            }
                            num[mw] = (ysp[mw] > R(0)) ? ydotl[mw] : ydotr[mw];
                        }
                        limiter_values<V5, W>(num, wn2, [&](int mw) { return meth.lim(mw); }, phi);
#pragma unroll
                        for (int mw = 0; mw < W; ++mw)
#pragma unroll
                            for (int m = 0; m < M; ++m)
                                if (SOL::nz(mw, wave_rel(2, m))) w[mw][m] = phi[mw] * w[mw][m];
                    }
#pragma unroll
                    for (int mw = 0; mw < W; ++mw) {
                        const R as = fabs(ysp[mw]);
                        const R k = abs_sign(ysp[mw]) * (R(1) - as * rdtdy);
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            if (!SOL::nz(mw, wave_rel(2, m))) continue;
                            cq[m] = mw == 0 ? k * w[mw][m] : cq[m] + k * w[mw][m];
                        }
                    }
                }
                R am[M], ap[M];
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    R fmv = god ? yam[m] : R(0);
                    R fpv = god ? -yap[m] : R(0);
                    if (meth.second_order()) { fmv = fmv + R(0.5) * cq[m]; fpv = fpv + R(0.5) * cq[m]; }
                    FYm[m] = fmv;
                    FYp[m] = fpv;
                    am[m] = yam[m];
                    ap[m] = yap[m];
                    if (meth.transverse2() && god) { am[m] = am[m] + cq[m]; ap[m] = ap[m] - cq[m]; }
                }
                if constexpr (TR) {
                    R gLm[M], gLp[M];
                    if (meth.transverse() && fact) {
                        sol.rpt2(2, am, yR, R(0), R(0), gLm, gLp);
#pragma unroll
                        for (int m = 0; m < M; ++m) { gLm[m] = rhdtdy * gLm[m]; gLp[m] = rhdtdy * gLp[m]; }
                    } else {
#pragma unroll
                        for (int m = 0; m < M; ++m) gLm[m] = gLp[m] = R(0);
                    }
                    // cell row f-1 is complete: gadd(f-1,.,1) = (0 - gL(f)) - gR(f-1)
                    R* const keep = rb + L::KY;
                    if constexpr (L::KEEPY) {
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            gRm_prev[m] = keep[m * PNX];
                            gRp_prev[m] = keep[(M + m) * PNX];
                        }
                    }
                    if (R15 ? (f - 1 >= MBC && f - 1 <= MBC + MY) : f - 1 >= 1) {
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            GYd[m] = -(double)gLm[m] - (double)gRm_prev[m];
                            GYu[m] = -(double)gLp[m] - (double)gRp_prev[m];
                        }
                    }
                    if (meth.transverse() && fact) {
                        sol.rpt2(2, ap, yR, R(0), R(0), gRm_prev, gRp_prev);
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            gRm_prev[m] = rhdtdy * gRm_prev[m];
                            gRp_prev[m] = rhdtdy * gRp_prev[m];
                        }
                    } else {
#pragma unroll
                        for (int m = 0; m < M; ++m) gRm_prev[m] = gRp_prev[m] = R(0);
                    }
                    if constexpr (L::KEEPY) {
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            keep[m * PNX] = gRm_prev[m];
                            keep[(M + m) * PNX] = gRp_prev[m];
                        }
                    }
                }
            }
            if (active) {
                R* fym = rb + L::FYM + b0 * (M * PNX);
                R* fyp = rb + L::FYP + a2 * (M * PNX);
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    fym[m * PNX] = FYm[m];
                    fyp[m * PNX] = FYp[m];
                }
                if constexpr (TR) {
                    double* gy = db + L::GY + (b0 ^ 1) * (2 * M * PNX);
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        gy[m * PNX] = GYd[m];
                        gy[(M + m) * PNX] = GYu[m];
                    }
                }
            }
            // ---- the fluctuations of interface i, which is final next ----
            yR = yRn;
#pragma unroll
            for (int mw = 0; mw < W; ++mw) ydotl[mw] = ydotr[mw];
            if (yraw) {
                if constexpr (FWAVE) {
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        yam[m] = amn[m];
                        yap[m] = apn[m];
                    }
                } else {
                    load_pair();
                    R we[W][M], se[W];
                    sol.waves(2, yR, we, se);
                    sol.fluct(2, qD, qU, cD, cU, we, se, yam, yap);
                }
            } else {
#pragma unroll
                for (int m = 0; m < M; ++m) yam[m] = yap[m] = R(0);
            }
            if constexpr (FWAVE) {
                int w0 = 0;
#pragma unroll
                for (int mw = 0; mw < W; ++mw)
#pragma unroll
                    for (int m = 0; m < M; ++m)
                        if (SOL::nz(mw, wave_rel(2, m))) {
                            if (active) rb[L::KW + w0 * PNX] = wn[mw][m];
                            ++w0;
                        }
            }
            // ---- row s and its cell quantities ----
            if (ld) {
                R qr[M];
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    QT* ring = &qb[QO + (qs * M + m) * PNX];
                    if constexpr (ASYNC) qn[m] = *ring;
                    if constexpr (STRIP) {
                        if ((neg >> m) & 1u) {
                            qn[m] = -qn[m];
                            if constexpr (ASYNC) *ring = qn[m];
                        }
                    }
                    if (save_last) qlast[(m * NXC + s) * NXC] = qn[m];
                    if constexpr (!ASYNC) *ring = QT(qn[m]);
                    qr[m] = R(qn[m]);
                }
                if constexpr (NC > 0) {
                    typename SOL::Cell k;
                    sol.prep(qr, k);
                    const R* kk = reinterpret_cast<const R*>(&k);
#pragma unroll
                    for (int j = 0; j < NC; ++j) rb[L::CELL + (a0 * NC + j) * PNX] = kk[j];
                }
                if constexpr (NAUX > 0) {
#pragma unroll
                    for (int k = 0; k < NAUX; ++k) qb[AO + (a0 * NAUX + k) * PNX] = QT(an[k]);
                }
            }
            if constexpr (ASYNC) neg = neg1;
            row_barrier<2 * HALF>();
            const int n0 = a2;
            a2 = a1;
            a1 = a0;
            a0 = n0;
            qs = qs + 1 == NQ ? 0 : qs + 1;
        }
        smax = rdtdy * smax;
    } else {
        const R rdtdx = R(dtdx), rhdtdx = R(0.5 * dtdx);
        R xam[M], xap[M], gRm[M], gRp[M];  // fluctuations of row s-2, transverse parts of row s-3
        typename SOL::Roe xR{};
        double GXu_prev[M], GXs_prev[M];
        if constexpr (L::KEEPX) {
            if (active) {
#pragma unroll
                for (int m = 0; m < 2 * M; ++m) rb[L::KX + m * PNX] = R(0);
            }
        }
#pragma unroll
        for (int m = 0; m < M; ++m) {
            xam[m] = xap[m] = gRm[m] = gRp[m] = R(0);
            GXu_prev[m] = GXs_prev[m] = 0.0;
        }
        for (int s = 0; s <= s1; ++s) {
            const int b0 = s & 1;
            // ---- GX(c, k), k = s-3: GXu(row k-1) + GXd(row k) ----
            const int r = s - 4;
            const bool upd = active && r >= 0 && r <= NY - 2 &&
                             (V5 || STRIP ? (r >= MBC && r < MBC + MY && c >= MBC && c < MBC + MX) : c <= NX - 2);
            double qold[M];
            int64_t at = (int64_t)r * NXC;  // of the cell in the patch's column (strip: in the arenas)
            if constexpr (STRIP) {
                if (upd) {
                    const int y = y0 + r - MBC;
                    if (r == MBC || (y & ((1 << a.strip.lg) - 1)) == 0) pslot = strip_slot(a.strip, xs, y);
                    at = (int64_t)pslot * a.q_stride + strip_cell(a.strip, xs, y);
                }
            }
#pragma unroll
            for (int m = 0; m < M; ++m) {
                if constexpr (ASYNC) qold[m] = qb[QO + (qslot(4) * M + m) * PNX];
                else qold[m] = upd ? (STRIP ? a.qsrc : qin)[at + m * plane] : 0.0;
            }
            double GXs_new[M];
            if constexpr (TR) {
                const int k = s - 3;
                const bool xint = active && k >= 1 && k <= NY - 2 && (V5 ? (c >= MBC && c <= MBC + MX) : c >= 1);
                const R* gl = rb + L::GL + (b0 ^ 1) * (2 * M * PNX);
                if constexpr (L::KEEPX) {
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        gRm[m] = rb[L::KX + m * PNX];
                        gRp[m] = rb[L::KX + (M + m) * PNX];
                    }
                }
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    double gxd = 0.0, gxu = 0.0;
                    if (xint) {
                        if (c + 1 <= NX - 1) {
                            gxd = -(double)gl[m * PNX + 1] - (double)gRm[m];
                            gxu = -(double)gl[(M + m) * PNX + 1] - (double)gRp[m];
                        } else {
                            gxd = -(double)gRm[m];
                            gxu = -(double)gRp[m];
                        }
                    }
                    GXs_new[m] = GXu_prev[m] + gxd;
                    GXu_prev[m] = gxu;
                }
            }
            // ---- update of cell row r = s-4 ----
            bool tsr = false;
            const int ti = c - MBC + 1, tj = r - MBC + 1;
            if constexpr (TSYNC) {
                // the boundary fluctuations of the cells next to the patch edges
                // (clawpack46_time_sync_accumulate_waves, clawpack5_time_sync_accumulate_waves),
                // which the clawpack 5 update computes but does not apply to ghost cells
                const bool iin = ti >= 1 && ti <= MX, jin = tj >= 1 && tj <= MX;
                const bool iedge = ti == 0 || ti == 1 || ti == MX || ti == MX + 1;
                const bool jedge = tj == 0 || tj == 1 || tj == MX || tj == MX + 1;
                tsr = active && r >= 0 && r <= NY - 2 && ((iedge && jin) || (jedge && iin));
            }
            if (upd || tsr) {
                const R* fx = rb + L::FX + a1 * (2 * M * PNX);
                const double* gy = db + L::GY + b0 * (2 * M * PNX);
                const R* fym = rb + L::FYM + (b0 ^ 1) * (M * PNX);
                const R* fyp = rb + L::FYP + a1 * (M * PNX);
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const double fxm1 = fx[m * PNX + 1];  // FP32 flux parts widen exactly
                    const double fxp0 = fx[(M + m) * PNX];
                    double fmv = fxm1, fpv = fxp0, gmv = fym[m * PNX], gpv = fyp[m * PNX];
                    if constexpr (TR) {
                        const double gyu_l = (c >= 1) ? gy[(M + m) * PNX - 1] : 0.0;
                        const double gyd_r = gy[m * PNX + 1];
                        fmv = (fxm1 + gy[(M + m) * PNX]) + gyd_r;  // fm(i+1, j)
                        fpv = (fxp0 + gyu_l) + gy[m * PNX];        // fp(i, j)
                        gmv = GXs_new[m] + gmv;                    // gm(i, j+1)
                        gpv = GXs_prev[m] + gpv;                   // gp(i, j)
                    }
                    if (upd) (STRIP ? a.q : q)[at + m * plane] = qold[m] - dtdx * (fmv - fpv) - dtdy * (gmv - gpv);
                    if constexpr (TSYNC) {
                        if (tsr) {
                            // each register element has exactly one writer
                            const RegLayout RL{MXP, MXP, M};
                            double* Rg = a.treg + (int64_t)slot * a.treg_stride;
                            const double tdy = pdt * pdy, tdx = pdt * pdx;
                            if (tj >= 1 && tj <= MX) {
                                const int k = (tj - 1) + MX * m;
                                if (ti == 1) Rg[RL.fp(0) + k] = Rg[RL.fp(0) + k] - tdy * fpv;
                                if (ti == 0) Rg[RL.fm(0) + k] = Rg[RL.fm(0) + k] + tdy * fmv;       // fm(1, j)
                                if (ti == MX) Rg[RL.fm(1) + k] = Rg[RL.fm(1) + k] + tdy * fmv;      // fm(mx+1, j)
                                if (ti == MX + 1) Rg[RL.fp(1) + k] = Rg[RL.fp(1) + k] - tdy * fpv;  // fp(mx+1, j)
                            }
                            if (ti >= 1 && ti <= MX) {
                                const int k = (ti - 1) + MX * m;
                                if (tj == 1) Rg[RL.gp(0) + k] = Rg[RL.gp(0) + k] - tdx * gpv;
                                if (tj == 0) Rg[RL.gm(0) + k] = Rg[RL.gm(0) + k] + tdx * gmv;       // gm(i, 1)
                                if (tj == MX) Rg[RL.gm(1) + k] = Rg[RL.gm(1) + k] + tdx * gmv;      // gm(i, my+1)
                                if (tj == MX + 1) Rg[RL.gp(1) + k] = Rg[RL.gp(1) + k] - tdx * gpv;  // gp(i, my+1)
                            }
                        }
                    }
                }
            }
            if constexpr (TR) {
#pragma unroll
                for (int m = 0; m < M; ++m) GXs_prev[m] = GXs_new[m];
            }
            // ---- x-row k = s-2: limiter, corrections, transverse parts ----
            {
                const int k = s - 2;
                if (active && k >= 0 && k <= NY - 2) {
                    R* fx = rb + L::FX + a2 * (2 * M * PNX);
                    R* gl = rb + L::GL + b0 * (2 * M * PNX);
                    const bool xint = k >= 1 && (R15 ? (c >= MBC && c <= MBC + MX) : c >= 1);
                    if (xint) {
                        const R* xw = rb + L::XW + b0 * (SOL::NWV * PNX);
                        R cq[M], xwl[W][M], xsl[W];
                        sol.speeds(xR, xsl);
                        {
                            int w0 = 0;
#pragma unroll
                            for (int mw = 0; mw < W; ++mw)
#pragma unroll
                                for (int m = 0; m < M; ++m)
                                    if (SOL::nz(mw, m)) xwl[mw][m] = xw[(w0++) * PNX];
                        }
#pragma unroll
                        for (int m = 0; m < M; ++m) cq[m] = R(0);
                        if (meth.second_order()) {
                            if (c >= MBC && c <= MBC + MX) {
                                R num[W], wn2[W], phi[W];
                                int w0 = 0;
#pragma unroll
                                for (int mw = 0; mw < W; ++mw) {
                                    R dl = R(0), dr = R(0);
                                    wn2[mw] = R(0);
                                    bool first = true;
#pragma unroll
                                    for (int m = 0; m < M; ++m) {
                                        if (!SOL::nz(mw, m)) continue;
                                        const R wc = xwl[mw][m];
                                        const R p = wc * wc, l = xw[w0 * PNX - 1] * wc, g = wc * xw[w0 * PNX + 1];
                                        wn2[mw] = first ? p : wn2[mw] + p;
                                        dl = first ? l : dl + l;
                                        dr = first ? g : dr + g;
                                        first = false;
                                        ++w0;
                                    }
                                    num[mw] = (xsl[mw] > R(0)) ? dl : dr;
                                }
                                limiter_values<V5, W>(num, wn2, [&](int mw) { return meth.lim(mw); }, phi);
#pragma unroll
                                for (int mw = 0; mw < W; ++mw)
#pragma unroll
                                    for (int m = 0; m < M; ++m)
                                        if (SOL::nz(mw, m)) xwl[mw][m] = phi[mw] * xwl[mw][m];
                            }
#pragma unroll
                            for (int mw = 0; mw < W; ++mw) {
                                const R as = fabs(xsl[mw]);
                                const R kk = abs_sign(xsl[mw]) * (R(1) - as * rdtdx);
#pragma unroll
                                for (int m = 0; m < M; ++m) {
                                    if (!SOL::nz(mw, m)) continue;
                                    cq[m] = mw == 0 ? kk * xwl[mw][m] : cq[m] + kk * xwl[mw][m];
                                }
                            }
                        }
                        R am[M], ap[M];
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            R fmv = (c <= NX - 2) ? xam[m] : R(0);
                            R fpv = (c <= NX - 2) ? -xap[m] : R(0);
                            if (meth.second_order()) { fmv = fmv + R(0.5) * cq[m]; fpv = fpv + R(0.5) * cq[m]; }
                            fx[m * PNX] = fmv;
                            fx[(M + m) * PNX] = fpv;
                            am[m] = xam[m];
                            ap[m] = xap[m];
                            if (meth.transverse2() && c <= NX - 2) { am[m] = am[m] + cq[m]; ap[m] = ap[m] - cq[m]; }
                        }
                        if constexpr (TR) {
                            if (meth.transverse()) {
                                R bm[M], bp[M];
                                sol.rpt2(1, am, xR, R(0), R(0), bm, bp);
#pragma unroll
                                for (int m = 0; m < M; ++m) {
                                    gl[m * PNX] = rhdtdx * bm[m];
                                    gl[(M + m) * PNX] = rhdtdx * bp[m];
                                }
                                sol.rpt2(1, ap, xR, R(0), R(0), bm, bp);
#pragma unroll
                                for (int m = 0; m < M; ++m) {
                                    gRm[m] = rhdtdx * bm[m];
                                    gRp[m] = rhdtdx * bp[m];
                                }
                            } else {
#pragma unroll
                                for (int m = 0; m < M; ++m) {
                                    gl[m * PNX] = gl[(M + m) * PNX] = R(0);
                                    gRm[m] = gRp[m] = R(0);
                                }
                            }
                            if constexpr (L::KEEPX) {
#pragma unroll
                                for (int m = 0; m < M; ++m) {
                                    rb[L::KX + m * PNX] = gRm[m];
                                    rb[L::KX + (M + m) * PNX] = gRp[m];
                                }
                            }
                        }
                    } else {
#pragma unroll
                        for (int m = 0; m < M; ++m) {
                            fx[m * PNX] = R(0);
                            fx[(M + m) * PNX] = R(0);
                            if constexpr (TR) gl[m * PNX] = gl[(M + m) * PNX] = R(0);
                        }
                    }
                }
            }
            // ---- x-row k = s-1: Riemann problem at x-interface c ----
            {
                const int k = s - 1;
                if (active && k >= 1 && k <= NY - 2 && c >= 1) {
                    const QT* qr = qb + QO + qslot(1) * (M * PNX);
                    QT qL[M], qR[M];
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        qL[m] = qr[m * PNX - 1];
                        qR[m] = qr[m * PNX];
                    }
                    R xwl[W][M], xsl[W];
                    if constexpr (FWAVE) {
                        bool bd = false;
                        const QT* ax = qb + AO + a1 * (NAUX * PNX);
                        sol.rpn2b(1, qL, qR, ax[-1], ax[0], xwl, xsl, xam, xap, bd);
                        bad = bad || bd;
#pragma unroll
                        for (int mw = 0; mw < W; ++mw) xR.s[mw] = xsl[mw];
                    } else {
                        typename SOL::Cell cl, cr;
                        R* kl = reinterpret_cast<R*>(&cl);
                        R* kr = reinterpret_cast<R*>(&cr);
#pragma unroll
                        for (int j = 0; j < NC; ++j) {
                            kl[j] = rb[L::CELL + (a1 * NC + j) * PNX - 1];
                            kr[j] = rb[L::CELL + (a1 * NC + j) * PNX];
                        }
                        sol.roe(1, qL, qR, cl, cr, xR);
                        sol.waves(1, xR, xwl, xsl);
                        sol.fluct(1, qL, qR, cl, cr, xwl, xsl, xam, xap);
                    }
                    R* xw = rb + L::XW + (b0 ^ 1) * (SOL::NWV * PNX);
                    int w0 = 0;
#pragma unroll
                    for (int mw = 0; mw < W; ++mw) {
#pragma unroll
                        for (int m = 0; m < M; ++m)
                            if (SOL::nz(mw, m)) xw[(w0++) * PNX] = xwl[mw][m];
                        if (c >= MBC && c <= MBC + MX) smax = absmax(smax, xsl[mw]);
                    }
                }
            }
            row_barrier<2 * HALF>();
            const int n0 = a2;
            a2 = a1;
            a1 = a0;
            a0 = n0;
            qs = qs + 1 == NQ ? 0 : qs + 1;
        }
        smax = rdtdx * smax;
    }

    // ---- CFL: flux2's max(dtdx*s, -dtdx*s).  Rounding is monotone, so one
    // product with the largest |s| gives the reference's value exactly. ----
    double cfl = (double)smax;
    if (bad) cfl = __longlong_as_double(0x7ff8000000000000LL);  // NaN: wins the max, reported by the host
    const int lane = threadIdx.x & 31;
    if (a.desc) {
        // patches of different solves share warps: reduce over the lanes of each
        // solve (max of the non-negative bit patterns, high word then low word)
        const unsigned grp = __match_any_sync(0xffffffffu, req);
        const unsigned long long b = (unsigned long long)__double_as_longlong(active ? cfl : 0.0);
        const unsigned hi = __reduce_max_sync(grp, (unsigned)(b >> 32));
        const unsigned lo = __reduce_max_sync(grp, ((unsigned)(b >> 32) == hi) ? (unsigned)b : 0u);
        if (req >= 0 && lane == __ffs(grp) - 1 && a.cfl_out)
            atomicMax(a.cfl_out + req, ((unsigned long long)hi << 32) | lo);
    } else {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) cfl = nanmax(cfl, __shfl_xor_sync(0xffffffffu, cfl, off));
        if (lane == 0 && a.cfl_out) atomicMax(a.cfl_out, (unsigned long long)__double_as_longlong(cfl));
    }
}

// ---------------------------------------------------------------------------
// Host-side launcher
// ---------------------------------------------------------------------------
namespace {

// A launch of G CTAs on an SM array that holds W at once ends with a wave of
// G mod W CTAs that lasts a whole patch sweep.  Rather than fill all waves but
// the last, the patches are spread over as many CTAs as the same number of
// waves holds: every CTA sweeps fewer patches, and its rows take less time.
inline int split_patches_per_cta(int n, int most, int per_wave) {
    const int waves = (n + most * per_wave - 1) / (most * per_wave);
    return std::min(most, std::max(1, (n + waves * per_wave - 1) / (waves * per_wave)));
}

template <class SOL, int MXP, int NAUX, int HALF, int LIM, bool TSYNC>
cudaError_t launch_split_one(const StepArgs& a, cudaStream_t st) {
    constexpr int NXC = MXP == 0 ? HALF : MXP + 4;
    constexpr int PPB = HALF / NXC;
    static_assert(PPB >= 1, "patch wider than half a CTA");
    using L = SplitSmem<SOL, PPB * NXC, NAUX>;
    static_assert(L::BYTES <= 227 * 1024, "shared memory of the CTA");
    constexpr auto kernel = step_kernel_split<SOL, MXP, NAUX, HALF, LIM, TSYNC>;
    if (a.npatches <= 0) return cudaSuccess;
    static PerDevice<> kept;
    int per_wave = 0;  // CTAs the SM array holds at once
    const cudaError_t e = per_device(kept, &per_wave, [&](int* n) {
        const cudaError_t f = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES);
        return f != cudaSuccess ? f : resident_ctas(kernel, 2 * HALF, L::BYTES, n);
    });
    if (e != cudaSuccess) return e;
    StepArgs b = a;
    int blocks;
    if constexpr (MXP == 0) {
        strip_plan(b.strip, HALF - 4, per_wave, 7);
        blocks = b.strip.nsx * b.strip.nsy;
    } else {
        b.ppc = split_patches_per_cta(a.npatches, PPB, per_wave);
        blocks = (a.npatches + b.ppc - 1) / b.ppc;
    }
    kernel<<<blocks, 2 * HALF, L::BYTES, st>>>(b);
    return cudaGetLastError();
}

// Threads of each half of a CTA (one CTA per SM).  As many columns as fit without
// spills, which cost more than the warps they add: FP64 shallow water 118 registers at
// 2 x 256 threads (1,024 patches of mx = 32: 0.139 ms; 2 x 192: 0.175), Euler 156 at
// 2 x 192, where its 1.2 KB of shared memory per column end (0.282 ms; 2 x 128: 0.348).
// The mixed forms of Euler and GeoClaw at 2 x 320 (Euler, 4,096 patches of mx = 16:
// 0.121 ms; 2 x 256 0.167, 2 x 384 0.155), of shallow water at 2 x 384 (strips of a
// 1024 x 1024 mesh 0.069 ms; 2 x 256 0.084, 2 x 320 0.073).
template <class SOL>
constexpr int split_half() {
    if (sizeof(typename SOL::Real) == 4) return SOL::M == 3 && !SOL::FWAVE ? 384 : 320;
    return SOL::M == 4 ? 192 : 256;
}

template <class SOL, int MXP, int NAUX, bool TSYNC>
cudaError_t launch_split_lim(const StepArgs& a, cudaStream_t st) {
    constexpr int HALF = split_half<SOL>();
    bool mc = a.order0 == 2 && (SOL::FWAVE || a.order1 == 2);  // the f-wave solver has no transverse parts
    for (int mw = 0; mw < SOL::W; ++mw) mc = mc && a.mthlim[mw] == 4;
    if (mc) return launch_split_one<SOL, MXP, NAUX, HALF, 4, TSYNC>(a, st);
    return launch_split_one<SOL, MXP, NAUX, HALF, 0, TSYNC>(a, st);
}

template <class SOL, int MXP, int NAUX>
cudaError_t launch_split_ts(const StepArgs& a, cudaStream_t st) {
    if constexpr (MXP > 0 && split_time_sync<SOL>())
        if (a.treg) return launch_split_lim<SOL, MXP, NAUX, true>(a, st);
    return launch_split_lim<SOL, MXP, NAUX, false>(a, st);
}

template <class SOL, int NAUX>
cudaError_t launch_split_mx(int mx, const StepArgs& a, cudaStream_t st) {
    if (a.strip.grid && a.strip.patches) return cudaErrorNotSupported;
    if (a.strip.grid) return launch_split_ts<SOL, 0, NAUX>(a, st);  // strips take patches of any size
    switch (mx) {
        case 8: return launch_split_ts<SOL, 8, NAUX>(a, st);
        case 16: return launch_split_ts<SOL, 16, NAUX>(a, st);
        case 32: return launch_split_ts<SOL, 32, NAUX>(a, st);
        case 64:
            if constexpr (sizeof(typename SOL::Real) == 8 && !SOL::V5 && !SOL::FWAVE) return launch_split_ts<SOL, 64, NAUX>(a, st);
            return cudaErrorNotSupported;
        default: return cudaErrorNotSupported;
    }
}

}  // namespace

}  // namespace fcb
