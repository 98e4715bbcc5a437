// Scalar advection on a mesh of one level: step2 + flux2 + conservative update in
// strips of columns and rows (fcb_strip.cuh), the ghost exchange folded into the loads.
// One thread per column, rows streamed top to bottom, one CTA barrier per row.
//
// Reference: src/solvers/fc2d_clawpack4.6/fortran_source/clawpack46_step2.f,
// clawpack46_flux2.f, clawpack46_step2_wrap.f with advection/2d/all/clawpack46_rpn2adv.f,
// clawpack46_rpt2adv.f and swirl's b4step2.f (the clawpack 5 routines have the same
// arithmetic on interior cells).  Every operation keeps the reference's association,
// and the flux sums their order:
//   fm(i,j) = (FXm + GYu[col i-1]) + GYd[col i],   gm(i,j) = (GXu[row j-1] + GXd[row j]) + FYm
//   q = q - dtdx*(fm(i+1,j) - fp(i,j)) - dtdy*(gm(i,j+1) - gp(i,j)).
//
// Iteration s (row s arrived): x-interfaces of row s-1 (waves from the states of
// columns c-2 .. c+1, so Riemann problem, limiter and corrections are one stage);
// y-interface s-1; transverse sums of x-row s-2; update of cell row s-3.
//
// What bounds it: instruction issue.  A cell needs about 103 FP64 operations (0.094 ms
// for 16.8 M cells at the FP64 rate).  So every lane runs every stage without tests on
// its column: lanes outside the strip's interior compute values nobody reads, and
// only the store asks.  The split velocities min(u, 0), max(u, 0) are formed once per
// cell from the sign bit and exchanged, instead of twelve times by compare and select.
// B200, level 8, mx = 16 (16.8 M cells), one step: FP64 0.369 ms with the pipelined form
// on the same strips, 0.274 ms here; mixed 0.272 and 0.196 ms.  4.2 M cells: 43.6 M
// warp instructions against 63 M, FP64 pipe 39 % busy, issue slots 56 %.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "fcb_device.h"
#include "fcb_launch.hpp"
#include "fcb_solvers.cuh"
#include "fcb_strip.cuh"

namespace fcb {

namespace {

// min(x, 0) and max(x, 0): x where its sign bit says so, else zero.  A NaN stays in one or
// both, and so in |u|, from which the CFL number is taken (comparisons would drop it).
__device__ __forceinline__ void split_sign(double x, double& neg, double& pos) {
    const int hi = __double2hiint(x), lo = __double2loint(x), mask = hi >> 31;
    neg = __hiloint2double(hi & mask, lo & mask);
    pos = __hiloint2double(hi & ~mask, lo & ~mask);
}
__device__ __forceinline__ void split_sign(float x, float& neg, float& pos) {
    asm("min.NaN.f32 %0, %1, 0f00000000;" : "=f"(neg) : "f"(x));
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(pos) : "f"(x));
}

// A product that is rounded by itself: the mixed form's fluctuations round as those of
// fcb_step_pipe.cuh, whose products and sums are in different stages.
__device__ __forceinline__ double mul_alone(double x, double y) { return x * y; }
__device__ __forceinline__ float mul_alone(float x, float y) { return __fmul_rn(x, y); }

// psi at a node: (sin^2(pi x) sin^2(pi y))/pi.  The FP64 form rounds the quotient as
// the reference's division does; the mixed form multiplies by 1/pi (one more
// rounding, far below its FP32 solves).
template <typename R>
__device__ __forceinline__ double adv_psi(double tx, double ty) {
    if constexpr (sizeof(R) == sizeof(double)) return div_pi(tx * ty);
    else return (tx * ty) * (1.0 / 3.141592653589793);
}

// Rings [slot][column] of a CTA of TPB columns; columns c-2 .. c+1 are read, so two
// elements before the first ring and one after the last belong to the buffer.
template <int TPB, typename R>
struct AdvSmem {
    static constexpr int GYD = 0, GYU = 2 * TPB, ND = 4 * TPB + 2;  // FP64: y transverse sums, 2 slots each
    static constexpr int NQ = sizeof(R) == 8 ? 4 : 2;
    static constexpr int Q = 0;              // NQ slots: states (FP64: the old value of the update too)
    static constexpr int UP = Q + NQ * TPB;  // 4 slots: max(u, 0)
    static constexpr int VM = UP + 4 * TPB;  // 4 slots: min(v, 0)
    static constexpr int VP = VM + 4 * TPB;  // 2 slots: max(v, 0)
    static constexpr int FX = VP + 2 * TPB;  // 4 slots: x fluxes (left part)
    static constexpr int FXP = FX + 4 * TPB;   // 4 slots each: x fluxes (right part), y fluxes (upper part),
    static constexpr int FYP = FXP + 4 * TPB;  // own column
    static constexpr int GLM = FYP + 4 * TPB, GLP = GLM + 2 * TPB;  // 2 slots each: x transverse parts to the left
    static constexpr int NR = GLP + 2 * TPB + 4;
    static constexpr int TY = (ND + 2) * 8 + ((NR * (int)sizeof(R) + 15) / 16) * 16;  // bytes: sin^2 of the node rows
    static constexpr int bytes(int rows) { return TY + (rows + 6) * 8; }
};

// Values a thread carries from one row to the next.
template <typename R>
struct AdvState {
    double q0, q1, q2, q3, qn;      // rows s, s-1, s-2, s-3 (the last two in the mixed form only); row s+1
    double pc, pr;                  // psi at the nodes (c, s+1), (c+1, s+1)
    R um0, um1, um2;                // min(u, 0) of rows s, s-1, s-2 (the other parts are in the rings)
    R upn;                          // max(u, 0) of column c+1, row s-2
    R dy, dotl;                     // y-interface s-1: wave, its product with that of s-2
    R gym, gyp;                     // y transverse parts of interface s-2 into row s-2
    R gxm, gxp;                     // x transverse parts of row s-2 to the right
    double gxu, gxs;                // GXu of row s-3; GX of row s-3
    R fym1;                         // y flux (lower part) of interface s-2
    R sx, sy;                       // largest |u|, |v| over the CFL interfaces
    int sslot, dslot;
};

// Row `row` of this thread's column (rows come in order).
template <typename R>
__device__ __forceinline__ double adv_load(const StepArgs& a, int x, int y0, AdvState<R>& S, int row) {
    const StripArgs& g = a.strip;
    const int ym = y0 - 2 + row;
    bool wall;  // a scalar is not negated at a wall
    const int y = strip_inside(ym, g.n, g.bc[2], g.bc[3], wall);
    if (row == 0 || ym <= 0 || ym >= g.n || (y & ((1 << g.lg) - 1)) == 0) S.sslot = strip_slot(g, x, y);
    return a.qsrc[(int64_t)S.sslot * a.q_stride + strip_cell(g, x, y)];
}

struct AdvConst {
    double dtdx, dtdy, vty, vtx, tx, tx1;
    int x, xm, y0, ny;
    bool in;  // an interior column
};

// J >= 0: s = J (mod 4), so every ring slot is a constant.
template <typename R, int AUXK, int TPB, int LIM, int J>
__device__ __forceinline__ void adv_row(const StepArgs& a, const AdvConst& T, AdvState<R>& S, R* rb, double* db,
                                        const double* ty, int s) {
    using L = AdvSmem<TPB, R>;
    auto sl = [&](int d, int n) -> int { return (J >= 0 ? ((J - d) % n + n) % n : (s - d) & (n - 1)) * TPB; };
    const bool second = LIM > 0 || a.order0 == 2, trans = LIM > 0 || a.order1 > 0,
               trans2 = LIM > 0 || (a.order0 > 1 && a.order1 == 2);
    const int mth = LIM > 0 ? LIM : a.mthlim[0];
    const R rdx = R(T.dtdx), rdy = R(T.dtdy), hdx = R(0.5 * T.dtdx), hdy = R(0.5 * T.dtdy);
    const int ny = T.ny;
    // row s+2 for the iteration after next
    double qnn = 0.0;
    if (s + 2 < ny) qnn = adv_load(a, T.x, T.y0, S, s + 2);

    // ---- speeds of row s+1 ----
    R u = R(0), v = R(0), um, up, vm, vp;
    if constexpr (AUXK == AUX_SWIRL) {
        // swirl/user_4.6/b4step2.f, psi.f: u = vty*(psi(c,j+1) - psi(c,j)), v = -vtx*(psi(c+1,j) - psi(c,j))
        const double t = ty[min(s + 2, ny)];
        const double pc = adv_psi<R>(T.tx, t), pr = adv_psi<R>(T.tx1, t);
        u = R(T.vty * (pc - S.pc));
        v = R(-T.vtx * (S.pr - S.pc));
        S.pc = pc;
        S.pr = pr;
    } else {
        const int row = min(s + 1, ny - 1);
        u = R(strip_aux(a, T.xm, T.y0 - 2 + row, 0));
        v = R(strip_aux(a, T.xm, T.y0 - 2 + row, 1));
    }
    split_sign(u, um, up);
    split_sign(v, vm, vp);

    // ---- x-interface c of row s-1 and y-interface s-1 ----
    const R* Q = rb + L::Q + sl(1, L::NQ);
    const R q = R(S.q1), ql = Q[-1], qll = Q[-2], qr = Q[1];
    const R dx = q - ql, dxl = ql - qll, dxr = qr - q;
    const R dn = R(S.q0) - q;  // wave of y-interface s
    const R up1 = rb[L::UP + sl(1, 4)], vm1 = rb[L::VM + sl(1, 4)], vp1 = rb[L::VP + sl(1, 2)], vp0 = rb[L::VP + sl(0, 2)];
    const R au = up1 - S.um1, av = vp1 - vm1;  // |u|, |v|: one part is zero
    R amx = mul_alone(S.um1, dx), apx = mul_alone(up1, dx);
    R amy = mul_alone(vm1, S.dy), apy = mul_alone(vp1, S.dy);
    const R dotr = S.dy * dn;
    R cx = R(0), cy = R(0);
    if (second) {
        const R wn2[2] = {dx * dx, S.dy * S.dy};
        const R num[2] = {up1 > R(0) ? dxl * dx : dx * dxr, vp1 > R(0) ? S.dotl : dotr};
        R phi[2];
        limiter_values<false, 2>(num, wn2, [&](int) { return mth; }, phi);
        cx = au * (R(1) - au * rdx) * (phi[0] * dx);
        cy = av * (R(1) - av * rdy) * (phi[1] * S.dy);
    }
    R fxm = amx, fxp = -apx, fym = amy, fyp = -apy;
    if (second) {
        fxm = fxm + R(0.5) * cx;
        fxp = fxp + R(0.5) * cx;
        fym = fym + R(0.5) * cy;
        fyp = fyp + R(0.5) * cy;
    }
    if (trans2) {
        amx = amx + cx;
        apx = apx - cx;
        amy = amy + cy;
        apy = apy - cy;
    }
    R glm = R(0), glp = R(0), grm = R(0), grp = R(0), hlm = R(0), hlp = R(0), hrm = R(0), hrp = R(0);
    const R upn = rb[L::UP + sl(1, 4) + 1];  // max(u, 0) of column c+1, row s-1
    if (trans) {
        // into rows below and above: v of columns c-1 (left) and c (right), rows s-1 and s
        glm = hdx * (rb[L::VM + sl(1, 4) - 1] * amx);
        glp = hdx * (rb[L::VP + sl(0, 2) - 1] * amx);
        grm = hdx * (vm1 * apx);
        grp = hdx * (vp0 * apx);
        // into columns left and right: u of columns c and c+1, rows s-2 (below) and s-1
        hlm = hdy * (S.um2 * amy);
        hlp = hdy * (S.upn * amy);
        hrm = hdy * (S.um1 * apy);
        hrp = hdy * (upn * apy);
    }
    // ---- transverse sums of x-row s-2: GX = GXu(row below) + GXd(row) ----
    const double gxd = -(double)rb[L::GLM + sl(2, 2) + 1] - (double)S.gxm;
    const double gxu = -(double)rb[L::GLP + sl(2, 2) + 1] - (double)S.gxp;
    const double gx = S.gxu + gxd;
    // ---- update of cell row s-3 ----
    {
        const double fxm1 = rb[L::FX + sl(3, 4) + 1];
        const double* yd = db + L::GYD + sl(3, 2);
        const double* yu = db + L::GYU + sl(3, 2);
        const double fmv = (fxm1 + yu[0]) + yd[1];
        const double fpv = ((double)rb[L::FXP + sl(3, 4)] + yu[-1]) + yd[0];
        const double gmv = gx + (double)S.fym1;
        const double gpv = S.gxs + (double)rb[L::FYP + sl(3, 4)];
        double qold;
        if constexpr (L::NQ == 4) qold = rb[L::Q + sl(3, 4)];
        else qold = S.q3;
        const double qv = qold - T.dtdx * (fmv - fpv) - T.dtdy * (gmv - gpv);
        const int r = s - 3;
        if (T.in && r >= 2 && r < ny - 2) {
            const int y = T.y0 + r - 2;
            if (r == 2 || (y & ((1 << a.strip.lg) - 1)) == 0) S.dslot = strip_slot(a.strip, T.x, y);
            a.q[(int64_t)S.dslot * a.q_stride + strip_cell(a.strip, T.x, y)] = qv;
        }
    }
    // ---- y transverse sums of row s-2; CFL interfaces: x of rows 1 .. ny-2, y 2 .. ny-2 ----
    const double gyd = -(double)hlm - (double)S.gym, gyu = -(double)hlp - (double)S.gyp;
    if (s >= 2 && s < ny) S.sx = absmax(S.sx, au);
    if (s >= 3 && s < ny) S.sy = absmax(S.sy, av);
    // ---- publish ----
    rb[L::Q + sl(0, L::NQ)] = R(S.q0);
    rb[L::UP + sl(-1, 4)] = up;
    rb[L::VM + sl(-1, 4)] = vm;
    rb[L::VP + sl(-1, 2)] = vp;
    rb[L::FX + sl(1, 4)] = fxm;
    rb[L::FXP + sl(1, 4)] = fxp;
    rb[L::FYP + sl(1, 4)] = fyp;
    rb[L::GLM + sl(1, 2)] = glm;
    rb[L::GLP + sl(1, 2)] = glp;
    db[L::GYD + sl(2, 2)] = gyd;
    db[L::GYU + sl(2, 2)] = gyu;
    // ---- the next row ----
    if constexpr (L::NQ == 2) {
        S.q3 = S.q2;
        S.q2 = S.q1;
    }
    S.q1 = S.q0;
    S.q0 = S.qn;
    S.qn = qnn;
    S.um2 = S.um1;
    S.um1 = S.um0;
    S.um0 = um;
    S.upn = upn;
    S.dy = dn;
    S.dotl = dotr;
    S.gym = hrm;
    S.gyp = hrp;
    S.gxm = grm;
    S.gxp = grp;
    S.gxu = gxu;
    S.gxs = gx;
    S.fym1 = fym;
    __syncthreads();
}

// CTAs per SM the registers are cut to: FP64 4 (128 registers, one spilled: 0.274 ms
// for 16.8 M cells; 5: 0.317, 6: 0.338), mixed 6 (0.196 ms; 7: 0.201, 8: 0.217).
template <typename R>
constexpr int kAdvCtas = sizeof(R) == 4 ? 6 : 4;

template <typename R, int AUXK, int TPB, int LIM>
__global__ void __launch_bounds__(TPB, kAdvCtas<R>) step_kernel_adv(const StepArgs a) {
    using L = AdvSmem<TPB, R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const StripArgs& g = a.strip;
    const int c = threadIdx.x;
    double* const db = reinterpret_cast<double*>(smem_raw) + 2 + c;
    R* const rb = reinterpret_cast<R*>(smem_raw + (L::ND + 2) * 8) + 2 + c;
    double* const ty = reinterpret_cast<double*>(smem_raw + L::TY);

    const int x0 = blockIdx.x % g.nsx * g.w, y0 = blockIdx.x / g.nsx * g.h;
    const int mxs = min(g.w, g.n - x0), mys = min(g.h, g.n - y0);
    AdvConst T;
    T.y0 = y0;
    T.ny = mys + 4;
    T.in = c >= 2 && c < mxs + 2;
    T.xm = min(x0 - 2 + c, g.n + 1);  // lanes beyond the strip repeat its last column
    bool wall;
    T.x = strip_inside(T.xm, g.n, g.bc[0], g.bc[1], wall);
    const PatchMeta& meta = a.meta[__ldg(g.grid)];  // every patch has the same cell size
    const double ddx = meta.dx, ddy = meta.dy;
    const double dt = step_dt(a, meta.level);
    T.dtdx = dt / ddx;
    T.dtdy = dt / ddy;
    T.vty = T.vtx = T.tx = T.tx1 = 0.0;
    AdvState<R> S{};
    R u0, v0;  // speeds of row 0
    S.q0 = adv_load(a, T.x, y0, S, 0);
    S.qn = adv_load(a, T.x, y0, S, 1);
    if constexpr (AUXK == AUX_SWIRL) {
        // cell edges are exact multiples of the spacing (checked on the host), so psi is
        // evaluated once per node
        constexpr double pi = 3.141592653589793;  // 4*atan(1) in double precision
        const double vt = step_vt(a, meta.level);
        T.vty = vt / ddy;
        T.vtx = vt / ddx;
        const double sc = sin(pi * (g.ax + (double)T.xm * ddx)), sr = sin(pi * (g.ax + (double)(T.xm + 1) * ddx));
        T.tx = sc * sc;
        T.tx1 = sr * sr;
        for (int k = c; k <= T.ny; k += TPB) {
            const double sy = sin(pi * (g.ay + (double)(y0 - 2 + k) * ddy));
            ty[k] = sy * sy;
        }
        __syncthreads();
        const double p0 = adv_psi<R>(T.tx, ty[0]), r0 = adv_psi<R>(T.tx1, ty[0]);
        S.pc = adv_psi<R>(T.tx, ty[1]);
        S.pr = adv_psi<R>(T.tx1, ty[1]);
        u0 = R(T.vty * (S.pc - p0));
        v0 = R(-T.vtx * (r0 - p0));
    } else {
        u0 = R(strip_aux(a, T.xm, y0 - 2, 0));
        v0 = R(strip_aux(a, T.xm, y0 - 2, 1));
    }
    R up0, vm0, vp0;
    split_sign(u0, S.um0, up0);
    split_sign(v0, vm0, vp0);
    // every ring starts at zero: the first rows read slots that no row has filled
    for (int k = c - 2; k < L::ND; k += TPB) (db - c)[k] = 0.0;
    for (int k = c - 2; k < L::NR - 2; k += TPB) (rb - c)[k] = R(0);
    __syncthreads();
    rb[L::UP] = up0;
    rb[L::VM] = vm0;
    rb[L::VP] = vp0;
    __syncthreads();

    int s = 0;
    for (; s + 4 <= T.ny + 1; s += 4) {
        adv_row<R, AUXK, TPB, LIM, 0>(a, T, S, rb, db, ty, s);
        adv_row<R, AUXK, TPB, LIM, 1>(a, T, S, rb, db, ty, s + 1);
        adv_row<R, AUXK, TPB, LIM, 2>(a, T, S, rb, db, ty, s + 2);
        adv_row<R, AUXK, TPB, LIM, 3>(a, T, S, rb, db, ty, s + 3);
    }
    for (; s <= T.ny; ++s) adv_row<R, AUXK, TPB, LIM, -1>(a, T, S, rb, db, ty, s);

    // CFL: flux2's max(dtdx*s, -dtdx*s); rounding is monotone, so one product with the
    // largest |s| gives the reference's value exactly.  x-interfaces of columns 2 .. mxs+2,
    // y-interfaces of columns 1 .. mxs+2.
    double cfl = 0.0;
    if (c >= 1 && c <= mxs + 2) {
        const R cy = R(T.dtdy) * S.sy, cx = c >= 2 ? R(T.dtdx) * S.sx : R(0);
        cfl = (double)nanmax(cx, cy);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) cfl = nanmax(cfl, __shfl_xor_sync(0xffffffffu, cfl, off));
    if ((c & 31) == 0 && a.cfl_out) atomicMax(a.cfl_out, (unsigned long long)__double_as_longlong(cfl));
}

template <typename R, int AUXK, int TPB, int LIM>
cudaError_t launch_adv_one(const StepArgs& a, cudaStream_t st) {
    using L = AdvSmem<TPB, R>;
    constexpr auto kernel = step_kernel_adv<R, AUXK, TPB, LIM>;
    static PerDevice<> kept;
    int per_wave = 0;
    const cudaError_t e = per_device(kept, &per_wave, [&](int* n) {
        const cudaError_t f = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::bytes(kStripRowsMax));
        return f != cudaSuccess ? f : resident_ctas(kernel, TPB, L::bytes(256), n);
    });
    if (e != cudaSuccess) return e;
    StepArgs b = a;
    strip_plan(b.strip, TPB - 4, per_wave, 5);
    kernel<<<b.strip.nsx * b.strip.nsy, TPB, L::bytes(b.strip.h), st>>>(b);
    return cudaGetLastError();
}

// One scalar advection step in strips (a.strip and a.qsrc set).  Order (2, 2) with the MC
// or van Leer limiter is fixed at compile time.
template <typename R>
cudaError_t launch_adv(int aux_kind, int claw_version, const StepArgs& a0, cudaStream_t st) {
    if (!a0.strip.grid || a0.desc || !a0.qsrc || a0.qsrc == a0.q) return cudaErrorInvalidValue;
    StepArgs a = a0;
    // clawpack5_inlinelimiter.f sends codes above 5 to its first branch (minmod)
    if (claw_version == 5 && a.mthlim[0] > 5) a.mthlim[0] = 1;
    const int lim = a.order0 == 2 && a.order1 == 2 && (a.mthlim[0] == 3 || a.mthlim[0] == 4) ? a.mthlim[0] : 0;
    if (aux_kind == AUX_SWIRL) {
        if (lim == 4) return launch_adv_one<R, AUX_SWIRL, 128, 4>(a, st);
        if (lim == 3) return launch_adv_one<R, AUX_SWIRL, 128, 3>(a, st);
        return launch_adv_one<R, AUX_SWIRL, 128, 0>(a, st);
    }
    if (aux_kind != AUX_STORED || a.maux < 2) return cudaErrorNotSupported;
    if (lim == 4) return launch_adv_one<R, AUX_STORED, 128, 4>(a, st);
    if (lim == 3) return launch_adv_one<R, AUX_STORED, 128, 3>(a, st);
    return launch_adv_one<R, AUX_STORED, 128, 0>(a, st);
}

}  // namespace

}  // namespace fcb
