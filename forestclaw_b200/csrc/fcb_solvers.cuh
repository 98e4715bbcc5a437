// Point-wise Riemann solvers and the wave limiter for the device step kernel.
//
// Each solver restates one reference Fortran routine for a single interface
// (V5: the clawpack 5 twin of the routine where its arithmetic differs)
// (the reference loops over a whole 1-D slice; the per-interface arithmetic is
// the same).  The Roe averages that the reference passes from rpn2 to rpt2
// through COMMON /comroe/ travel here in an explicit per-interface struct.
// Association of every expression follows the Fortran source so that, compiled
// without FMA contraction, the results equal the reference's bit for bit.
#pragma once
#include <cuda_runtime.h>

#include "fcb_arith.cuh"

namespace fcb {

template <typename T>
__device__ __forceinline__ T dmax(T a, T b) { return a > b ? a : b; }
template <typename T>
__device__ __forceinline__ T dmin(T a, T b) { return a < b ? a : b; }
// Maximum for the CFL number that keeps a NaN: a NaN wave speed (a negative
// depth, say) must reach the host as a NaN CFL, which the library reports as
// FCB_ERR_NUMERIC.  For numbers it equals dmax.
template <typename T>
__device__ __forceinline__ T nanmax(T a, T b) { return (b > a || b != b) ? b : a; }
// max(m, |s|) for m >= 0 as the unsigned maximum of the bit patterns: for
// non-negative numbers the same value as dmax, and a NaN (its magnitude's bits
// are the largest) is kept, at the cost of one integer compare-select.
__device__ __forceinline__ double absmax(double m, double s) {
    const unsigned long long a = (unsigned long long)__double_as_longlong(m);
    const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(s));
    return __longlong_as_double((long long)(a > b ? a : b));
}
__device__ __forceinline__ float absmax(float m, float s) {
    const unsigned a = __float_as_uint(m), b = __float_as_uint(fabsf(s));
    return __uint_as_float(a > b ? a : b);
}

// ---------------------------------------------------------------------------
// Scalar advection: applications/clawpack/advection/2d/all/clawpack46_rpn2adv.f,
// clawpack46_rpt2adv.f.  The normal speed is the edge velocity aux(i,j,ixy);
// the transverse splitting uses the two edge velocities of the cell pair.
// ---------------------------------------------------------------------------
// clawpack5_rpn2adv.f90 / clawpack5_rpt2adv.f90 have the same arithmetic.
template <int W_, typename R = double, bool V5_ = false>
struct AdvectionSolver {
    using Real = R;
    static constexpr bool V5 = V5_;
    static constexpr bool FWAVE = false;
    static constexpr int M = 1;
    static constexpr int W = W_;
    struct Roe {};
    // no per-cell quantities to share between the interfaces of a cell
    struct Cell {};
    static constexpr int NC = 0;
    R grav, gamma, gamma1, drytol;  // unused
    __device__ __forceinline__ void prep(const R*, Cell&) const {}
    __device__ __forceinline__ void rpn2c(int ixy, const R* qL, const R* qR, const Cell&, const Cell&, R speed,
                                          R (*wave)[M], R* s, R* amdq, R* apdq, Roe& rr) const {
        rpn2(ixy, qL, qR, speed, wave, s, amdq, apdq, rr);
    }
    __device__ __forceinline__ void rpn2(int /*ixy*/, const R* qL, const R* qR, R speed,
                                         R (*wave)[M], R* s, R* amdq, R* apdq,
                                         Roe&) const {
        const R delta = qR[0] - qL[0];
#pragma unroll
        for (int mw = 0; mw < W; ++mw) {
            wave[mw][0] = delta;
            s[mw] = speed;
        }
        // the reference starts both sums at 0; starting at the first term differs
        // only in the sign of a zero result
        R am = dmin(s[0], R(0.0)) * wave[0][0];
        R ap = dmax(s[0], R(0.0)) * wave[0][0];
#pragma unroll
        for (int mw = 1; mw < W; ++mw) {
            am = am + dmin(s[mw], R(0.0)) * wave[mw][0];
            ap = ap + dmax(s[mw], R(0.0)) * wave[mw][0];
        }
        amdq[0] = am;
        apdq[0] = ap;
    }
    // aux_dn = aux2(i1,kv), aux_up = aux3(i1,kv)
    __device__ __forceinline__ void rpt2(int /*ixy*/, const R* asdq, const Roe&, R aux_dn,
                                         R aux_up, R* bm, R* bp) const {
        bm[0] = dmin(aux_dn, R(0.0)) * asdq[0];
        bp[0] = dmax(aux_up, R(0.0)) * asdq[0];
    }
};

// Scalar advection on a mapped grid: applications/clawpack/advection/2d/all/
// clawpack46_rpn2adv_manifold.f, clawpack46_rpt2adv_manifold.f.  The arithmetic
// of rpn2adv / rpt2adv with the edge velocities in aux(2:3), after the
// capacity kappa = area / (dx dy) in aux(1) (mcapa = 1), which the step then
// applies (clawpack46_step2.f:122-126,191-195, clawpack46_flux2.f:134-220,
// clawpack46_step2_wrap.f:118-121).
// V5: clawpack5_rpn2adv_manifold.f90 / rpt2adv_manifold.f90, the same arithmetic.
template <int W_, bool V5_ = false>
struct AdvectionManifoldSolver : AdvectionSolver<W_, double, V5_> {};

// Stored-aux layout of a solver: the first aux component its Riemann solvers
// read, and whether aux(1) is the capacity.
template <class SOL>
struct AuxLayout {
    static constexpr int SHIFT = 0;
    static constexpr bool CAPA = false;
};
template <int W_, bool V5_>
struct AuxLayout<AdvectionManifoldSolver<W_, V5_>> {
    static constexpr int SHIFT = 1;
    static constexpr bool CAPA = true;
};

// ---------------------------------------------------------------------------
// Shallow water, Roe with entropy fix:
// applications/clawpack/shallow/2d/rp/clawpack46_rpn2.f:1-247, clawpack46_rpt2.f:1-74
// ---------------------------------------------------------------------------
// V5: clawpack5_rpn2.f90, clawpack5_rpt2.f90 (a1, a3 scaled by 0.5/a instead
// of divided by 2a; the Roe averages clawpack5_rpt2 recomputes equal rpn2's).
//
// A Riemann problem is solved in three parts, so that a kernel can keep the Roe
// averages and wave strengths (roe) and form the waves (waves) or the fluctuations
// (fluct) when it needs them.  Each takes the common case without branches: the
// quotients with one divisor share its reciprocal (fcb_arith.cuh), and the entropy
// fix, which needs the speeds of the states left and right of the middle waves only
// for their signs, decides those by comparing squares (u > c exactly when u > 0 and
// (hu)^2 > g h^3) with a margin of 0.1 %, far above rounding.  A transonic wave, a
// comparison inside the margin and operands near underflow take the reference's
// formulas as they stand (exact_*).
template <typename R, bool V5_ = false>
struct SweRoeT {
    using Real = R;
    static constexpr bool V5 = V5_;
    static constexpr bool FWAVE = false;
    static constexpr int M = 3;
    static constexpr int W = 3;
    // y: what divides by 2a (clawpack 5: 0.5/a; 0: use the operator); a1..a3: wave strengths
    struct Roe { R u, v, a, y, a1, a2, a3; };
    // Quantities of one cell that every Riemann problem it takes part in (two
    // x- and two y-interfaces) evaluates with the same operations on the same
    // operands: sqrt(h), hu/sqrt(h), hv/sqrt(h); and g h^3 for the sign tests.
    // The step kernels compute them once per cell; the values are bit-identical.
    struct Cell { R sq, rq[2], gh3; };
    static constexpr int NC = 4;
    // wave components that are not zero by construction (component order: depth,
    // normal and transverse momentum): the middle wave is a shear
    static constexpr int NWV = 7;
    __host__ __device__ static constexpr bool nz(int mw, int rel) { return mw != 1 || rel == 2; }
    R grav, gamma, gamma1, drytol;  // drytol: GeoClaw only
    __device__ __forceinline__ void prep(const R* q, Cell& k) const {
        bool ok = true;
        k.sq = sqrt_ok(q[0], ok);
        const Dv<R> d(k.sq, ok);
        k.rq[0] = d(q[1], ok);
        k.rq[1] = d(q[2], ok);
        if (!ok) {
            seldom();
            k.sq = sqrt(q[0]);
            k.rq[0] = q[1] / k.sq;
            k.rq[1] = q[2] / k.sq;
        }
        k.gh3 = grav * q[0] * q[0] * q[0];
    }
    __device__ __forceinline__ void rpn2(int ixy, const R* qL, const R* qR, R speed,
                                         R (*wave)[M], R* s, R* amdq, R* apdq,
                                         Roe& rr) const {
        Cell cl, cr;
        prep(qL, cl);
        prep(qR, cr);
        rpn2c(ixy, qL, qR, cl, cr, speed, wave, s, amdq, apdq, rr);
    }
    __device__ __forceinline__ void rpn2c(int ixy, const R* qL, const R* qR, const Cell& cl, const Cell& cr,
                                          R /*speed*/, R (*wave)[M], R* s, R* amdq, R* apdq,
                                          Roe& rr) const {
        roe(ixy, qL, qR, cl, cr, rr);
        waves(ixy, rr, wave, s);
        fluct(ixy, qL, qR, cl, cr, wave, s, amdq, apdq);
    }
    __device__ __forceinline__ void roe(int ixy, const R* qL, const R* qR, const Cell& cl, const Cell& cr,
                                        Roe& rr) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        bool ok = true;
        const R h = (qL[0] + qR[0]) / R(2.0);
        const R hsq2 = cl.sq + cr.sq;  // sqrt(qL(1)) + sqrt(qR(1))
        const R su = cl.rq[mu - 1] + cr.rq[mu - 1], sv = cl.rq[mv - 1] + cr.rq[mv - 1];
        const Dv<R> dh(hsq2, ok);
        const R u = dh(su, ok);  // (qL(mu)/hsqrtl + qR(mu)/hsqrtr)/hsq2
        const R v = dh(sv, ok);
        const R a = sqrt_ok(grav * h, ok);
        const Dv<R> da(V5 ? a : R(2.0) * a, ok);
        rr.u = u; rr.v = v; rr.a = a;
        rr.y = V5 ? da.scaled(R(0.5)) : da.y;
        const R d1 = qR[0] - qL[0];
        const R d2 = qR[mu] - qL[mu];
        const R d3 = qR[mv] - qL[mv];
        rr.a1 = V5 ? ((u + a) * d1 - d2) * rr.y : da((u + a) * d1 - d2, ok);
        rr.a2 = -(v * d1) + d3;
        rr.a3 = V5 ? (-((u - a) * d1) + d2) * rr.y : da(-((u - a) * d1) + d2, ok);
        if (!ok) {
            seldom();
            rr = exact_roe(hsq2, su, sv, grav * h, d1, d2, d3);
        }
    }
    __device__ __forceinline__ void speeds(const Roe& rr, R* s) const {
        s[0] = rr.u - rr.a;
        s[1] = rr.u;
        s[2] = rr.u + rr.a;
    }
    __device__ __forceinline__ void waves(int ixy, const Roe& rr, R (*wave)[M], R* s) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        speeds(rr, s);
        wave[0][0] = rr.a1; wave[0][mu] = rr.a1 * s[0]; wave[0][mv] = rr.a1 * rr.v;
        wave[1][0] = R(0.0); wave[1][mu] = R(0.0); wave[1][mv] = rr.a2;
        wave[2][0] = rr.a3; wave[2][mu] = rr.a3 * s[2]; wave[2][mv] = rr.a3 * rr.v;
    }
    __device__ __forceinline__ void fluct(int ixy, const R* qL, const R* qR, const Cell& cl, const Cell& cr,
                                          const R (*wave)[M], const R* s, R* amdq, R* apdq) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        // entropy fix: left of the first wave the speed s0 = u - c of qL, right of it s1
        const R g = grav, lo = R(0.999), hi = R(1.001);
        const R mL = qL[mu], mL2 = mL * mL;
        const bool supL = mL > R(0.0) && mL2 > hi * cl.gh3;   // s0 > 0
        const bool subL = mL <= R(0.0) || mL2 < lo * cl.gh3;  // s0 < 0
        const R h1 = qL[0] + wave[0][0], hu1 = mL + wave[0][mu];
        const bool sub1 = h1 > R(0.0) && (hu1 <= R(0.0) || hu1 * hu1 < lo * (g * h1 * h1 * h1));  // s1 < 0
        // right of the third wave s03 = u + c of qR, left of it s3
        const bool right = s[1] <= R(0.0);
        const R mR = qR[mu];
        const bool supR = mR < R(0.0) && mR * mR > hi * cr.gh3;  // s03 < 0
        const R h3 = qR[0] - wave[2][0], hu3 = mR - wave[2][mu];
        const bool sub3 = h3 > R(0.0) && (hu3 >= R(0.0) || hu3 * hu3 < lo * (g * h3 * h3 * h3));  // s3 > 0
        const bool ok = (qL[0] > R(0.0)) & (supL | (subL & sub1)) & ((s[1] > R(0.0)) | (right & (sub3 | supR)));
        const R k0 = s[0] < R(0.0) ? s[0] : R(0.0);
        const R k1 = right ? s[1] : R(0.0);
        const R k2 = right && s[2] < R(0.0) ? s[2] : R(0.0);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            R am = k0 * wave[0][m];
            if (m == mv) am = am + k1 * wave[1][m];  // the other components are zero
            amdq[m] = am + k2 * wave[2][m];
        }
        if (!ok) {
            seldom();
            const Fluct e = exact_fluct(qL[0], mL, qL[mv], qR[0], mR, qR[mv], grav, wave[0][0], wave[1][mv], wave[2][0],
                                        wave[0][mu], wave[0][mv], wave[2][mu], wave[2][mv], s[0], s[1], s[2]);
            amdq[0] = e.am[0];
            amdq[mu] = e.am[1];
            amdq[mv] = e.am[2];
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            R df = s[0] * wave[0][m];
#pragma unroll
            for (int mw = 1; mw < W; ++mw)
                if (nz(mw, m == mv ? 2 : m == 0 ? 0 : 1)) df = df + s[mw] * wave[mw][m];
            apdq[m] = df - amdq[m];
        }
    }
    // The reference's formulas from the cells' quantities.  (From the states, with their
    // roots and quotients once more, the momenta of 1e-290 and less in the tail of a front
    // cost a first-order step of 16 patches of mx = 64 at CFL 0.02 189 us; 159 so.)
    static __device__ __forceinline__ Roe exact_roe(R hsq2, R su, R sv, R gh, R d1, R d2, R d3) {
        Roe rr;
        const R u = rr.u = su / hsq2;
        const R v = rr.v = sv / hsq2;
        const R a = rr.a = sqrt(gh);
        rr.a1 = V5 ? ((u + a) * d1 - d2) * (R(0.5) / a) : ((u + a) * d1 - d2) / (R(2.0) * a);
        rr.a2 = -(v * d1) + d3;
        rr.a3 = V5 ? (-((u - a) * d1) + d2) * (R(0.5) / a) : (-((u - a) * d1) + d2) / (R(2.0) * a);
        bool in = true;
        const Dv<R> da(V5 ? a : R(2.0) * a, in);
        rr.y = V5 ? R(0.5) / a : in ? da.y : R(0.0);
        return rr;
    }
    // The same, components in the order depth, normal, transverse.
    struct Fluct { R am[3]; };
    static __device__ __forceinline__ Fluct exact_fluct(R l0, R l1, R l2, R r0, R r1, R r2, R grav, R w00, R w12, R w20,
                                                     R w01, R w02, R w21, R w22, R sA, R sB, R sC) {
        Fluct e;
        R* am = e.am;
        const R s0 = l1 / l0 - sqrt(grav * l0);
        R sfract;
        if (s0 > R(0.0) && sA > R(0.0)) {
            am[0] = am[1] = am[2] = R(0.0);
            return e;
        }
        const R h1 = l0 + w00;
        const R hu1 = l1 + w01;
        const R s1 = hu1 / h1 - sqrt(grav * h1);
        if (s0 < R(0.0) && s1 > R(0.0)) sfract = s0 * ((s1 - sA) / (s1 - s0));
        else if (sA < R(0.0)) sfract = sA;
        else sfract = R(0.0);
        am[0] = sfract * w00;
        am[1] = sfract * w01;
        am[2] = sfract * w02;
        if (sB > R(0.0)) return e;
        am[2] = am[2] + sB * w12;  // the other components are zero
        const R s03 = r1 / r0 + sqrt(grav * r0);
        const R h3 = r0 - w20;
        const R hu3 = r1 - w21;
        const R s3 = hu3 / h3 + sqrt(grav * h3);
        if (s3 < R(0.0) && s03 > R(0.0)) sfract = s3 * ((s03 - sC) / (s03 - s3));
        else if (sC < R(0.0)) sfract = sC;
        else return e;
        am[0] = am[0] + sfract * w20;
        am[1] = am[1] + sfract * w21;
        am[2] = am[2] + sfract * w22;
        return e;
    }
    __device__ __forceinline__ void rpt2(int ixy, const R* asdq, const Roe& rr, R, R,
                                         R* bm, R* bp) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        const R u = rr.u, v = rr.v, a = rr.a;
        const R x1 = (v + a) * asdq[0] - asdq[mv], x3 = -((v - a) * asdq[0]) + asdq[mv];
        R a1, a3;
        if constexpr (V5) {
            a1 = rr.y * x1;  // y = 0.5/a
            a3 = rr.y * x3;
        } else {
            bool ok = sizeof(R) == 4 || rr.y != R(0.0);
            const Dv<R> d(2 * a, rr.y);
            a1 = d(x1, ok);
            a3 = d(x3, ok);
            if (!ok) {
                seldom();
                a1 = x1 / (2 * a);
                a3 = x3 / (2 * a);
            }
        }
        const R a2 = asdq[mu] - u * asdq[0];
        R waveb[3][3], sb[3];
        waveb[0][0] = a1; waveb[mu][0] = a1 * u; waveb[mv][0] = a1 * (v - a); sb[0] = v - a;
        waveb[0][1] = R(0.0); waveb[mu][1] = a2; waveb[mv][1] = R(0.0); sb[1] = v;
        waveb[0][2] = a3; waveb[mu][2] = a3 * u; waveb[mv][2] = a3 * (v + a); sb[2] = v + a;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            R m1 = dmin(sb[0], R(0.0)) * waveb[m][0], p1 = dmax(sb[0], R(0.0)) * waveb[m][0];
#pragma unroll
            for (int mw = 1; mw < 3; ++mw) {
                if (mw == 1 && m != mu) continue;  // waveb[m][1] is zero
                m1 = m1 + dmin(sb[mw], R(0.0)) * waveb[m][mw];
                p1 = p1 + dmax(sb[mw], R(0.0)) * waveb[m][mw];
            }
            bm[m] = m1;
            bp[m] = p1;
        }
    }
};

// ---------------------------------------------------------------------------
// Euler (4 equations), Roe with entropy fix:
// applications/clawpack/euler/2d/rp/clawpack46_rpn2_euler4.f:1-289,
// clawpack46_rpt2_euler4.f:290-386
// ---------------------------------------------------------------------------
// clawpack5_rpn2_euler4.f90 / clawpack5_rpt2_euler4.f90 have the same arithmetic.
template <typename R, bool V5_ = false>
struct Euler4RoeT {
    using Real = R;
    static constexpr bool V5 = V5_;
    static constexpr bool FWAVE = false;
    static constexpr int M = 4;
    static constexpr int W = 4;
    // y: what divides by 2a (0: use the operator); a1..a4: wave strengths
    struct Roe { R u, v, a, enth, g1a2, y, a1, a2, a3, a4; };
    // Quantities of one cell shared by the four Riemann problems it takes part
    // in: sqrt(rho), rho u/sqrt(rho), rho v/sqrt(rho), (E + p)/sqrt(rho); and
    // gamma p rho for the sign tests.  Every value is bit-identical.
    struct Cell { R sq, rq[2], rh, gpr; };
    static constexpr int NC = 5;
    // wave components that are not zero by construction (density, normal and
    // transverse momentum, energy): the second wave is a shear
    static constexpr int NWV = 14;
    __host__ __device__ static constexpr bool nz(int mw, int rel) { return mw != 1 || rel >= 2; }
    R grav, gamma, gamma1, drytol;  // drytol: GeoClaw only
    __device__ __forceinline__ void prep(const R* q, Cell& k) const {
        bool ok = true;
        k.sq = sqrt_ok(q[0], ok);
        const Dv<R> dr(q[0], ok), ds(k.sq, ok);
        const R ke = R(0.5) * (q[1] * q[1] + q[2] * q[2]);
        R p = gamma1 * (q[3] - dr(ke, ok));
        k.rq[0] = ds(q[1], ok);
        k.rq[1] = ds(q[2], ok);
        k.rh = ds(q[3] + p, ok);
        if (!ok) {
            seldom();
            k.sq = sqrt(q[0]);
            p = gamma1 * (q[3] - ke / q[0]);
            k.rq[0] = q[1] / k.sq;
            k.rq[1] = q[2] / k.sq;
            k.rh = (q[3] + p) / k.sq;
        }
        k.gpr = gamma * p * q[0];
    }
    __device__ __forceinline__ void rpn2(int ixy, const R* qL, const R* qR, R speed,
                                         R (*wave)[M], R* s, R* amdq, R* apdq,
                                         Roe& rr) const {
        Cell cl, cr;
        prep(qL, cl);
        prep(qR, cr);
        rpn2c(ixy, qL, qR, cl, cr, speed, wave, s, amdq, apdq, rr);
    }
    __device__ __forceinline__ void rpn2c(int ixy, const R* qL, const R* qR, const Cell& cl, const Cell& cr, R,
                                          R (*wave)[M], R* s, R* amdq, R* apdq,
                                          Roe& rr) const {
        roe(ixy, qL, qR, cl, cr, rr);
        waves(ixy, rr, wave, s);
        fluct(ixy, qL, qR, cl, cr, wave, s, amdq, apdq);
    }
    // The three parts of a Riemann problem as the shallow-water solver has them:
    // u > c exactly when rho u > 0 and (rho u)^2 > gamma p rho.
    __device__ __forceinline__ void roe(int ixy, const R* qL, const R* qR, const Cell& cl, const Cell& cr,
                                        Roe& rr) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        bool ok = true;
        const R rhsq2 = cl.sq + cr.sq;
        const R su = cl.rq[mu - 1] + cr.rq[mu - 1], sv = cl.rq[mv - 1] + cr.rq[mv - 1], sh = cl.rh + cr.rh;
        const Dv<R> dh(rhsq2, ok);
        const R u = dh(su, ok);  // (qL(mu)/rhsqrtl + qR(mu)/rhsqrtr)/rhsq2
        const R v = dh(sv, ok);
        const R enth = dh(sh, ok);  // ((qL(4)+pl)/rhsqrtl + (qR(4)+pr)/rhsqrtr)/rhsq2
        const R u2v2 = u * u + v * v;
        const R a2s = gamma1 * (enth - R(0.5) * u2v2);
        const R a = sqrt_ok(a2s, ok);
        const Dv<R> d2s(a2s, ok), da(R(2.0) * a, ok);
        rr.u = u; rr.v = v; rr.a = a; rr.enth = enth; rr.y = da.y;
        rr.g1a2 = d2s(gamma1, ok);
        const R d1 = qR[0] - qL[0];
        const R d2 = qR[mu] - qL[mu];
        const R d3 = qR[mv] - qL[mv];
        const R d4 = qR[3] - qL[3];
        rr.a3 = rr.g1a2 * ((enth - u2v2) * d1 + u * d2 + v * d3 - d4);
        rr.a2 = d3 - v * d1;
        rr.a4 = da(d2 + (a - u) * d1 - a * rr.a3, ok);
        rr.a1 = d1 - rr.a3 - rr.a4;
        if (!ok) {
            seldom();
            rr = exact_roe(rhsq2, su, sv, sh, d1, d2, d3, d4, gamma1);
        }
    }
    __device__ __forceinline__ void speeds(const Roe& rr, R* s) const {
        s[0] = rr.u - rr.a;
        s[1] = s[2] = rr.u;
        s[3] = rr.u + rr.a;
    }
    __device__ __forceinline__ void waves(int ixy, const Roe& rr, R (*wave)[M], R* s) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        const R u = rr.u, v = rr.v, ua = u * rr.a, u2v2 = u * u + v * v;
        speeds(rr, s);
        wave[0][0] = rr.a1; wave[0][mu] = rr.a1 * s[0]; wave[0][mv] = rr.a1 * v; wave[0][3] = rr.a1 * (rr.enth - ua);
        wave[1][0] = R(0.0); wave[1][mu] = R(0.0); wave[1][mv] = rr.a2; wave[1][3] = rr.a2 * v;
        wave[2][0] = rr.a3; wave[2][mu] = rr.a3 * u; wave[2][mv] = rr.a3 * v; wave[2][3] = rr.a3 * R(0.5) * u2v2;
        wave[3][0] = rr.a4; wave[3][mu] = rr.a4 * s[3]; wave[3][mv] = rr.a4 * v; wave[3][3] = rr.a4 * (rr.enth + ua);
    }
    __device__ __forceinline__ void fluct(int ixy, const R* qL, const R* qR, const Cell& cl, const Cell& cr,
                                          const R (*wave)[M], const R* s, R* amdq, R* apdq) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        // entropy fix: left of the first wave the speed s0 = u - c of qL, right of it s1.
        // The products with the density cancel where the pressure is small against
        // the energy: such states are left to exact_fluct().
        const R lo = R(0.999), hi = R(1.001), pmin = sizeof(R) == 8 ? R(1e-8) : R(1e-2);
        const R mL = qL[mu], mL2 = mL * mL;
        const bool posL = qL[0] > R(0.0) && cl.gpr > R(0.0), posR = qR[0] > R(0.0) && cr.gpr > R(0.0);
        const bool supL = posL && mL > R(0.0) && mL2 > hi * cl.gpr;     // s0 > 0
        const bool subL = posL && (mL <= R(0.0) || mL2 < lo * cl.gpr);  // s0 < 0
        const R r1 = qL[0] + wave[0][0], m1 = mL + wave[0][mu], t1 = qL[mv] + wave[0][mv];
        const R e1 = (qL[3] + wave[0][3]) * r1, pr1 = gamma1 * (e1 - R(0.5) * (m1 * m1 + t1 * t1));
        const bool sub1 = r1 > R(0.0) && pr1 > pmin * e1 && (m1 <= R(0.0) || m1 * m1 < lo * (gamma * pr1));  // s1 < 0
        // right of the fourth wave s3 = u + c of qR, left of it s2
        const bool right = s[1] < R(0.0);
        const R mR = qR[mu];
        const bool supR = posR && mR < R(0.0) && mR * mR > hi * cr.gpr;  // s3 < 0
        const R r2 = qR[0] - wave[3][0], m2 = mR - wave[3][mu], t2 = qR[mv] - wave[3][mv];
        const R e2 = (qR[3] - wave[3][3]) * r2, pr2 = gamma1 * (e2 - R(0.5) * (m2 * m2 + t2 * t2));
        const bool sub2 = r2 > R(0.0) && pr2 > pmin * e2 && (m2 >= R(0.0) || m2 * m2 < lo * (gamma * pr2));  // s2 > 0
        const bool ok = (supL | (subL & sub1)) & ((s[1] >= R(0.0)) | (right & (sub2 | supR)));
        const R k0 = s[0] < R(0.0) ? s[0] : R(0.0);
        const R k1 = right ? s[1] : R(0.0);
        const R k3 = right && s[3] < R(0.0) ? s[3] : R(0.0);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            R am = k0 * wave[0][m];
            if (m == mv || m == 3) am = am + k1 * wave[1][m];  // the other components are zero
            am = am + k1 * wave[2][m];                         // s[2] == s[1]
            amdq[m] = am + k3 * wave[3][m];
        }
        if (!ok) {
            seldom();
            ExactIn e;
            const int at[4] = {0, mu, mv, 3};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                e.l[m] = qL[at[m]];
                e.r[m] = qR[at[m]];
#pragma unroll
                for (int mw = 0; mw < 4; ++mw) e.w[mw][m] = wave[mw][at[m]];
                e.s[m] = s[m];
            }
            const Fluct f = exact_fluct(e, gamma, gamma1);
#pragma unroll
            for (int m = 0; m < 4; ++m) amdq[at[m]] = f.am[m];
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            R df = s[0] * wave[0][m];
#pragma unroll
            for (int mw = 1; mw < W; ++mw)
                if (mw != 1 || m == mv || m == 3) df = df + s[mw] * wave[mw][m];  // the shear's other components are zero
            apdq[m] = df - amdq[m];
        }
    }
    // The reference's formulas from the cells' quantities.
    static __device__ __forceinline__ Roe exact_roe(R rhsq2, R su, R sv, R sh, R d1, R d2, R d3, R d4, R gamma1) {
        Roe rr;
        const R u = rr.u = su / rhsq2;
        const R v = rr.v = sv / rhsq2;
        const R enth = rr.enth = sh / rhsq2;
        const R u2v2 = u * u + v * v;
        const R a2s = gamma1 * (enth - R(0.5) * u2v2);
        const R a = rr.a = sqrt(a2s);
        rr.g1a2 = gamma1 / a2s;
        rr.a3 = rr.g1a2 * ((enth - u2v2) * d1 + u * d2 + v * d3 - d4);
        rr.a2 = d3 - v * d1;
        rr.a4 = (d2 + (a - u) * d1 - a * rr.a3) / (R(2.0) * a);
        rr.a1 = d1 - rr.a3 - rr.a4;
        bool in = true;
        const Dv<R> da(R(2.0) * a, in);
        rr.y = in ? da.y : R(0.0);
        return rr;
    }
    // The same, components in the order density, normal and transverse momentum, energy.
    struct ExactIn { R l[4], r[4], w[4][4], s[4]; };
    struct Fluct { R am[4]; };
    static __device__ __forceinline__ Fluct exact_fluct(const ExactIn e, R gamma, R gamma1) {
        Fluct f;
        R* am = f.am;
        const R* s = e.s;
        const R pl = gamma1 * (e.l[3] - R(0.5) * (e.l[1] * e.l[1] + e.l[2] * e.l[2]) / e.l[0]);
        const R s0 = e.l[1] / e.l[0] - sqrt(gamma * pl / e.l[0]);
        R sfract;
        if (s0 >= R(0.0) && s[0] > R(0.0)) {
            am[0] = am[1] = am[2] = am[3] = R(0.0);
            return f;
        }
        {
            const R rho1 = e.l[0] + e.w[0][0];
            const R rhou1 = e.l[1] + e.w[0][1];
            const R rhov1 = e.l[2] + e.w[0][2];
            const R en1 = e.l[3] + e.w[0][3];
            const R p1 = gamma1 * (en1 - R(0.5) * (rhou1 * rhou1 + rhov1 * rhov1) / rho1);
            const R c1 = sqrt(gamma * p1 / rho1);
            const R s1 = rhou1 / rho1 - c1;
            if (s0 < R(0.0) && s1 > R(0.0)) sfract = s0 * (s1 - s[0]) / (s1 - s0);
            else if (s[0] < R(0.0)) sfract = s[0];
            else sfract = R(0.0);
            for (int m = 0; m < 4; ++m) am[m] = sfract * e.w[0][m];
        }
        if (s[1] >= R(0.0)) return f;
        for (int m = 0; m < 4; ++m) {
            if (m >= 2) am[m] = am[m] + s[1] * e.w[1][m];  // the other components are zero
            am[m] = am[m] + s[2] * e.w[2][m];
        }
        {
            const R pr = gamma1 * (e.r[3] - R(0.5) * (e.r[1] * e.r[1] + e.r[2] * e.r[2]) / e.r[0]);
            const R s3 = e.r[1] / e.r[0] + sqrt(gamma * pr / e.r[0]);
            const R rho2 = e.r[0] - e.w[3][0];
            const R rhou2 = e.r[1] - e.w[3][1];
            const R rhov2 = e.r[2] - e.w[3][2];
            const R en2 = e.r[3] - e.w[3][3];
            const R p2 = gamma1 * (en2 - R(0.5) * (rhou2 * rhou2 + rhov2 * rhov2) / rho2);
            const R c2 = sqrt(gamma * p2 / rho2);
            const R s2 = rhou2 / rho2 + c2;
            if (s2 < R(0.0) && s3 > R(0.0)) sfract = s2 * (s3 - s[3]) / (s3 - s2);
            else if (s[3] < R(0.0)) sfract = s[3];
            else return f;
            for (int m = 0; m < 4; ++m) am[m] = am[m] + sfract * e.w[3][m];
        }
        return f;
    }
    __device__ __forceinline__ void rpt2(int ixy, const R* asdq, const Roe& rr, R, R,
                                         R* bm, R* bp) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        const R u = rr.u, v = rr.v, a = rr.a, enth = rr.enth;
        const R u2v2 = u * u + v * v, euv = enth - u2v2;  // as rpn2 has them
        const R a3 = rr.g1a2 * (euv * asdq[0] + u * asdq[mu] + v * asdq[mv] - asdq[3]);
        const R a2 = asdq[mu] - u * asdq[0];
        const R x4 = asdq[mv] + (a - v) * asdq[0] - a * a3;
        bool ok = sizeof(R) == 4 || rr.y != R(0.0);
        R a4 = Dv<R>(R(2.0) * a, rr.y)(x4, ok);
        if (!ok) {
            seldom();
            a4 = x4 / (R(2.0) * a);
        }
        const R a1 = asdq[0] - a3 - a4;
        R waveb[4][3], sb[3];
        waveb[0][0] = a1; waveb[mu][0] = a1 * u; waveb[mv][0] = a1 * (v - a); waveb[3][0] = a1 * (enth - v * a);
        sb[0] = v - a;
        waveb[0][1] = a3; waveb[mu][1] = a3 * u + a2; waveb[mv][1] = a3 * v;
        waveb[3][1] = a3 * R(0.5) * u2v2 + a2 * u; sb[1] = v;
        waveb[0][2] = a4; waveb[mu][2] = a4 * u; waveb[mv][2] = a4 * (v + a); waveb[3][2] = a4 * (enth + v * a);
        sb[2] = v + a;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            R m1 = dmin(sb[0], R(0.0)) * waveb[m][0], p1 = dmax(sb[0], R(0.0)) * waveb[m][0];
#pragma unroll
            for (int mw = 1; mw < 3; ++mw) {
                m1 = m1 + dmin(sb[mw], R(0.0)) * waveb[m][mw];
                p1 = p1 + dmax(sb[mw], R(0.0)) * waveb[m][mw];
            }
            bm[m] = m1;
            bp[m] = p1;
        }
    }
};

using SweRoeSolver = SweRoeT<double>;
using Euler4RoeSolver = Euler4RoeT<double>;


// ---------------------------------------------------------------------------
// GeoClaw f-wave solver: applications/clawpack/shallow/2d/rp/rpn2_geoclaw.f90
// with geoclaw_riemann_utils.f (riemanntype, riemann_aug_JCP, maxiter = 1).
// The reference stops on a negative depth or a sonic state; here such an
// interface sets `bad`, which the kernel reports as a NaN CFL.  The
// reference's rpt2_geoclaw stops on entry, so no transverse solver exists.
//
// R = double is the reference's arithmetic.  R = float is the mixed form: the
// speed estimates, the 3x3 f-wave solve and the waves in FP32, while the
// hydrostatic part stays FP64 -- the states, dry-state and wall handling, the
// bathymetry jump and the jumps del = (delh - deldelh, delhu, delphi -
// deldelphi) the waves are solved for -- so that a lake at rest gives del = 0
// and no waves.  Every R expression keeps the FP64 form's association, so
// R = double compiles to the same arithmetic.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double fsignd(double a, double b) { return signbit(b) ? -fabs(a) : fabs(a); }

template <typename R>
__device__ __forceinline__ void geo_riemanntype(R hL, R hR, R uL, R uR, R& hm, R& s1m, R& s2m, R drytol, R g) {
    const R h_min = fmin(hR, hL), h_max = fmax(hR, hL);
    const R delu = uR - uL;
    if (h_min <= drytol) {
        hm = R(0.0);
        s1m = uR + uL - R(2.0) * sqrt(g * hR) + R(2.0) * sqrt(g * hL);
        s2m = s1m;
    } else {
        const R F_min = delu + R(2.0) * (sqrt(g * h_min) - sqrt(g * h_max));
        const R F_max = delu + (h_max - h_min) * (sqrt(R(.5) * g * (h_max + h_min) / (h_max * h_min)));
        if (F_min > R(0.0)) {
            const R t = dmax(R(0.0), -delu + R(2.0) * (sqrt(g * hL) + sqrt(g * hR)));
            hm = (R(1.0) / (R(16.0) * g)) * (t * t);
            s1m = uL + R(2.0) * sqrt(g * hL) - R(3.0) * sqrt(g * hm);
            s2m = uR - R(2.0) * sqrt(g * hR) + R(3.0) * sqrt(g * hm);
        } else if (F_max <= R(0.0)) {
            R h0 = h_max;
            {
                const R gL = sqrt(R(.5) * g * (R(1) / h0 + R(1) / hL));
                const R gR = sqrt(R(.5) * g * (R(1) / h0 + R(1) / hR));
                const R F0 = delu + (h0 - hL) * gL + (h0 - hR) * gR;
                const R dfdh = gL - g * (h0 - hL) / (R(4.0) * (h0 * h0) * gL) + gR -
                               g * (h0 - hR) / (R(4.0) * (h0 * h0) * gR);
                const R slope = R(2.0) * sqrt(h0) * dfdh;
                const R t = sqrt(h0) - F0 / slope;
                h0 = t * t;
            }
            hm = h0;
            const R u1m = uL - (hm - hL) * sqrt((R(.5) * g) * (R(1) / hm + R(1) / hL));
            const R u2m = uR + (hm - hR) * sqrt((R(.5) * g) * (R(1) / hm + R(1) / hR));
            s1m = u1m - sqrt(g * hm);
            s2m = u2m + sqrt(g * hm);
        } else {
            R h0 = h_min;
            {
                const R F0 = delu + R(2.0) * (sqrt(g * h0) - sqrt(g * h_max)) +
                             (h0 - h_min) * sqrt(R(.5) * g * (R(1) / h0 + R(1) / h_min));
                const R slope = (F_max - F0) / (h_max - h_min);
                h0 = h0 - F0 / slope;
            }
            hm = h0;
            if (hL > hR) {
                s1m = uL + R(2.0) * sqrt(g * hL) - R(3.0) * sqrt(g * hm);
                s2m = uL + R(2.0) * sqrt(g * hL) - sqrt(g * hm);
            } else {
                s2m = uR - R(2.0) * sqrt(g * hR) + R(3.0) * sqrt(g * hm);
                s1m = uR - R(2.0) * sqrt(g * hR) + sqrt(g * hm);
            }
        }
    }
}

// riemann_aug_JCP with maxiter = 1 and rarecorrectortest = .false.; returns false on a sonic state
template <typename R>
__device__ __forceinline__ bool geo_riemann_aug(double hL, double hR, double huL, double huR, double bL, double bR,
                                                double uL, double uR, double vL, double vR, double phiL, double phiR,
                                                R sE1, R sE2, double drytol, double g, R sw[3], R fw[3][3]) {
    const double rho = -9999999.0, pL = 0.0, pR = 0.0;
    const double delh = hR - hL, delhu = huR - huL, delphi = phiR - phiL, delb = bR - bL, delP = pR - pL;
    R hm, s1m, s2m;
    geo_riemanntype<R>(R(hL), R(hR), R(uL), R(uR), hm, s1m, s2m, R(drytol), R(g));
    R lambda[3];
    lambda[0] = dmin(sE1, s2m);
    lambda[2] = dmax(sE2, s1m);
    sE1 = lambda[0];
    sE2 = lambda[2];
    const R hstarHLL = dmax((R(huL) - R(huR) + sE2 * R(hR) - sE1 * R(hL)) / (sE2 - sE1), R(0.0));
    R r[3][3];
#pragma unroll
    for (int mw = 0; mw < 3; ++mw) {
        r[0][mw] = R(1.0);
        r[1][mw] = (mw == 1) ? R(0.0) : lambda[mw];
        r[2][mw] = (mw == 1) ? R(0.0) : lambda[mw] * lambda[mw];
    }
    lambda[1] = R(0.5) * (lambda[0] + lambda[2]);
    r[0][1] = R(0.0);
    r[1][1] = R(0.0);
    r[2][1] = R(1.0);
    const double criticaltol = dmax(drytol * g, 1e-6);
    const double criticaltol_2 = sqrt(criticaltol);
    const double hbar = dmax(0.5 * (hL + hR), 0.0);
    const double s1s2bar = 0.25 * ((uL + uR) * (uL + uR)) - g * hbar;
    const double s1s2tilde = dmax(0.0, uL * uR) - g * hbar;
    const double dE1 = sE1, dE2 = sE2, ds1m = s1m, ds2m = s2m;
    bool sonic = false;
    if (fabs(s1s2bar) <= criticaltol) sonic = true;
    else if (s1s2bar * s1s2tilde <= criticaltol * criticaltol) sonic = true;
    else if (s1s2bar * dE1 * dE2 <= criticaltol * criticaltol) sonic = true;
    else if (dmin(fabs(dE1), fabs(dE2)) < criticaltol_2) sonic = true;
    else if (dE1 < criticaltol_2 && ds1m > -criticaltol_2) sonic = true;
    else if (dE2 > -criticaltol_2 && ds2m < criticaltol_2) sonic = true;
    else if ((uL + sqrt(g * hL)) * (uR + sqrt(g * hR)) < 0.0) sonic = true;
    else if ((uL - sqrt(g * hL)) * (uR - sqrt(g * hR)) < 0.0) sonic = true;
    double deldelh = delb * g * hbar / s1s2bar;
    if (dE1 < -criticaltol && dE2 > criticaltol) {
        deldelh = dmin(deldelh, (double)(hstarHLL * (sE2 - sE1) / sE2));
        deldelh = dmax(deldelh, (double)(hstarHLL * (sE2 - sE1) / sE1));
    } else if (dE1 >= criticaltol) {
        deldelh = dmin(deldelh, (double)(hstarHLL * (sE2 - sE1) / sE1));
        deldelh = dmax(deldelh, -hL);
    } else if (dE2 <= -criticaltol) {
        deldelh = dmin(deldelh, hR);
        deldelh = dmax(deldelh, (double)(hstarHLL * (sE2 - sE1) / sE2));
    }
    deldelh = deldelh - delP / (rho * g);
    double deldelphi = -(delb * g * hbar * s1s2tilde / s1s2bar);
    deldelphi = dmin(deldelphi, g * dmax(-hL * delb, -hR * delb));
    deldelphi = dmax(deldelphi, g * dmin(-hL * delb, -hR * delb));
    deldelphi = deldelphi - hbar * delP / rho;
    const R del[3] = {R(delh - deldelh), R(delhu), R(delphi - deldelphi)};
    R det1 = r[0][0] * (r[1][1] * r[2][2] - r[1][2] * r[2][1]);
    R det2 = r[0][1] * (r[1][0] * r[2][2] - r[1][2] * r[2][0]);
    R det3 = r[0][2] * (r[1][0] * r[2][1] - r[1][1] * r[2][0]);
    const R determinant = det1 - det2 + det3;
    R beta[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        R A[3][3];
#pragma unroll
        for (int mw = 0; mw < 3; ++mw)
#pragma unroll
            for (int m = 0; m < 3; ++m) A[m][mw] = (mw == k) ? del[m] : r[m][mw];
        det1 = A[0][0] * (A[1][1] * A[2][2] - A[1][2] * A[2][1]);
        det2 = A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0]);
        det3 = A[0][2] * (A[1][0] * A[2][1] - A[1][1] * A[2][0]);
        beta[k] = (det1 - det2 + det3) / determinant;
    }
#pragma unroll
    for (int mw = 0; mw < 3; ++mw) {
        sw[mw] = lambda[mw];
        fw[0][mw] = beta[mw] * r[1][mw];
        fw[1][mw] = beta[mw] * r[2][mw];
        fw[2][mw] = beta[mw] * r[1][mw];
    }
    fw[2][0] = fw[2][0] * R(vL);
    fw[2][2] = fw[2][2] * R(vR);
    fw[2][1] = R(0.0);
    const double hustar_interface = huL + (double)fw[0][0];
    const R dvflux = R(hR * uR * vR - hL * uL * vL);
    if (hustar_interface <= 0.0) fw[2][0] = fw[2][0] + (dvflux - fw[2][0] - fw[2][2]);
    else fw[2][2] = fw[2][2] + (dvflux - fw[2][0] - fw[2][2]);
    return !sonic;
}

template <typename R, bool V5_ = false>
struct GeoclawFwaveT {
    using Real = R;
    static constexpr bool V5 = V5_;
    static constexpr bool FWAVE = true;
    static constexpr int M = 3;
    static constexpr int W = 3;
    struct Roe { R s[3]; };  // the wave speeds: no Roe averages, there is no transverse solver
    struct Cell {};
    static constexpr int NC = 0;
    // wave components that are not zero by construction: the middle wave moves
    // momentum in the normal direction alone
    static constexpr int NWV = 7;
    __host__ __device__ static constexpr bool nz(int mw, int rel) { return mw != 1 || rel == 1; }
    __device__ __forceinline__ void speeds(const Roe& rr, R* s) const {
        s[0] = rr.s[0];
        s[1] = rr.s[1];
        s[2] = rr.s[2];
    }
    R grav, gamma, gamma1, drytol;
    // The common interface (both sides wet, subcritical) without a branch per
    // division (fcb_arith.cuh): the eigenvectors' zeros and ones multiplied out, the
    // sign tests that bound deldelh made on products with a margin of 0.1 %.  Every
    // other interface, and operands near underflow, take rpn2b_plain.
    __device__ __forceinline__ void rpn2b(int ixy, const double* qL, const double* qR, double bL, double bR,
                                          R (*wave)[M], R* s, R* amdq, R* apdq, bool& bad) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        const double g = gdbl, dtol = drytol_d;
        const double hL = qL[0], hR = qR[0], huL = qL[mu], huR = qR[mu];
        bool ok = hL > dtol && hR > dtol;
        const Dv<double> dL(hL, ok), dR(hR, ok);
        const double uL = dL(huL, ok), vL = dL(qL[mv], ok), phiL = 0.5 * g * (hL * hL) + dL(huL * huL, ok);
        const double uR = dR(huR, ok), vR = dR(qR[mv], ok), phiR = 0.5 * g * (hR * hR) + dR(huR * huR, ok);
        const double cL = sqrt_ok(g * hL, ok), cR = sqrt_ok(g * hR, ok);
        const R rg = R(g), ruL = R(uL), ruR = R(uR), rhL = R(hL), rhR = R(hR);
        R rcL, rcR;
        if constexpr (sizeof(R) == 8) { rcL = cL; rcR = cR; }
        else { rcL = sqrt(rg * rhL); rcR = sqrt(rg * rhR); }
        const R uhat = Dv<R>(rcR + rcL, ok)(rcL * ruL + rcR * ruR, ok);
        const R chat = sqrt_ok(rg * R(0.5) * (rhR + rhL), ok);
        R sE1 = dmin(ruL - rcL, uhat - chat), sE2 = dmax(ruR + rcR, uhat + chat);
        // riemanntype, both sides wet: the speeds of the middle state's outer waves
        R s1m, s2m;
        {
            const R delu = ruR - ruL;
            const bool leftmin = rhL < rhR;
            const R hmin = leftmin ? rhL : rhR, hmax = leftmin ? rhR : rhL;
            const R cmin = leftmin ? rcL : rcR, cmax = leftmin ? rcR : rcL;
            const R fmin_ = delu + R(2.0) * (cmin - cmax);
            const R fmax_ = delu + (hmax - hmin) * sqrt_ok(Dv<R>(hmax * hmin, ok)(R(.5) * rg * (hmax + hmin), ok), ok);
            if (fmin_ <= R(0.0) && fmax_ <= R(0.0)) {  // two shocks
                const Dv<R> d0(hmax, ok), l(rhL, ok), r(rhR, ok);
                const R i0 = d0(R(1), ok), iL = l(R(1), ok), iR = r(R(1), ok);
                const R gL = sqrt_ok(R(.5) * rg * (i0 + iL), ok), gR = sqrt_ok(R(.5) * rg * (i0 + iR), ok);
                const R F0 = delu + (hmax - rhL) * gL + (hmax - rhR) * gR;
                const R hh = R(4.0) * (hmax * hmax);
                const R dfdh = gL - Dv<R>(hh * gL, ok)(rg * (hmax - rhL), ok) + gR -
                               Dv<R>(hh * gR, ok)(rg * (hmax - rhR), ok);
                const R sq0 = sqrt_ok(hmax, ok);
                const R slope = R(2.0) * sq0 * dfdh;
                const R t = sq0 - Dv<R>(slope, ok)(F0, ok);
                const R hm = t * t;
                const R im = Dv<R>(hm, ok)(R(1), ok), cm = sqrt_ok(rg * hm, ok);
                s1m = ruL - (hm - rhL) * sqrt_ok((R(.5) * rg) * (im + iL), ok) - cm;
                s2m = ruR + (hm - rhR) * sqrt_ok((R(.5) * rg) * (im + iR), ok) + cm;
            } else {
                const bool rare = fmin_ > R(0.0);  // two rarefactions, else a shock and a rarefaction
                // (a shock and a rarefaction: F0 at h_min is fmin_, a zero added)
                const R slope = Dv<R>(rare ? R(1) : hmax - hmin, ok)(rare ? R(1) : fmax_ - fmin_, ok);
                const R step = Dv<R>(slope, ok)(rare ? R(0) : -fmin_, ok);  // fmin_ <= 0 here
                const R t = dmax(R(0.0), -delu + R(2.0) * (rcL + rcR));
                const R i16 = Dv<R>(R(16.0) * rg, ok)(R(1), ok);
                const R hm = rare ? i16 * (t * t) : hmin + step;
                const R cm = sqrt_ok(rg * hm, ok);
                const R ul = ruL + R(2.0) * rcL, ur = ruR - R(2.0) * rcR;
                const bool left = rhL > rhR;
                s1m = rare || left ? ul - R(3.0) * cm : ur + cm;
                s2m = rare || !left ? ur + R(3.0) * cm : ul - cm;
            }
        }
        const R l0 = dmin(sE1, s2m), l2 = dmax(sE2, s1m), l1 = R(0.5) * (l0 + l2);
        const Dv<R> dl(l2 - l0, ok);  // sE2 - sE1, and minus the determinant
        const R hstarHLL = dmax(dl(R(huL) - R(huR) + l2 * rhR - l0 * rhL, ok), R(0.0));
        const double ctol = dmax(dtol * g, 1e-6);
        const double hbar = dmax(0.5 * (hL + hR), 0.0);
        const double s1s2bar = 0.25 * ((uL + uR) * (uL + uR)) - g * hbar;
        const double s1s2tilde = dmax(0.0, uL * uR) - g * hbar;
        const double dE1 = l0, dE2 = l2;
        bool sonic = false;
        if (fabs(s1s2bar) <= ctol) sonic = true;
        if (s1s2bar * s1s2tilde <= ctol * ctol) sonic = true;
        if (s1s2bar * dE1 * dE2 <= ctol * ctol) sonic = true;
        if (dmin(fabs(dE1), fabs(dE2)) < ctol2) sonic = true;
        if (dE1 < ctol2 && (double)s1m > -ctol2) sonic = true;
        if (dE2 > -ctol2 && (double)s2m < ctol2) sonic = true;
        if ((uL + cL) * (uR + cR) < 0.0) sonic = true;
        if ((uL - cL) * (uR - cR) < 0.0) sonic = true;
        const double delb = bR - bL, w = delb * g * hbar;
        const Dv<double> dbar(-s1s2bar, ok);  // subcritical: negative
        const double deldelh = -dbar(w, ok);
        // deldelh stays inside [HLL / sE1, HLL / sE2]
        const double hll = (double)(hstarHLL * (l2 - l0));
        ok = ok && dE1 < -ctol && dE2 > ctol && hll > 0.0 && deldelh * dE2 < 0.999 * hll && deldelh * dE1 < 0.999 * hll;
        double deldelphi = dbar(w * s1s2tilde, ok);
        deldelphi = dmin(deldelphi, g * dmax(-hL * delb, -hR * delb));
        deldelphi = dmax(deldelphi, g * dmin(-hL * delb, -hR * delb));
        const R d0 = R((hR - hL) - deldelh), d1 = R(huR - huL), d2 = R((phiR - phiL) - deldelphi);
        const R q0 = l0 * l0, q2 = l2 * l2;
        const R b0 = -dl(d0 * -l2 + d1, ok), b2 = -dl(-d1 + d0 * l0, ok);
        const R b1 = -dl((d1 * q2 - l2 * d2) - d0 * (l0 * q2 - l2 * q0) + (l0 * d2 - d1 * q0), ok);
        R f0 = b0 * l0 * R(vL), f2 = b2 * l2 * R(vR);
        const R dvflux = R(hR * uR * vR - hL * uL * vL), rest = dvflux - f0 - f2;
        if (huL + (double)(b0 * l0) <= 0.0) f0 = f0 + rest;
        else f2 = f2 + rest;
        s[0] = l0; s[1] = l1; s[2] = l2;
        wave[0][0] = b0 * l0; wave[0][mu] = b0 * q0; wave[0][mv] = f0;
        wave[1][0] = R(0.0); wave[1][mu] = b1; wave[1][mv] = R(0.0);
        wave[2][0] = b2 * l2; wave[2][mu] = b2 * q2; wave[2][mv] = f2;
        if (!ok) {
            seldom();
            rpn2b_plain(ixy, qL, qR, bL, bR, wave, s, bad);
        } else if (sonic) {
            bad = true;
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            R am = R(0.0), ap = R(0.0);
#pragma unroll
            for (int mw = 0; mw < 3; ++mw) {
                if (mw == 1 && m != mu) continue;  // zero
                const R half = R(0.5) * wave[mw][m];
                am = am + (s[mw] < R(0.0) ? wave[mw][m] : s[mw] > R(0.0) ? R(0.0) : half);
                ap = ap + (s[mw] > R(0.0) ? wave[mw][m] : s[mw] < R(0.0) ? R(0.0) : half);
            }
            amdq[m] = am;
            apdq[m] = ap;
        }
    }
    // one interface of rpn2_geoclaw.f90; the states and bL, bR (aux(1) of the
    // two cells) in FP64
    __device__ __forceinline__ void rpn2b_plain(int ixy, const double* qL, const double* qR, double bL, double bR,
                                                R (*wave)[M], R* s, bool& bad) const {
        const int mu = (ixy == 1) ? 1 : 2;
        const int mv = (ixy == 1) ? 2 : 1;
        // the FP64 hydrostatic part reads gravity and the dry tolerance in FP64
        const double g = gdbl, dtol = drytol_d;
#pragma unroll
        for (int mw = 0; mw < 3; ++mw) {
            s[mw] = R(0.0);
            wave[mw][0] = R(0.0); wave[mw][1] = R(0.0); wave[mw][2] = R(0.0);
        }
        if (qL[0] < 0.0 || qR[0] < 0.0) bad = true;
        if (!(qL[0] <= dtol && qR[0] <= dtol)) {
            double hL = qL[0], hR = qR[0], huL = qL[mu], huR = qR[mu], hvL = qL[mv], hvR = qR[mv];
            double uR, vR, phiR, uL, vL, phiL;
            if (hR > dtol) {
                uR = huR / hR; vR = hvR / hR;
                phiR = 0.5 * g * (hR * hR) + (huR * huR) / hR;
            } else {
                hR = 0.0; huR = 0.0; hvR = 0.0; uR = 0.0; vR = 0; phiR = 0.0;
            }
            if (hL > dtol) {
                uL = huL / hL; vL = hvL / hL;
                phiL = 0.5 * g * (hL * hL) + (huL * huL) / hL;
            } else {
                hL = 0.0; huL = 0.0; hvL = 0.0; uL = 0.0; vL = 0.0; phiL = 0.0;
            }
            R wall[3] = {R(1.0), R(1.0), R(1.0)};
            double hstar, s1m, s2m;
            if (hR <= dtol) {
                geo_riemanntype<double>(hL, hL, uL, -uL, hstar, s1m, s2m, dtol, g);
                const double hstartest = dmax(hL, hstar);
                if (hstartest + bL < bR) {
                    wall[1] = R(0.0); wall[2] = R(0.0);
                    hR = hL; huR = -huL; bR = bL; phiR = phiL; uR = -uL; vL = vR;
                } else if (hL + bL < bR) {
                    bR = hL + bL;
                }
            } else if (hL <= dtol) {
                geo_riemanntype<double>(hR, hR, -uR, uR, hstar, s1m, s2m, dtol, g);
                const double hstartest = dmax(hR, hstar);
                if (hstartest + bR < bL) {
                    wall[0] = R(0.0); wall[1] = R(0.0);
                    hL = hR; huL = -huR; bL = bR; phiL = phiR; uL = -uR; vR = vL;
                } else if (hR + bR < bL) {
                    bL = hR + bR;
                }
            }
            const R rg = R(g);
            const R sL = R(uL) - sqrt(rg * R(hL));
            const R sR = R(uR) + sqrt(rg * R(hR));
            const R uhat = (sqrt(rg * R(hL)) * R(uL) + sqrt(rg * R(hR)) * R(uR)) / (sqrt(rg * R(hR)) + sqrt(rg * R(hL)));
            const R chat = sqrt(rg * R(0.5) * (R(hR) + R(hL)));
            const R sE1 = dmin(sL, uhat - chat), sE2 = dmax(sR, uhat + chat);
            R sw[3], fw[3][3];
            if (!geo_riemann_aug<R>(hL, hR, huL, huR, bL, bR, uL, uR, vL, vR, phiL, phiR, sE1, sE2, dtol, g, sw, fw))
                bad = true;
#pragma unroll
            for (int mw = 0; mw < 3; ++mw) {
                s[mw] = sw[mw] * wall[mw];
                wave[mw][0] = fw[0][mw] * wall[mw];
                wave[mw][mu] = fw[1][mw] * wall[mw];
                wave[mw][mv] = fw[2][mw] * wall[mw];
            }
        }
    }
    double gdbl, drytol_d;  // gravity and dry tolerance in FP64, set by the step kernel
    double ctol2;           // the root of the critical tolerance, likewise
    // never called: order (2, 0) is enforced for this solver
    __device__ __forceinline__ void rpt2(int, const R* asdq, const Roe&, R, R, R* bm, R* bp) const {
#pragma unroll
        for (int m = 0; m < M; ++m) bm[m] = bp[m] = R(0) * asdq[m];
    }
    __device__ __forceinline__ void rpn2(int, const R*, const R*, R, R (*)[M], R*, R*, R*, Roe&) const {}
};

// clawpack46_inlinelimiter.f:4-118: phi(r) for limiter code `mth`
// (clawpack5_inlinelimiter.f:4-109 knows codes 1-5; callers map the others to 1).
template <typename R>
__device__ __forceinline__ R limiter_phi(int mth, R r) {
    switch (mth) {
        case 2: return dmax(dmax(R(0.0), dmin(R(1.0), R(2.0) * r)), dmin(R(2.0), r));
        case 3: return (r + fabs(r)) / (R(1.0) + fabs(r));
        case 4: {
            const R c = (R(1.0) + r) / R(2.0);
            return dmax(R(0.0), dmin(dmin(c, R(2.0)), R(2.0) * r));
        }
        case 5: return r;
        case 6: {
            const R th = R((double)1.3f);  // REAL*4 literal in the reference
            return dmax(R(0.0), dmin(dmin(th * r, (1 + r) / R(2.0)), th));
        }
        default: return dmax(R(0.0), dmin(R(1.0), r));
    }
}

// num / wn2, wn2 > 0.  The tails of a front leave waves of 1e-136 and less over whole
// strips of a mesh, whose squares and products are near underflow: both operands
// times 2^400 (exact) stay in the range of the method.
__device__ __forceinline__ double limiter_ratio(double num, double wn2, bool& ok) {
    const double r = Dv<double>(wn2 * 0x1p400, ok, 1400u).quotient(num * 0x1p400);
    // zero, or |r| >= 2^-1000 (not rounded to a denormal) and finite (an infinite num, or
    // one that overflows with the factor, gives a NaN here)
    const unsigned h = (unsigned)__double2hiint(r);
    ok = ok & ((h + h - (46u << 20) < (4048u << 20)) | (r == 0.0));
    return r;
}
__device__ __forceinline__ float limiter_ratio(float num, float wn2, bool&) { return num / wn2; }

// Limiter values of the W waves of an interface: phi(num / wn2) for limiter code
// lim(mw), 1 where the wave vanishes or is not limited.  The quotients are formed
// together (fcb_arith.cuh), and again with the operator when one of them leaves the
// range of that method.  Where the state is constant, whole warps have no wave and
// skip all of it.
template <bool V5, int W, typename R, class LIM>
__device__ __forceinline__ void limiter_values(const R* num, const R* wn2, const LIM& lim, R* phi) {
    bool any = false;
#pragma unroll
    for (int mw = 0; mw < W; ++mw) {
        phi[mw] = R(1);
        any = any | (wn2[mw] != R(0));
    }
    if (any) {
        bool ok = true;
        R r[W];
#pragma unroll
        for (int mw = 0; mw < W; ++mw) {
            r[mw] = limiter_ratio(num[mw], wn2[mw] == R(0) ? R(1) : wn2[mw], ok);
        }
        if (!ok) {
            seldom();
#pragma unroll
            for (int mw = 0; mw < W; ++mw) r[mw] = num[mw] / wn2[mw];
        }
#pragma unroll
        for (int mw = 0; mw < W; ++mw) {
            const int mth = lim(mw);
            R p;
            if (mth == 3) {  // van Leer: the quotient without branches
                bool ok3 = true;
                const Dv<R> d(R(1.0) + fabs(r[mw]), ok3);
                p = d(r[mw] + fabs(r[mw]), ok3);
                if (!ok3) {
                    seldom();
                    p = limiter_phi(3, r[mw]);
                }
            } else {
                p = limiter_phi((V5 && mth > 5) ? 1 : mth, r[mw]);
            }
            phi[mw] = (mth == 0 || wn2[mw] == R(0)) ? R(1) : p;
        }
    }
}

}  // namespace fcb
