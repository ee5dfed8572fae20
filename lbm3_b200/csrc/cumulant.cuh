// Well-conditioned D3Q27 cumulant collision (Geier et al. 2017), in registers.
//
// Follows the reference's applyCollision (include/applyCollision.h:17-491):
// shifted populations f_i - w_i are transformed to central moments with the
// weight-moment constants K (chimera transform z, then y, then x), converted
// to cumulants, relaxed (K17 with limiter, or AllOne when the limiter is
// <= 0), and transformed back (x, then y, then z).  Sums in the forward
// transform and the cumulant algebra keep the reference's grouping; the back
// transform is refactored into fused multiply-adds with per-cell constants
// (algebraically the reference's Eqs. 57-65, rounded differently).  Every
// quantity that depends only on the viscosity (omega1, omega3..5, A, B) is
// computed once per grid on the host (CollisionConsts) instead of per cell.
//
// The 16-bit kernels, and the FP32 ones whose domain fits the L2 cache, are
// bound by the number of these operations, so: the limiter is one product and
// one reciprocal (in place of a quotient, a blend and a complement), products
// that are added to something are fused explicitly (the packed intrinsics are
// not contracted), the fourth order is written in the strain rates it reduces
// to, and 1 / rho of a cell pair takes a Newton step on the hardware estimate
// instead of two scalar correctly rounded reciprocals.  Step of eight 64^3
// periodic boxes in FP16 88 -> 79 us, of a 160^3 one 167 -> 149, of a 64^3 one in
// FP32 12.3 -> 11.2, of a 128^3 one 84.5 -> 79.7.  Against the FP64 evaluation
// the populations, mass and momentum err as before (2.3e-7 relative at
// |u| = 0.03, 1.95e-9 and 3.28e-9 rms).
//
// The arithmetic is a template over the value type: `float` collides one
// cell, `Pair` collides two cells at once with the packed FP32x2 instructions
// of sm_100 (add/mul/fma .rn.f32x2), which issue once for both cells (both
// lanes follow exactly the scalar sequence of operations), and `double` is
// the FP64 build that serves as the reference of the storage-precision study.
#pragma once

#include "lattice.h"

#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif

namespace lbm {

template <class T> struct CollisionConstsT {
    T omega1;      // 1 / (3 nu nuMultiplier + 1/2)
    T omega3, omega4, omega5, A, B;  // K17 parameters (:241-262)
    T tauTerm;     // 1/omega1 - 1/2
    T lambda;      // collision limiter, at most 1e30 (K17 when > 0 and nuMultiplier <= 1)
    int useK17;
    // products of the above that every cell needs
    T mHalfW1;     // -omega1 * 0.5
    T w1x15;       // 1.5 * omega1
    T mW1x3;       // -3 * omega1
    T oneMinusW1;  // 1 - omega1
    T halfW1c;     // 1 - 0.5 * omega1
    T oneMinusW3, oneMinusW4, oneMinusW5;
    T c43;         // (2/3) * tauTerm * A
    T cB;          // -(1/3) * tauTerm * B
};
using CollisionConsts = CollisionConstsT<float>;

// Host-side evaluation of the per-grid constants, with the reference's
// expressions (include/applyCollision.h:193-262), in the arithmetic type T.
template <class T> inline CollisionConstsT<T> makeCollisionConstsT(T nu, T nuMultiplier, T limiter) {
    CollisionConstsT<T> k{};
    const T omega1 = T(1) / (T(3) * (nu * nuMultiplier) + T(0.5));
    const T omega2 = T(1);
    k.omega1 = omega1;
    k.omega3 = T(8) * (omega1 - T(2)) * (omega2 * (T(3) * omega1 - T(1)) - T(5) * omega1) /
               (T(8) * (T(5) - T(2) * omega1) * omega1 + omega2 * (T(8) + omega1 * (T(9) * omega1 - T(26))));
    k.omega4 = T(8) * (omega1 - T(2)) * (omega1 + omega2 * (T(3) * omega1 - T(7))) /
               (omega2 * (T(56) - T(42) * omega1 + T(9) * omega1 * omega1) - T(8) * omega1);
    k.omega5 = T(24) * (omega1 - T(2)) *
               (T(4) * omega1 * omega1 + omega1 * omega2 * (T(18) - T(13) * omega1) +
                omega2 * omega2 * (T(2) + omega1 * (T(6) * omega1 - T(11)))) /
               (T(16) * omega1 * omega1 * (omega1 - T(6)) -
                T(2) * omega1 * omega2 * (T(216) + T(5) * omega1 * (T(9) * omega1 - T(46))) +
                omega2 * omega2 * (omega1 * (T(3) * omega1 - T(10)) * (T(15) * omega1 - T(28)) - T(48)));
    k.A = (T(4) * omega1 * omega1 + T(2) * omega1 * omega2 * (omega1 - T(6)) +
           omega2 * omega2 * (omega1 * (T(10) - T(3) * omega1) - T(4))) /
          ((omega1 - omega2) * (omega2 * (T(2) + T(3) * omega1) - T(8) * omega1));
    k.B = (T(4) * omega1 * omega2 * (T(9) * omega1 - T(16)) - T(4) * omega1 * omega1 -
           T(2) * omega2 * omega2 * (T(2) + T(9) * omega1 * (omega1 - T(2)))) /
          (T(3) * (omega1 - omega2) * (omega2 * (T(2) + T(3) * omega1) - T(8) * omega1));
    k.tauTerm = T(1) / omega1 - T(0.5);
    // an infinite limiter (none) makes (1 - omega) lambda v / (lambda + |v|) a
    // quotient of infinities, and the reciprocal of 2^126 or more flushes to
    // zero; 1e30 is above any |v| by more than FP64 resolves
    k.lambda = limiter < T(1e30) ? limiter : T(1e30);
    k.useK17 = (limiter > T(0)) && (nuMultiplier <= T(1));
    k.mHalfW1 = -omega1 * T(0.5);
    k.w1x15 = T(1.5) * omega1;
    k.mW1x3 = T(-3) * omega1;
    k.oneMinusW1 = T(1) - omega1;
    k.halfW1c = T(1) - T(0.5) * omega1;
    k.oneMinusW3 = T(1) - k.omega3;
    k.oneMinusW4 = T(1) - k.omega4;
    k.oneMinusW5 = T(1) - k.omega5;
    k.c43 = (T(2) / T(3)) * k.tauTerm * k.A;
    k.cB = -(T(1) / T(3)) * k.tauTerm * k.B;
    return k;
}
inline CollisionConsts makeCollisionConsts(float nu, float nuMultiplier, float limiter) {
    return makeCollisionConstsT<float>(nu, nuMultiplier, limiter);
}

// ---- value types -----------------------------------------------------------
// Scalar: plain float operators (the compiler fuses a*b+c on the device).
LBM_HD float fmaR(float a, float b, float c) { return a * b + c; }
LBM_HD float addAbs(float a, float b) { return a + fabsf(b); }
LBM_HD float bcast(float a, float) { return a; }
// a / b for the limiter weights: the hardware reciprocal on the device
// (two ulp), an exact division on the host; b is a normal number.
LBM_HD float divFast(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fdividef(a, b);
#else
    return a / b;
#endif
}
LBM_HD float posMin(float a) { return a < 1.17549435e-38f ? 1.17549435e-38f : a; }  // smallest normal
LBM_HD double posMin(double a) { return a; }
LBM_HD float rcpR(float a) {
#ifdef __CUDA_ARCH__
    return __frcp_rn(a);  // the correctly rounded 1 / a
#else
    return 1.f / a;
#endif
}
// Double: the FP64 build of the kernels (reference for storage precision).
LBM_HD double fmaR(double a, double b, double c) { return fma(a, b, c); }
LBM_HD double addAbs(double a, double b) { return a + fabs(b); }
LBM_HD double bcast(double a, double) { return a; }
LBM_HD double divFast(double a, double b) { return a / b; }
LBM_HD double rcpR(double a) { return 1.0 / a; }

// Scalar type of a value type (the type of its constants).
template <class R> struct ScalarOf { using type = R; };

#ifdef __CUDACC__
// Two cells in the two lanes of a packed FP32x2 register pair.
struct Pair {
    float2 v;
};
__device__ __forceinline__ Pair mkPair(float a, float b) { return {make_float2(a, b)}; }
__device__ __forceinline__ Pair bcast(float a, Pair) { return {make_float2(a, a)}; }
__device__ __forceinline__ Pair operator+(Pair a, Pair b) { return {__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ Pair operator*(Pair a, Pair b) { return {__fmul2_rn(a.v, b.v)}; }
// a - b as a + (-1) b: one packed FMA, exact like a subtraction
__device__ __forceinline__ Pair operator-(Pair a, Pair b) { return {__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)}; }
__device__ __forceinline__ Pair fmaR(Pair a, Pair b, Pair c) { return {__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ Pair operator+(Pair a, float b) { return a + Pair{make_float2(b, b)}; }
__device__ __forceinline__ Pair operator+(float a, Pair b) { return Pair{make_float2(a, a)} + b; }
__device__ __forceinline__ Pair operator-(Pair a, float b) { return a + Pair{make_float2(-b, -b)}; }
__device__ __forceinline__ Pair operator-(float a, Pair b) { return Pair{make_float2(a, a)} - b; }
__device__ __forceinline__ Pair operator*(Pair a, float b) { return a * Pair{make_float2(b, b)}; }
__device__ __forceinline__ Pair operator*(float a, Pair b) { return Pair{make_float2(a, a)} * b; }
__device__ __forceinline__ Pair fmaR(Pair a, float b, Pair c) { return fmaR(a, Pair{make_float2(b, b)}, c); }
__device__ __forceinline__ Pair fmaR(float a, Pair b, Pair c) { return fmaR(Pair{make_float2(a, a)}, b, c); }
__device__ __forceinline__ Pair fmaR(Pair a, Pair b, float c) { return fmaR(a, b, Pair{make_float2(c, c)}); }
__device__ __forceinline__ Pair addAbs(float a, Pair b) { return {make_float2(a + fabsf(b.v.x), a + fabsf(b.v.y))}; }
// the hardware reciprocal estimate (one ulp) of normal values
__device__ __forceinline__ float rcpEstimate(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ Pair rcpEstimate(Pair a) { return {make_float2(rcpEstimate(a.v.x), rcpEstimate(a.v.y))}; }
__device__ __forceinline__ Pair divFast(Pair a, Pair b) { return a * rcpEstimate(b); }
// 1 / a by one Newton-Raphson step r + r (1 - a r) on the estimate, both lanes at
// once (the error of the step is the estimate's squared plus one rounding)
__device__ __forceinline__ Pair rcpR(Pair a) {
    const Pair r = rcpEstimate(a);
    return fmaR(r, fmaR(a * -1.f, r, 1.f), r);
}
template <> struct ScalarOf<Pair> { using type = float; };

// One cell with the operations of one Pair lane, so that a cell collided alone
// comes out bit for bit as on a lane (the compiler contracts plain floats as
// each kernel suits it).
struct Single {
    float v;
};
__device__ __forceinline__ Single bcast(float a, Single) { return {a}; }
__device__ __forceinline__ Single operator+(Single a, Single b) { return {__fadd_rn(a.v, b.v)}; }
__device__ __forceinline__ Single operator*(Single a, Single b) { return {__fmul_rn(a.v, b.v)}; }
__device__ __forceinline__ Single operator-(Single a, Single b) { return {__fsub_rn(a.v, b.v)}; }
__device__ __forceinline__ Single fmaR(Single a, Single b, Single c) { return {__fmaf_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ Single operator+(Single a, float b) { return a + Single{b}; }
__device__ __forceinline__ Single operator+(float a, Single b) { return Single{a} + b; }
__device__ __forceinline__ Single operator-(Single a, float b) { return a - Single{b}; }
__device__ __forceinline__ Single operator-(float a, Single b) { return Single{a} - b; }
__device__ __forceinline__ Single operator*(Single a, float b) { return a * Single{b}; }
__device__ __forceinline__ Single operator*(float a, Single b) { return Single{a} * b; }
__device__ __forceinline__ Single fmaR(Single a, float b, Single c) { return fmaR(a, Single{b}, c); }
__device__ __forceinline__ Single fmaR(float a, Single b, Single c) { return fmaR(Single{a}, b, c); }
__device__ __forceinline__ Single fmaR(Single a, Single b, float c) { return fmaR(a, b, Single{c}); }
__device__ __forceinline__ Single addAbs(float a, Single b) { return {__fadd_rn(a, fabsf(b.v))}; }
__device__ __forceinline__ Single divFast(Single a, Single b) { return {__fmul_rn(a.v, rcpEstimate(b.v))}; }
__device__ __forceinline__ Single rcpR(Single a) {
    const float r = rcpEstimate(a.v);
    return {__fmaf_rn(r, __fmaf_rn(-a.v, r, 1.f), r)};
}
template <> struct ScalarOf<Single> { using type = float; };
#endif

namespace detail {

// exact fractions rounded once to the scalar type
template <class Sc> struct Frac {
    static constexpr Sc third = Sc(1) / Sc(3);
    static constexpr Sc ninth = Sc(1) / Sc(9);
    static constexpr Sc n27th = Sc(1) / Sc(27);
    static constexpr Sc twoThirds = Sc(2) / Sc(3);
};

// Weight moments of the shifted transform, as the literal fractions the
// reference uses (K_aa0 ... K_c02, include/applyCollision.h:24-38).
// Index 0 = -1, 1 = 0, 2 = +1 along an axis.
template <class Sc = float> LBM_HD constexpr Sc kZ(int a, int b) {  // z stage: sum of w over the (a,b) line
    return (a == 1 && b == 1) ? Sc(4) / Sc(9) : (a == 1 || b == 1) ? Sc(1) / Sc(9) : Sc(1) / Sc(36);
}
template <class Sc = float> LBM_HD constexpr Sc kY(int a, int n) {  // y stage: order-n z moment of the x=a plane
    return n == 1 ? Sc(0)
         : n == 0 ? (a == 1 ? Sc(2) / Sc(3) : Sc(1) / Sc(6))
                  : (a == 1 ? Sc(2) / Sc(9) : Sc(1) / Sc(18));
}
template <class Sc = float> LBM_HD constexpr Sc kX(int b, int n) {  // x stage: order (y, z) moment of the weights
    return (b == 1 || n == 1) ? Sc(0) : (b == 0 && n == 0) ? Sc(1) : (b == 2 && n == 2) ? Sc(1) / Sc(9) : Sc(1) / Sc(3);
}

// Per-cell constants of one axis for the backward transform, formed where its
// stage begins (three axes' worth held from the start would spill).
template <class R> struct Axis {
    R u2, m2u;           // u^2, -2u
    R omu2, hlo, hhi;    // 1 - u^2, (u^2 - u) / 2, (u^2 + u) / 2
    R um, up;            // u - 1/2, u + 1/2
};
template <class R> LBM_HD Axis<R> axisOf(R u) {
    Axis<R> c;
    c.u2 = u * u;
    c.m2u = u * -2.f;
    c.omu2 = 1.f - c.u2;
    const R hu2 = c.u2 * 0.5f;
    c.hlo = fmaR(u, -0.5f, hu2);
    c.hhi = fmaR(u, 0.5f, hu2);
    c.um = u - 0.5f;
    c.up = u + 0.5f;
    return c;
}

// Forward chimera step of one line (sum s and difference d of its plus and
// minus values) with the order-0 sum k0 and the weight moment K: orders 1 and 2
// about velocity u,
//   r1 = d - u (k0 + K),  r2 = s - 2u d + u^2 (k0 + K).
// mu = -u, m2u = -2u, u2 = u^2.
template <class R> struct Shift {
    R mu, m2u, u2;
};
template <class R> LBM_HD Shift<R> shiftOf(R u) { return {u * -1.f, u * -2.f, u * u}; }
template <class R, class Sc>
LBM_HD void fwd(R s, R d, R k0, Sc K, const Shift<R>& c, R& r1, R& r2) {
    const R kk = K != Sc(0) ? k0 + K : k0;
    r1 = fmaR(c.mu, kk, d);
    r2 = fmaR(c.u2, kk, fmaR(c.m2u, d, s));
}

// Backward chimera step of one line from orders (s0, s1, s2) to the values at
// velocities -1, 0, +1 (Eqs. 57-65 of the reference's applyCollision):
//   zero  = s0 (1 - u^2) - 2u s1 - s2 - K u^2,
//   minus = ((s0 + K)(u^2 - u) + s1 (2u - 1) + s2) / 2,
//   plus  = ((s0 + K)(u^2 + u) + s1 (2u + 1) + s2) / 2.
// mKu2 = -K u^2 of this line's K (a per-cell constant).  (Through the line's raw
// moments it is one operation less, but the density then drifts by other
// rounding errors than the reference's, by more than the field bar in 1,000
// steps.)
template <class R, class Sc>
LBM_HD void bwd(R s0, R s1, R s2, Sc K, R mKu2, const Axis<R>& c, R& lo, R& mid, R& hi) {
    const R h2 = s2 * 0.5f;
    const R sK = K != Sc(0) ? s0 + K : s0;
    lo = fmaR(sK, c.hlo, fmaR(s1, c.um, h2));
    hi = fmaR(sK, c.hhi, fmaR(s1, c.up, h2));
    const R t = K != Sc(0) ? fmaR(s2, -1.f, mKu2) : s2 * -1.f;
    mid = fmaR(s0, c.omu2, fmaR(c.m2u, s1, t));
}

}  // namespace detail

// f: shifted populations, in place.  gx,gy,gz: body force (half applied
// before and half after collision, :70-72 and the sign flip of first-order
// moments before the back transform).  lambda: limiter for this cell (the
// same for both lanes of a Pair).
template <class R>
LBM_HD void collideCumulantT(R (&f)[27], const CollisionConstsT<typename ScalarOf<R>::type>& P,
                             typename ScalarOf<R>::type lambda, typename ScalarOf<R>::type gx,
                             typename ScalarOf<R>::type gy, typename ScalarOf<R>::type gz) {
    using namespace detail;
    using Sc = typename ScalarOf<R>::type;
    constexpr Sc kThird = Frac<Sc>::third, kNinth = Frac<Sc>::ninth, k27th = Frac<Sc>::n27th;
    // m[x][y][z]: after the z stage z holds the moment order, etc.
    R m[3][3][3];
    R zs[3][3], zd[3][3];
    // ---- z stage: populations -> (x,y) lines of z moments ----
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const R pm = f[dirOf(a - 1, b - 1, -1)];
            const R po = f[dirOf(a - 1, b - 1, 0)];
            const R pp = f[dirOf(a - 1, b - 1, 1)];
            zs[a][b] = pp + pm;
            zd[a][b] = pp - pm;
            m[a][b][0] = zs[a][b] + po;
        }
    // density and momentum from the zeroth z moments (:49-69)
    const R dRho = ((m[0][0][0] + m[0][1][0]) + m[0][2][0]) +
                   ((m[1][0][0] + m[1][1][0]) + m[1][2][0]) +
                   ((m[2][0][0] + m[2][1][0]) + m[2][2][0]);
    const R rho = dRho + 1.f;
    const R rhoInv = rcpR(rho);
    const R momX = ((m[2][0][0] + m[2][1][0]) + m[2][2][0]) - ((m[0][0][0] + m[0][1][0]) + m[0][2][0]);
    const R momY = ((m[0][2][0] + m[1][2][0]) + m[2][2][0]) - ((m[0][0][0] + m[1][0][0]) + m[2][0][0]);
    // z momentum: pairs (P - M) summed in the reference's grouping (:62-65)
    const R momZ = (((zd[0][0] + zd[0][1]) + (zd[0][2] + zd[1][0])) + ((zd[1][1] + zd[1][2]) + (zd[2][0] + zd[2][1]))) +
                   zd[2][2];

    const R ux = (momX + 0.5f * gx) * rhoInv;
    const R uy = (momY + 0.5f * gy) * rhoInv;
    const R uz = (momZ + 0.5f * gz) * rhoInv;
    const Shift<R> sx = shiftOf(ux), sy = shiftOf(uy), sz = shiftOf(uz);

#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) fwd(zs[a][b], zd[a][b], m[a][b][0], kZ<Sc>(a, b), sz, m[a][b][1], m[a][b][2]);
    // ---- y stage ----
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            const R lo = m[a][0][n], mid = m[a][1][n], hi = m[a][2][n];
            const R s = hi + lo;
            const R k0 = s + mid;
            fwd(s, hi - lo, k0, kY<Sc>(a, n), sy, m[a][1][n], m[a][2][n]);
            m[a][0][n] = k0;
        }
    // ---- x stage: central moments k[ord x][ord y][ord z] ----
    R k[3][3][3];
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            const R lo = m[0][b][n], mid = m[1][b][n], hi = m[2][b][n];
            const R s = hi + lo;
            const R k0 = (b == 0 && n == 0) ? dRho : s + mid;
            fwd(s, hi - lo, k0, kX<Sc>(b, n), sx, k[1][b][n], k[2][b][n]);
            k[0][b][n] = k0;
        }

    // ---- central moments -> cumulants (:164-187) ----
    const R C110 = k[1][1][0], C101 = k[1][0][1], C011 = k[0][1][1];
    const R C200 = k[2][0][0], C020 = k[0][2][0], C002 = k[0][0][2];
    const R C111 = k[1][1][1];
    const R C120 = k[1][2][0], C102 = k[1][0][2], C210 = k[2][1][0];
    const R C012 = k[0][1][2], C201 = k[2][0][1], C021 = k[0][2][1];
    const R dRhoNinth = dRho * rhoInv * kNinth;
    // C211, C121, C112, C220, C022, C202 (:170-187) only enter the reference's
    // relaxation multiplied by (1 - omega6..8) = 0, so they are not formed.
    const R k000 = dRho;

    // ---- relaxation (:193-342); omega2 = omega6 = omega7 = omega8 = 1, so
    // the (1 - omega) terms of those rates vanish and are not evaluated.  Every
    // product that is added to something is an explicit fused multiply-add:
    // the packed operations are not contracted by the compiler. ----
    const R A20 = C200 - C020, A02 = C200 - C002;
    const R trace = (C200 + C020) + C002 - k000;
    const R Dxu = rhoInv * fmaR(P.mHalfW1, A20 + A02, trace * -0.5f);
    const R rw15 = P.w1x15 * rhoInv;
    const R Dyv = fmaR(rw15, A20, Dxu);
    const R Dzw = fmaR(rw15, A02, Dxu);

    const R Cs110 = P.oneMinusW1 * C110;
    const R Cs101 = P.oneMinusW1 * C101;
    const R Cs011 = P.oneMinusW1 * C011;
    const R mr3 = rho * (Sc(-3) * P.halfW1c);
    const R xD = sx.u2 * Dxu, yD = sy.u2 * Dyv, zD = sz.u2 * Dzw;
    const R e33 = fmaR(mr3, xD - yD, P.oneMinusW1 * A20);
    const R e34 = fmaR(mr3, xD - zD, P.oneMinusW1 * A02);
    const R e35 = fmaR(rho * -1.5f, (xD + yD) + zD, k000);
    // the differences Cs200 - Cs020 = e33 and Cs200 - Cs002 = e34, the sum e35
    const R Cs200 = ((e33 + e34) + e35) * kThird;
    const R Cs020 = Cs200 - e33;
    const R Cs002 = Cs200 - e34;

    R Cs120 = bcast(Sc(0), dRho), Cs102 = Cs120, Cs210 = Cs120, Cs012 = Cs120, Cs201 = Cs120, Cs021 = Cs120;
    R Cs111 = Cs120;
    // fourth-order cumulants, with the rest of the moment they enter
    R f220 = dRhoNinth * -1.f, f202 = f220, f022 = f220, f211 = Cs120, f121 = Cs120, f112 = Cs120;
    const bool k17 = P.useK17 && lambda > Sc(0);
    if (k17) {
        // K17 with limiter: third-order rates pushed from omega3..5 towards 1
        // where the cumulant is large compared with lambda (:270-306):
        // 1 - (om + (1 - om) |v| / (lambda + |v|)) = (1 - om) lambda / (lambda + |v|),
        // applied to v (the denominator kept a normal number); the halves of
        // the sums and differences below are part of the factor
        const Sc lam = posMin(lambda);
        auto relax = [&](Sc factor, R v) { return divFast((factor * lam) * v, addAbs(lam, v)); };
        const Sc h3 = Sc(0.5) * P.oneMinusW3, h4 = Sc(0.5) * P.oneMinusW4;
        const R e117 = relax(h3, C120 + C102), e120 = relax(h4, C120 - C102);
        const R e118 = relax(h3, C210 + C012), e121 = relax(h4, C210 - C012);
        const R e119 = relax(h3, C201 + C021), e122 = relax(h4, C201 - C021);
        Cs120 = e117 + e120;
        Cs102 = e117 - e120;
        Cs210 = e118 + e121;
        Cs012 = e118 - e121;
        Cs201 = e119 + e122;
        Cs021 = e119 - e122;
        Cs111 = relax(P.oneMinusW5, C111);
        // fourth order (:310-323): omega6 = omega7 = 1 make the coefficient of the
        // trace, e45 = -(4/3) tau A rho (Dxu + Dyv + Dzw), minus twice that of
        // e43 and e44, c43 rho: the combinations reduce to two strain rates
        // each, and rho times the shear rates to the moments they came from
        const R mrc43 = rho * -P.c43;
        f220 = fmaR(mrc43, Dxu + Dyv, f220);
        f202 = fmaR(mrc43, Dxu + Dzw, f202);
        f022 = fmaR(mrc43, Dyv + Dzw, f022);
        const Sc cB3 = P.cB * P.mW1x3;
        f211 = cB3 * C011;
        f121 = cB3 * C101;
        f112 = cB3 * C110;
    }

    // ---- cumulants -> central moments (:348-384) ----
    R s[3][3][3];
    const R a3 = Cs200 + kThird, b3 = Cs020 + kThird, c3 = Cs002 + kThird;
    const R t200 = Cs200 * kThird, t020 = Cs020 * kThird, t002 = Cs002 * kThird;
    const R d110 = Cs110 + Cs110, d101 = Cs101 + Cs101, d011 = Cs011 + Cs011;
    const R m110 = Cs110 * Cs110, m101 = Cs101 * Cs101, m011 = Cs011 * Cs011;
    s[0][1][1] = Cs011; s[1][0][1] = Cs101; s[1][1][0] = Cs110; s[1][1][1] = Cs111;
    s[0][0][2] = Cs002; s[0][2][0] = Cs020; s[2][0][0] = Cs200;
    s[0][1][2] = Cs012; s[0][2][1] = Cs021; s[1][0][2] = Cs102;
    s[2][0][1] = Cs201; s[1][2][0] = Cs120; s[2][1][0] = Cs210;
    s[2][1][1] = fmaR(fmaR(a3, Cs011, Cs101 * d110), rhoInv, f211);
    s[1][2][1] = fmaR(fmaR(b3, Cs101, Cs011 * d110), rhoInv, f121);
    s[1][1][2] = fmaR(fmaR(c3, Cs110, Cs101 * d011), rhoInv, f112);
    s[2][2][0] = fmaR(fmaR(Cs020, a3, fmaR(m110, 2.f, t200)), rhoInv, f220);
    s[0][2][2] = fmaR(fmaR(Cs002, b3, fmaR(m011, 2.f, t020)), rhoInv, f022);
    s[2][0][2] = fmaR(fmaR(Cs200, c3, fmaR(m101, 2.f, t002)), rhoInv, f202);
    const R q111 = Cs111 * 4.f;
    if (k17) {
        s[1][2][2] = rhoInv * fmaR(b3, Cs102, fmaR(c3, Cs120, fmaR(q111, Cs011, fmaR(d110, Cs012, d101 * Cs021))));
        s[2][1][2] = rhoInv * fmaR(c3, Cs210, fmaR(a3, Cs012, fmaR(q111, Cs101, fmaR(d011, Cs201, d110 * Cs102))));
        s[2][2][1] = rhoInv * fmaR(a3, Cs021, fmaR(b3, Cs201, fmaR(q111, Cs110, fmaR(d101, Cs120, d011 * Cs210))));
    } else {
        // AllOne: every third-order cumulant is zero, and so are these moments
        s[1][2][2] = Cs120;
        s[2][1][2] = Cs120;
        s[2][2][1] = Cs120;
    }
    {
        R lin = fmaR(Cs200, s[0][2][2], fmaR(Cs020, s[2][0][2], Cs002 * s[2][2][0]));
        lin = fmaR(fmaR(Cs011, s[2][1][1], fmaR(Cs101, s[1][2][1], Cs110 * s[1][1][2])), 4.f, lin);
        if (k17) {
            lin = fmaR(q111, Cs111, lin);
            lin = fmaR(fmaR(Cs120, Cs102, fmaR(Cs210, Cs012, Cs201 * Cs021)), 2.f, lin);
        }
        const R p = Cs200 * Cs020, q = Cs200 + Cs020, sum = q + Cs002;
        // half the cubic term
        const R cub = fmaR(fmaR(d110 * d101, Cs011, fmaR(m101, Cs020, fmaR(m011, Cs200, m110 * Cs002))), 2.f, p * Cs002);
        const R sq = fmaR((m101 + m011) + m110, 2.f, fmaR(sum, kThird, fmaR(Cs002, q, p)));
        const R fourth = fmaR((s[0][2][2] + s[2][0][2]) + s[2][2][0], 3.f, sum);
        const R inner = fmaR(cub, 2.f, fmaR(sq, Frac<Sc>::twoThirds, fmaR(dRho, dRho, dRho * -1.f) * k27th));
        s[2][2][2] = rhoInv * fmaR(rhoInv * -1.f, inner, fmaR(fourth, kNinth, lin));
    }
    s[0][0][0] = k000;
    // the first-order moments change sign (:386-388): about the velocity with
    // half the force they are minus half the force before the collision
    s[1][0][0] = k[1][0][0] * -1.f;
    s[0][1][0] = k[0][1][0] * -1.f;
    s[0][0][1] = k[0][0][1] * -1.f;

    // ---- back transform, x stage (:390-418): s[ord x][..] -> m[pop x][ord y][ord z]
    {
        const Axis<R> X = axisOf(ux);
        const R mK1 = X.u2 * -1.f, mK3 = X.u2 * -kThird, mK9 = X.u2 * -kNinth;
#pragma unroll
        for (int b = 0; b < 3; ++b)
#pragma unroll
            for (int n = 0; n < 3; ++n) {
                const Sc K = kX<Sc>(b, n);
                const R mKu2 = (b == 0 && n == 0) ? mK1 : (b == 2 && n == 2) ? mK9 : mK3;
                bwd(s[0][b][n], s[1][b][n], s[2][b][n], K, mKu2, X, m[0][b][n], m[1][b][n], m[2][b][n]);
            }
    }
    // ---- y stage (:420-448)
    {
        const Axis<R> Y = axisOf(uy);
        const R mKa0 = Y.u2 * -kY<Sc>(0, 0), mKb0 = Y.u2 * -kY<Sc>(1, 0);
        const R mKa2 = Y.u2 * -kY<Sc>(0, 2), mKb2 = Y.u2 * -kY<Sc>(1, 2);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int n = 0; n < 3; ++n) {
                const Sc K = kY<Sc>(a, n);
                const R mKu2 = n == 0 ? (a == 1 ? mKb0 : mKa0) : (a == 1 ? mKb2 : mKa2);
                const R s0 = m[a][0][n], s1 = m[a][1][n], s2 = m[a][2][n];
                bwd(s0, s1, s2, K, mKu2, Y, m[a][0][n], m[a][1][n], m[a][2][n]);
            }
    }
    // ---- z stage (:450-490): back to populations
    {
        const Axis<R> Z = axisOf(uz);
        const R mKc = Z.u2 * -kZ<Sc>(1, 1), mKe = Z.u2 * -kZ<Sc>(0, 1), mKv = Z.u2 * -kZ<Sc>(0, 0);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const Sc K = kZ<Sc>(a, b);
                const R mKu2 = (a == 1 && b == 1) ? mKc : (a == 1 || b == 1) ? mKe : mKv;
                bwd(m[a][b][0], m[a][b][1], m[a][b][2], K, mKu2, Z, f[dirOf(a - 1, b - 1, -1)],
                    f[dirOf(a - 1, b - 1, 0)], f[dirOf(a - 1, b - 1, 1)]);
            }
    }
}

}  // namespace lbm
