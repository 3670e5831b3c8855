// collision_math.cuh -- per-node collision operators, held in registers.
//
// K17: the compressible cumulant collision of VirtualFluids
// (src/lbm/collision/K17CompressibleNavierStokes.h:87-591, TurbulenceModel::None),
// based on Geier et al., J. Comput. Phys. 348 (2017) 862-888 and 889-898.
// The operator is the reference's; its arithmetic is arranged for the fewest
// instructions, because the 16-bit storages and the adjoint are bound by the
// floating-point pipes (and FP32 by their power):
//   * orders 4..6 do not depend on their pre-collision values (O4 = O5 = O6 =
//     1), so only the 17 raw moments up to order 3 are formed, by sums and
//     differences along z, y and x (no multiplication), and those are shifted
//     to central moments about the velocity;
//   * the limiter O + (1 - O) |x| / (|x| + ql) enters as its complement
//     (1 - O) ql / (|x| + ql), one reciprocal and two multiplications;
//   * second moments are carried as deviations from rho / 3, in which the
//     Gaussian closure of orders 4..6 is short and well conditioned
//     (c200 c020 / rho = rho / 9 + (p + q) / 3 + p q / rho);
//   * every moment is carried times 1/2 per non-zero exponent, which folds the
//     halvings of the back transform into the operator's constants;
//   * the terms of a force are a block of their own, skipped for a launch
//     without one;
//   * rates that depend only on omega and the limiters are formed once per
//     launch on the host (K17Rates) with the reference's expressions.
// Live operations of one node (add, multiply, multiply-add; paired FP32): 450
// without a force, 470 with one, against 630 of the term-by-term arrangement
// (forward chimera sweeps on all 27 moments, cumulants by the reference's
// expressions), counted on a recorded trace.
// Results agree with the reference to rounding: FP64 fields within 1e-12
// relative of the oracle after many steps (tests/test_gpu_collision.py).
//
// BGK: src/gpu/core/Kernel/Compressible/NavierStokes/B92/B92CompressibleNavierStokes_Device.cu:194-234.
#pragma once

#include "d3q27.cuh"

namespace vfb
{

// The scalar type behind an arithmetic type R (R itself for float / double;
// a paired type maps to its element type), and the rational constants of the
// operator as compile-time scalars converted to R.
template <class R>
struct ScalarOf {
    using type = R;
};
template <class R>
__host__ __device__ __forceinline__ R cst(int n, int m)
{
    using S = typename ScalarOf<R>::type;
    return R(S(n) / S(m));
}

// Per-launch constants of the K17 collision (rates and factors of
// K17CompressibleNavierStokes.h:245-273 and :452-457, limiter inputs :176-178,
// combined and scaled as k17Collide uses them):
//   omega             relaxation rate (the BGK collision's too)
//   halfMinusOmega    -omega / 2           omegaThreeHalves  3 omega / 2
//   keepHalf          (1 - omega) / 2      corrHalf          -3/2 (1 - omega / 2)
//   keep, keepQuarter (1 - omega), (1 - omega) / 4
//   mixed4            (1 - omega) / 24 + fourthB / 8
//   limP, limM, limD  (1 - O) ql of the three limiters, over 8, 8 and 2
//   qlP, qlM, qlD     quartic limiters
//   fourthA4, minusFourthA4, fourthA24    fourthA / 4, its negative, fourthA / 24
//   twoFourthB        2 fourthB
// with fourthA = -(1/omega - 1/2) 2/3 A and fourthB = (1/omega - 1/2) omega B.
#define VFB_K17_RATES(X)                                                                                               \
    X(omega) X(halfMinusOmega) X(omegaThreeHalves) X(keepHalf) X(corrHalf) X(keep) X(keepQuarter) X(mixed4) X(limP)    \
    X(limM) X(limD) X(qlP) X(qlM) X(qlD) X(fourthA4) X(minusFourthA4) X(fourthA24) X(twoFourthB)

template <class R>
struct K17Rates {
#define VFB_FIELD(name) R name;
    VFB_K17_RATES(VFB_FIELD)
#undef VFB_FIELD
};

// A limiter above 2^60 (infinity too) leaves a moment's rate at O to rounding,
// one below 2^-100 relaxes it fully; inside these bounds the products with ql
// and the reciprocal stay finite in FP32.
template <class R>
inline R boundedLimiter(R ql)
{
    const R hi = R(1152921504606846976.0), lo = R(7.888609052210118e-31);
    return ql > hi ? hi : ql >= R(0) && ql < lo ? lo : ql;
}

template <class R>
inline K17Rates<R> makeK17Rates(R omega, R qlP, R qlM, R qlD)
{
    K17Rates<R> r;
    r.omega = omega;
    const R OxyyPxzz = R(8) * (-R(2) + omega) * (R(1) + R(2) * omega) / (-R(8) - R(14) * omega + R(7) * omega * omega);
    const R OxyyMxzz =
        R(8) * (-R(2) + omega) * (-R(7) + R(4) * omega) / (R(56) - R(50) * omega + R(9) * omega * omega);
    const R Oxyz = R(24) * (-R(2) + omega) * (-R(2) - R(7) * omega + R(3) * omega * omega) /
                   (R(48) + R(152) * omega - R(130) * omega * omega + R(29) * omega * omega * omega);
    const R factorA = (R(4) + R(2) * omega - R(3) * omega * omega) / (R(2) - R(7) * omega + R(5) * omega * omega);
    const R factorB = (R(4) + R(28) * omega - R(14) * omega * omega) / (R(6) - R(21) * omega + R(15) * omega * omega);
    const R minusTau = -R(1) * (R(1) / omega - cst<R>(1, 2));
    const R fourthA = minusTau * cst<R>(2, 3) * factorA;
    const R fourthB = minusTau * (-R(3) * omega) * cst<R>(1, 3) * factorB;
    r.halfMinusOmega = cst<R>(1, 2) * (-omega);
    r.omegaThreeHalves = omega * (cst<R>(3, 2));
    r.keep = R(1) - omega;
    r.keepHalf = r.keep * R(0.5);
    r.keepQuarter = r.keep * R(0.25);
    r.corrHalf = -cst<R>(3, 2) * (R(1) + cst<R>(1, 2) * (-omega));
    r.mixed4 = r.keep * cst<R>(1, 24) + fourthB * R(0.125);
    r.qlP = boundedLimiter(qlP);
    r.qlM = boundedLimiter(qlM);
    r.qlD = boundedLimiter(qlD);
    r.limP = (R(1) - OxyyPxzz) * r.qlP * R(0.125);
    r.limM = (R(1) - OxyyMxzz) * r.qlM * R(0.125);
    r.limD = (R(1) - Oxyz) * r.qlD * R(0.5);
    r.fourthA4 = fourthA * R(0.25);
    r.minusFourthA4 = -r.fourthA4;
    r.fourthA24 = fourthA * cst<R>(1, 24);
    r.twoFourthB = R(2) * fourthB;
    return r;
}

// -------------------------------------------------------------- transforms --
// Raw moments of order 0, 1, 2 of one lattice line (a, b, c) = (-1, 0, +1), in
// place: sums and differences only.
template <class R>
__host__ __device__ __forceinline__ void lineMoments(R& a, R& b, R& c)
{
    const R m2 = a + c;
    const R m1 = c - a;
    a = m2 + b;
    b = m1;
    c = m2;
}

// The back transform of one line: central moments (a, b, c) of order 0, 1, 2
// about the velocity v to the line's populations, the inverse of
// ChimeraTransformation.h:58-121 (Geier et al. 2015, appendix J) with the
// equilibrium part K of the zeroth moment.  b and c come as halves: with
//   r1 = (b + v (a + K)) / 2,   r2 = (c + v b + v (b + v (a + K))) / 2
// half the raw moments, the populations are r2 - r1, a - 2 r2 and r2 + r1.
template <class R>
struct Sweep {
    R v, half;
    __host__ __device__ __forceinline__ Sweep(R velocity)
    {
        v = velocity;
        half = R(0.5) * velocity;
    }
};

template <class R>
__host__ __device__ __forceinline__ void bwd(R& a, R& b, R& c, const Sweep<R>& w, typename ScalarOf<R>::type K)
{
    const R aK = K != 0 ? a + R(K) : a;
    const R r1 = fma(w.half, aK, b);
    const R r2 = fma(w.v, b + r1, c);
    b = fma(R(-2), r2, a);
    a = r2 - r1;
    c = r2 + r1;
}

// --------------------------------------------------------- macroscopic sums --
// MacroscopicQuantities.h:55-127 (pyramid summation)
template <class R>
__host__ __device__ __forceinline__ R pyramidDensity(const R* f)
{
    const R t1 = ((f[dPPP] + f[dMMM]) + (f[dMPM] + f[dPMP])) + ((f[dMPP] + f[dPMM]) + (f[dMMP] + f[dPPM]));
    const R t2 = (((f[d0MP] + f[d0PM]) + (f[d0MM] + f[d0PP])) + ((f[dM0P] + f[dP0M]) + (f[dM0M] + f[dP0P]))) +
                 ((f[dMP0] + f[dPM0]) + (f[dMM0] + f[dPP0]));
    const R t3 = ((f[dM00] + f[dP00]) + (f[d0M0] + f[d0P0])) + (f[d00M] + f[d00P]);
    return ((t1 + t2) + f[d000]) + t3;
}
template <class R>
__host__ __device__ __forceinline__ R pyramidJx(const R* f)
{
    return ((((f[dPPP] - f[dMMM]) + (f[dPMP] - f[dMPM])) + ((f[dPMM] - f[dMPP]) + (f[dPPM] - f[dMMP]))) +
            (((f[dP0M] - f[dM0P]) + (f[dP0P] - f[dM0M])) + ((f[dPM0] - f[dMP0]) + (f[dPP0] - f[dMM0])))) +
           (f[dP00] - f[dM00]);
}
template <class R>
__host__ __device__ __forceinline__ R pyramidJy(const R* f)
{
    return ((((f[dPPP] - f[dMMM]) + (f[dMPM] - f[dPMP])) + ((f[dMPP] - f[dPMM]) + (f[dPPM] - f[dMMP]))) +
            (((f[d0PM] - f[d0MP]) + (f[d0PP] - f[d0MM])) + ((f[dMP0] - f[dPM0]) + (f[dPP0] - f[dMM0])))) +
           (f[d0P0] - f[d0M0]);
}
template <class R>
__host__ __device__ __forceinline__ R pyramidJz(const R* f)
{
    return ((((f[dPPP] - f[dMMM]) + (f[dPMP] - f[dMPM])) + ((f[dMPP] - f[dPMM]) + (f[dMMP] - f[dPPM]))) +
            (((f[d0MP] - f[d0PM]) + (f[d0PP] - f[d0MM])) + ((f[dM0P] - f[dP0M]) + (f[dP0P] - f[dM0M])))) +
           (f[d00P] - f[d00M]);
}

// ------------------------------------------------------------------- K17 --
// 1 / x of the density.
template <class R>
__host__ __device__ __forceinline__ R reciprocal(R x)
{
    return R(1) / x;
}
// 1 / x of a limiter's denominator: in FP32 the hardware's approximate
// reciprocal (relative error about 1e-7 of a moment that is a small part of
// the populations)
template <class R>
__host__ __device__ __forceinline__ R limiterReciprocal(R x)
{
    return R(1) / x;
}
#ifdef __CUDA_ARCH__
__device__ __forceinline__ float approximateReciprocal(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// one Newton-Raphson step r (2 - x r) on the approximate reciprocal
template <>
__device__ __forceinline__ float reciprocal<float>(float x)
{
    const float r = approximateReciprocal(x);
    return fmaf(fmaf(-x, r, 1.0f), r, r);
}
template <>
__device__ __forceinline__ float limiterReciprocal<float>(float x)
{
    return approximateReciprocal(x);
}
// FP64: the single-precision reciprocal and two Newton-Raphson steps r (2 - x r),
// each of which squares the relative error: 1.5 * 2^-23 at most (x rounded to
// single precision, the approximation), then below 2^-44, then rounding.  A
// collision has eight reciprocals; as divisions they made Taylor-Green 128^3
// (two steps, B200) 345 us instead of 322, the 64^3 cavity 58.2 instead of 55.7.
// x: a density or a limiter's denominator, both far inside the range of FP32
// (boundedLimiter; tests/test_gpu_k17_limits.py).
__device__ __forceinline__ double newtonReciprocal(double x)
{
    double r = (double)approximateReciprocal((float)x);
    r = ::fma(::fma(-x, r, 1.0), r, r);
    return ::fma(::fma(-x, r, 1.0), r, r);
}
template <>
__device__ __forceinline__ double reciprocal<double>(double x)
{
    return newtonReciprocal(x);
}
template <>
__device__ __forceinline__ double limiterReciprocal<double>(double x)
{
    return newtonReciprocal(x);
}
#endif

// a third-order combination x relaxed by its limited rate: x (1 - O) ql / (|x| + ql)
template <class R>
__host__ __device__ __forceinline__ R limitedMoment(R x, R lim, R ql)
{
    return (x * lim) * limiterReciprocal(fabs(x) + ql);
}

// Central moments, scaled by 1/2 per non-zero exponent (in the slots of
// k17Collide's naming: m_abc in the slot of direction (a-1, b-1, c-1)), to
// populations: the back transform in x, then y, then z
// (K17CompressibleNavierStokes.h:525-557).  The equilibrium parts K carry the
// scale of their line.
template <class R>
__host__ __device__ __forceinline__ void scaledMomentsToPopulations(R* f, R vvx, R vvy, R vvz)
{
    using S = typename ScalarOf<R>::type;
    {
        const Sweep<R> w(vvx);
        bwd(f[dMMM], f[d0MM], f[dPMM], w, S(1));
        bwd(f[dM0M], f[d00M], f[dP0M], w, S(0));
        bwd(f[dMPM], f[d0PM], f[dPPM], w, cst<S>(1, 6));
        bwd(f[dMM0], f[d0M0], f[dPM0], w, S(0));
        bwd(f[dM00], f[d000], f[dP00], w, S(0));
        bwd(f[dMP0], f[d0P0], f[dPP0], w, S(0));
        bwd(f[dMMP], f[d0MP], f[dPMP], w, cst<S>(1, 6));
        bwd(f[dM0P], f[d00P], f[dP0P], w, S(0));
        bwd(f[dMPP], f[d0PP], f[dPPP], w, cst<S>(1, 36));
    }
    {
        const Sweep<R> w(vvy);
        bwd(f[dMMM], f[dM0M], f[dMPM], w, cst<S>(1, 6));
        bwd(f[dMM0], f[dM00], f[dMP0], w, S(0));
        bwd(f[dMMP], f[dM0P], f[dMPP], w, cst<S>(1, 36));
        bwd(f[d0MM], f[d00M], f[d0PM], w, cst<S>(2, 3));
        bwd(f[d0M0], f[d000], f[d0P0], w, S(0));
        bwd(f[d0MP], f[d00P], f[d0PP], w, cst<S>(1, 9));
        bwd(f[dPMM], f[dP0M], f[dPPM], w, cst<S>(1, 6));
        bwd(f[dPM0], f[dP00], f[dPP0], w, S(0));
        bwd(f[dPMP], f[dP0P], f[dPPP], w, cst<S>(1, 36));
    }
    {
        const Sweep<R> w(vvz);
        bwd(f[dMMM], f[dMM0], f[dMMP], w, cst<S>(1, 36));
        bwd(f[dM0M], f[dM00], f[dM0P], w, cst<S>(1, 9));
        bwd(f[dMPM], f[dMP0], f[dMPP], w, cst<S>(1, 36));
        bwd(f[d0MM], f[d0M0], f[d0MP], w, cst<S>(1, 9));
        bwd(f[d00M], f[d000], f[d00P], w, cst<S>(4, 9));
        bwd(f[d0PM], f[d0P0], f[d0PP], w, cst<S>(1, 9));
        bwd(f[dPMM], f[dPM0], f[dPMP], w, cst<S>(1, 36));
        bwd(f[dP0M], f[dP00], f[dP0P], w, cst<S>(1, 9));
        bwd(f[dPPM], f[dPP0], f[dPPP], w, cst<S>(1, 36));
    }
}

// the same from unscaled central moments (the interface interpolation,
// InterpolationCF.h:250-285): exact scalings first
template <class R>
__host__ __device__ __forceinline__ void centralMomentsToPopulations(R* f, R vvx, R vvy, R vvz)
{
#pragma unroll
    for (int d = 0; d < 27; ++d) {
        // the moment in the slot of direction d has a non-zero exponent on the axes where c_d >= 0
        const int nz = (cx(d) >= 0) + (cy(d) >= 0) + (cz(d) >= 0);
        if (nz)
            f[d] = f[d] * R(nz == 1 ? 0.5 : nz == 2 ? 0.25 : 0.125);
    }
    scaledMomentsToPopulations(f, vvx, vvy, vvz);
}

// One K17 collision on f[27] (pre-collision in, post-collision out).
// (fx, fy, fz) is half the acceleration already scaled by the level factor
// (RunCollision.cuh:111-113); forced = false promises that it is zero.
// Returns drho and the force-shifted velocity.
template <class R>
__host__ __device__ __forceinline__ void k17Collide(R* f, const K17Rates<R>& r, R fx, R fy, R fz, R& drho_out,
                                                    R& vx_out, R& vy_out, R& vz_out, bool forced = true)
{
    // moment names: m_abc (x^a y^b z^c) in the slot of direction (a-1, b-1, c-1)
    R& m000 = f[dMMM];
    R& m100 = f[d0MM];
    R& m200 = f[dPMM];
    R& m010 = f[dM0M];
    R& m110 = f[d00M];
    R& m210 = f[dP0M];
    R& m020 = f[dMPM];
    R& m120 = f[d0PM];
    R& m220 = f[dPPM];
    R& m001 = f[dMM0];
    R& m101 = f[d0M0];
    R& m201 = f[dPM0];
    R& m011 = f[dM00];
    R& m111 = f[d000];
    R& m211 = f[dP00];
    R& m021 = f[dMP0];
    R& m121 = f[d0P0];
    R& m221 = f[dPP0];
    R& m002 = f[dMMP];
    R& m102 = f[d0MP];
    R& m202 = f[dPMP];
    R& m012 = f[dM0P];
    R& m112 = f[d00P];
    R& m212 = f[dP0P];
    R& m022 = f[dMPP];
    R& m122 = f[d0PP];
    R& m222 = f[dPPP];

    // raw moments of the deviations, axis by axis (those above order 3 are
    // never used and cost nothing)
    lineMoments(f[dMMM], f[dMM0], f[dMMP]);
    lineMoments(f[dM0M], f[dM00], f[dM0P]);
    lineMoments(f[dMPM], f[dMP0], f[dMPP]);
    lineMoments(f[d0MM], f[d0M0], f[d0MP]);
    lineMoments(f[d00M], f[d000], f[d00P]);
    lineMoments(f[d0PM], f[d0P0], f[d0PP]);
    lineMoments(f[dPMM], f[dPM0], f[dPMP]);
    lineMoments(f[dP0M], f[dP00], f[dP0P]);
    lineMoments(f[dPPM], f[dPP0], f[dPPP]);

    lineMoments(f[dMMM], f[dM0M], f[dMPM]);
    lineMoments(f[dMM0], f[dM00], f[dMP0]);
    lineMoments(f[dMMP], f[dM0P], f[dMPP]);
    lineMoments(f[d0MM], f[d00M], f[d0PM]);
    lineMoments(f[d0M0], f[d000], f[d0P0]);
    lineMoments(f[d0MP], f[d00P], f[d0PP]);
    lineMoments(f[dPMM], f[dP0M], f[dPPM]);
    lineMoments(f[dPM0], f[dP00], f[dPP0]);
    lineMoments(f[dPMP], f[dP0P], f[dPPP]);

    lineMoments(f[dMMM], f[d0MM], f[dPMM]);
    lineMoments(f[dM0M], f[d00M], f[dP0M]);
    lineMoments(f[dMPM], f[d0PM], f[dPPM]);
    lineMoments(f[dMM0], f[d0M0], f[dPM0]);
    lineMoments(f[dM00], f[d000], f[dP00]);
    lineMoments(f[dMP0], f[d0P0], f[dPP0]);
    lineMoments(f[dMMP], f[d0MP], f[dPMP]);
    lineMoments(f[dM0P], f[d00P], f[dP0P]);

    const R drho = m000;
    const R rho = drho + R(1);
    const R oneOverRho = reciprocal(rho);
    const R vvx = fma(m100, oneOverRho, fx);
    const R vvy = fma(m010, oneOverRho, fy);
    const R vvz = fma(m001, oneOverRho, fz);
    const R nx = -vvx, ny = -vvy, nz = -vvz;
    const R vx2 = vvx * vvx, vy2 = vvy * vvy, vz2 = vvz * vvz;

    // central moments about v.  Second order (with j the momentum):
    //   c200 = m200 - vx jx,  c110 = m110 - vx jy
    // third order, with the raw second moments M = m + 1/3 and m011:
    //   c210 = m210 - vy M200 - 2 vx c110,  c111 = m111 - vx m011 - vy c101 - vz c110
    const R raw200 = m200 + cst<R>(1, 3), raw020 = m020 + cst<R>(1, 3), raw002 = m002 + cst<R>(1, 3);
    const R raw011 = m011;
    m200 = fma(nx, m100, m200);
    m020 = fma(ny, m010, m020);
    m002 = fma(nz, m001, m002);
    m110 = fma(nx, m010, m110);
    m101 = fma(nx, m001, m101);
    m011 = fma(ny, m001, m011);
    // with a force the first central moments are -rho (fx, fy, fz): their
    // contributions to the shifts, and their changed signs after the collision (:512-514)
    m100 = R(0);
    m010 = R(0);
    m001 = R(0);
    if (forced) {
        const R gx = rho * fx, gy = rho * fy, gz = rho * fz;
        m200 = fma(vvx, gx, m200);
        m020 = fma(vvy, gy, m020);
        m002 = fma(vvz, gz, m002);
        m110 = fma(vvy, gx, m110);
        m101 = fma(vvz, gx, m101);
        m011 = fma(vvz, gy, m011);
        m210 = fma(vx2, gy, m210);
        m201 = fma(vx2, gz, m201);
        m120 = fma(vy2, gx, m120);
        m021 = fma(vy2, gz, m021);
        m102 = fma(vz2, gx, m102);
        m012 = fma(vz2, gy, m012);
        m111 = fma(vvy * vvz, gx, m111);
        m100 = R(0.5) * gx;
        m010 = R(0.5) * gy;
        m001 = R(0.5) * gz;
    }
    const R n2x = nx + nx, n2y = ny + ny, n2z = nz + nz;
    m210 = fma(n2x, m110, fma(ny, raw200, m210));
    m201 = fma(n2x, m101, fma(nz, raw200, m201));
    m120 = fma(n2y, m110, fma(nx, raw020, m120));
    m021 = fma(n2y, m011, fma(nz, raw020, m021));
    m102 = fma(n2z, m101, fma(nx, raw002, m102));
    m012 = fma(n2z, m011, fma(ny, raw002, m012));
    m111 = fma(nz, m110, fma(ny, m101, fma(nx, raw011, m111)));

    // velocity gradients (:357-362), OxxPyyPzz = 1
    const R mxxMyy = m200 - m020;
    const R mxxMzz = m200 - m002;
    const R nonEq = drho - (m200 + m020 + m002);
    const R dxux = fma(r.halfMinusOmega, mxxMyy + mxxMzz, R(0.5) * nonEq);
    const R dyuy = fma(r.omegaThreeHalves, mxxMyy, dxux);
    const R dzuz = fma(r.omegaThreeHalves, mxxMzz, dxux);

    // second order relaxation with correction (:387-389).  p, q, s: halves of
    // the post-collision c200, c020, c002 less rho / 3; their sum is trace
    const R sx = vx2 * dxux, sy = vy2 * dyuy, sz = vz2 * dzuz;
    const R trace = R(-0.75) * (sx + sy + sz);
    const R xMy = fma(r.keepHalf, mxxMyy, r.corrHalf * (sx - sy));
    const R xMz = fma(r.keepHalf, mxxMzz, r.corrHalf * (sx - sz));
    const R p = cst<R>(1, 3) * (xMy + xMz + trace);
    const R q = p - xMy;
    const R s = p - xMz;
    // mixed moments: post-collision a = c011 / 4, b = c101 / 4, c = c110 / 4;
    // the linear part of the fourth-order mixed ones (c011 / 3 of the closure
    // and the optimised equilibrium, :452-457, both multiples of the pre-collision c011)
    const R a = r.keepQuarter * m011, b = r.keepQuarter * m101, c = r.keepQuarter * m110;
    const R a4 = r.keep * m011, b4 = r.keep * m101, c4 = r.keep * m110;
    const R la = r.mixed4 * m011, lb = r.mixed4 * m101, lc = r.mixed4 * m110;
    const R mixed = fma(c, m110, fma(b, m101, a * m011));

    // third order with quartic limiters (:404-417), scaled: t4 = c111 / 2, the rest / 8
    const R t4 = limitedMoment(m111, r.limD, r.qlD);
    const R xxyP = limitedMoment(m210 + m012, r.limP, r.qlP), xxyM = limitedMoment(m210 - m012, r.limM, r.qlM);
    const R xxzP = limitedMoment(m201 + m021, r.limP, r.qlP), xxzM = limitedMoment(m201 - m021, r.limM, r.qlM);
    const R xyyP = limitedMoment(m120 + m102, r.limP, r.qlP), xyyM = limitedMoment(m120 - m102, r.limM, r.qlM);
    m210 = xxyP + xxyM;
    m012 = xxyP - xxyM;
    m201 = xxzP + xxzM;
    m021 = xxzP - xxzM;
    m120 = xyyP + xyyM;
    m102 = xyyP - xyyM;

    // fourth order: Gaussian closure plus the modified equilibrium (:452-457, :478-488)
    const R n211 = fma(b4, c, p * a), n121 = fma(a4, c, q * b), n112 = fma(a4, b, s * c);
    const R n220 = fma(R(2) * c4, c, p * q), n202 = fma(R(2) * b4, b, p * s), n022 = fma(R(2) * a4, a, q * s);
    const R divergence = dxux + dyuy + dzuz;
    const R base = fma(r.fourthA4, divergence, fma(cst<R>(1, 6), trace, cst<R>(1, 36) * drho));
    m220 = fma(n220, oneOverRho, fma(-cst<R>(1, 6), s, fma(r.minusFourthA4, dzuz, base)));
    m202 = fma(n202, oneOverRho, fma(-cst<R>(1, 6), q, fma(r.minusFourthA4, dyuy, base)));
    m022 = fma(n022, oneOverRho, fma(-cst<R>(1, 6), p, fma(r.minusFourthA4, dxux, base)));
    m211 = fma(n211, oneOverRho, la);
    m121 = fma(n121, oneOverRho, lb);
    m112 = fma(n112, oneOverRho, lc);

    // fifth and sixth order: cumulants zero (:463-471, :489-505)
    {
        const R third = cst<R>(1, 3);
        const R n122 = fma(a4, t4, fma(b4, m021, fma(c4, m012, fma(q, m102, s * m120))));
        const R n212 = fma(b4, t4, fma(a4, m201, fma(c4, m102, fma(p, m012, s * m210))));
        const R n221 = fma(c4, t4, fma(b4, m120, fma(a4, m210, fma(q, m201, p * m021))));
        m122 = fma(n122, oneOverRho, third * xyyP);
        m212 = fma(n212, oneOverRho, third * xxyP);
        m221 = fma(n221, oneOverRho, third * xxzP);
        const R e = fma(m201, m021, fma(m210, m012, m120 * m102));
        const R g = fma(divergence, trace, -fma(p, dxux, fma(q, dyuy, s * dzuz)));
        const R first = fma(R(2), fma(R(2), e, t4 * t4),
                            fma(cst<R>(1, 6), n220 + n202 + n022, fma(r.twoFourthB, mixed, r.fourthA4 * g)));
        const R second = fma(R(2), fma(b4, n121, c4 * n112), p * n022);
        m222 = fma(fma(second, oneOverRho, first), oneOverRho,
                   fma(cst<R>(1, 6), base, r.fourthA24 * divergence));
    }

    // the remaining scaled moments; m000 = drho stays
    const R drho6 = cst<R>(1, 6) * drho;
    m200 = p + drho6;
    m020 = q + drho6;
    m002 = s + drho6;
    m011 = a;
    m101 = b;
    m110 = c;
    m111 = R(0.25) * t4;

    scaledMomentsToPopulations(f, vvx, vvy, vvz);

    drho_out = drho;
    vx_out = vvx;
    vy_out = vvy;
    vz_out = vvz;
}

// ------------------------------------------------------------------- BGK --
template <class R>
__host__ __device__ __forceinline__ void bgkCollide(R* f, R omega)
{
    R drho = (f[dPPP] + f[dMMM]) + (f[dMMP] + f[dPPM]) + (f[dPMP] + f[dMPM]) + (f[dMPP] + f[dPMM]) +
             (f[dPP0] + f[dMM0]) + (f[dMP0] + f[dPM0]) + (f[dP0P] + f[dM0M]) + (f[dP0M] + f[dM0P]) +
             (f[d0PP] + f[d0MM]) + (f[d0PM] + f[d0MP]) + (f[dP00] + f[dM00]) + (f[d0P0] + f[d0M0]) +
             (f[d00P] + f[d00M]) + f[d000];
    const R rho = drho + R(1);
    const R OORho = R(1) / rho;
    const R vx1 = OORho * ((f[dPPP] - f[dMMM]) + (f[dPPM] - f[dMMP]) + (f[dPMP] - f[dMPM]) + (f[dPMM] - f[dMPP]) +
                           (f[dPP0] - f[dMM0]) + (f[dPM0] - f[dMP0]) + (f[dP0P] - f[dM0M]) + (f[dP0M] - f[dM0P]) +
                           (f[dP00] - f[dM00]));
    const R vx2 = OORho * ((f[dPPP] - f[dMMM]) + (f[dPPM] - f[dMMP]) + (f[dMPM] - f[dPMP]) + (f[dMPP] - f[dPMM]) +
                           (f[dPP0] - f[dMM0]) + (f[dMP0] - f[dPM0]) + (f[d0PP] - f[d0MM]) + (f[d0PM] - f[d0MP]) +
                           (f[d0P0] - f[d0M0]));
    const R vx3 = OORho * ((f[dPPP] - f[dMMM]) + (f[dMMP] - f[dPPM]) + (f[dPMP] - f[dMPM]) + (f[dMPP] - f[dPMM]) +
                           (f[dP0P] - f[dM0M]) + (f[dM0P] - f[dP0M]) + (f[d0PP] - f[d0MM]) + (f[d0MP] - f[d0PM]) +
                           (f[d00P] - f[d00M]));
    const R cusq = R(1.5) * (vx1 * vx1 + vx2 * vx2 + vx3 * vx3);
    const R keep = R(1) + (-omega);
    // the weights as compile-time scalars (for a paired type R this avoids a
    // runtime division per direction; for float / double it is weight<R>)
    using S = typename ScalarOf<R>::type;
    f[d000] = f[d000] * keep - (-omega) * R(weight<S>(d000)) * (drho - rho * cusq);
#pragma unroll
    for (int d = 1; d < 27; ++d) {
        const R cu = cdot<R>(d, vx1, vx2, vx3);
        f[d] = f[d] * keep - (-omega) * R(weight<S>(d)) * (drho + rho * (R(3) * cu + R(4.5) * cu * cu - cusq));
    }
}

} // namespace vfb
