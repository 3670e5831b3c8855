// collision_math16.cuh -- the K17 collision of the 16-bit storages (FP32
// arithmetic): the same operator as k17Collide of collision_math.cuh, in the
// arrangement that follows the reference's expressions term by term (630
// operations a node against 450 there).
//
// The two arrangements round differently, by a few units of FP32 (the shorter
// one less).  In FP32 and FP64 storage that stays at rounding level.  A 16-bit
// store turns it into a different code wherever a value lies next to a rounding
// boundary, about one stored value in ten in the corner directions: after four
// steps of Taylor-Green 320^3 the z velocity (little more than noise there)
// differed by 1%, the two-level cube's FP16 populations by 1.7e-4, while the
// error against 64 bits stayed at that of the format.  The shorter arrangement
// would make these storages 9% to 12% faster; the collision keeps the codes it
// has stored so far (tests/test_gpu_16bit_codes.py).  The boundary lists and
// the refinement interface have one arrangement for all storages.
#pragma once

#include "collision_math.cuh"
#include "storage.cuh"

namespace vfb
{
namespace termwise
{
// per-launch constants (K17CompressibleNavierStokes.h:245-273, limiter inputs :176-178)
#define VFB_K17_TERM_RATES(X)                                                                                          \
    X(omega) X(minusOmega) X(OxyyPxzz) X(OxyyMxzz) X(Oxyz) X(oneMinusOxyyPxzz) X(oneMinusOxyyMxzz) X(oneMinusOxyz)     \
    X(halfMinusOmega) X(omegaThreeHalves) X(secondOrderCorrection) X(qlP) X(qlM) X(qlD) X(fourthA) X(fourthB)

template <class R>
struct Rates {
#define VFB_FIELD(name) R name;
    VFB_K17_TERM_RATES(VFB_FIELD)
#undef VFB_FIELD
};

inline Rates<float> makeRates(float omega, float qlP, float qlM, float qlD)
{
    using R = float;
    Rates<R> r;
    r.omega = omega;
    r.minusOmega = -omega;
    r.OxyyPxzz = R(8) * (-R(2) + omega) * (R(1) + R(2) * omega) / (-R(8) - R(14) * omega + R(7) * omega * omega);
    r.OxyyMxzz = R(8) * (-R(2) + omega) * (-R(7) + R(4) * omega) / (R(56) - R(50) * omega + R(9) * omega * omega);
    r.Oxyz = R(24) * (-R(2) + omega) * (-R(2) - R(7) * omega + R(3) * omega * omega) /
             (R(48) + R(152) * omega - R(130) * omega * omega + R(29) * omega * omega * omega);
    r.oneMinusOxyyPxzz = R(1) - r.OxyyPxzz;
    r.oneMinusOxyyMxzz = R(1) - r.OxyyMxzz;
    r.oneMinusOxyz = R(1) - r.Oxyz;
    const R factorA = (R(4) + R(2) * omega - R(3) * omega * omega) / (R(2) - R(7) * omega + R(5) * omega * omega);
    const R factorB = (R(4) + R(28) * omega - R(14) * omega * omega) / (R(6) - R(21) * omega + R(15) * omega * omega);
    const R minusTau = -R(1) * (R(1) / omega - cst<R>(1, 2));
    const R minusThreeOmega = -R(3) * omega;
    r.halfMinusOmega = cst<R>(1, 2) * (-omega);
    r.omegaThreeHalves = omega * (cst<R>(3, 2));
    r.secondOrderCorrection = R(3) * (R(1) + cst<R>(1, 2) * (-omega));
    r.qlP = qlP;
    r.qlM = qlM;
    r.qlD = qlD;
    r.fourthA = minusTau * cst<R>(2, 3) * factorA;
    r.fourthB = minusTau * minusThreeOmega * cst<R>(1, 3) * factorB;
    return r;
}

// Central-moment transforms of ChimeraTransformation.h:58-121 (Geier et al.
// 2015, appendix J), written in multiply-add form.  With the conditioning pair
// (Kinverse, K) of a line and Kq = Kinverse * K:
//   forward   a' = a + b + c
//             b' = Kq (m1 - vv m0) - K vv,      m1 = c - a, m2 = a + c, m0 = a'
//             c' = Kq (m2 - 2 vv m1 + v2 m0) + K v2
//   backward  a' = c/2 + b (vv - 1/2) + (a + K) (v2 - vv)/2
//             b' = (a - c) - 2 vv b - v2 (a + K)
//             c' = c/2 + b (vv + 1/2) + (a + K) (v2 + vv)/2
// which are the reference's expressions with the factors Kinverse and K
// multiplied out (every line has Kq = 1 except the last forward x line, whose
// pair (3, 1/9) gives Kq = 1/3; K = 0 gives the plain transforms).
template <class R>
struct Sweep {
    R vv, v2, nvv, n2vv, hm, vvm;
    __device__ __forceinline__ Sweep(R v)
    {
        vv = v;
        v2 = v * v;
        nvv = -v;
        n2vv = R(-2) * v;
        hm = R(0.5) * (v2 - v);
        vvm = v - R(0.5);
    }
};

template <class R>
__device__ __forceinline__ void fwd(R& a, R& b, R& c, const Sweep<R>& w, typename ScalarOf<R>::type K)
{
    const R m2 = a + c;
    const R m1 = c - a;
    const R m0 = m2 + b;
    const R m0K = K != 0 ? m0 + R(K) : m0;
    a = m0;
    b = fma(w.nvv, m0K, m1);
    c = fma(w.v2, m0K, fma(w.n2vv, m1, m2));
}

// the forward x line with (Kinverse, K) = (3, 1/9) of K17CompressibleNavierStokes.h:222
template <class R>
__device__ __forceinline__ void fwdThird(R& a, R& b, R& c, const Sweep<R>& w)
{
    const R m2 = a + c;
    const R m1 = c - a;
    const R m0 = m2 + b;
    a = m0;
    b = fma(cst<R>(1, 3), fma(w.nvv, m0, m1), w.nvv * (cst<R>(1, 9)));
    c = fma(cst<R>(1, 3), fma(w.v2, m0, fma(w.n2vv, m1, m2)), w.v2 * (cst<R>(1, 9)));
}

template <class R>
__device__ __forceinline__ void bwd(R& a, R& b, R& c, const Sweep<R>& w, typename ScalarOf<R>::type K)
{
    const R aK = K != 0 ? a + R(K) : a;
    const R hc = R(0.5) * c;
    const R na = fma(aK, w.hm, fma(b, w.vvm, hc));
    // (c' - a' = b + v (a + K), and the three populations sum to a)
    const R nc = na + fma(aK, w.vv, b);
    b = (a - na) - nc;
    a = na;
    c = nc;
}

// sixth-order correction term of K17CompressibleNavierStokes.h:320-330 / :489-500,
// regrouped as (A + B / rho) / rho: A collects the terms over rho, B those
// over rho^2 (the same terms, fused multiply-adds)
template <class R>
__device__ __forceinline__ R c222Term(R m111, R m200, R m020, R m002, R m022, R m202, R m220, R m011, R m101, R m110,
                                      R m211, R m121, R m112, R m120, R m102, R m210, R m012, R m201, R m021,
                                      R oneOverRho, R drho)
{
    const R s2 = m200 + m020 + m002;
    const R a1 = fma(m002, m220, fma(m020, m202, m200 * m022));
    const R a2 = fma(m110, m112, fma(m101, m121, m011 * m211));
    const R a3 = fma(m201, m021, fma(m210, m012, m120 * m102));
    R A = fma(R(-4), m111 * m111, -a1);
    A = fma(R(-4), a2, A);
    A = fma(R(-2), a3, A);
    A = fma(-cst<R>(1, 3), m022 + m202 + m220, A);
    A = fma(-cst<R>(1, 9), s2, A);
    const R q101 = m101 * m101, q011 = m011 * m011, q110 = m110 * m110;
    const R m200m020 = m200 * m020;
    const R b1 = fma(q110, m002, fma(q011, m200, q101 * m020));
    const R pairs = fma(m002, m020, fma(m002, m200, m200m020));
    const R inner = fma(cst<R>(1, 3), s2, fma(R(2), q101 + q011 + q110, pairs));
    R B = fma(R(2), m200m020 * m002, R(4) * b1);
    B = fma(R(16), (m110 * m101) * m011, B);
    B = fma(cst<R>(2, 3), inner, B);
    B = fma(cst<R>(1, 27), fma(drho, drho, -drho), B);
    return fma(B, oneOverRho, A) * oneOverRho;
}

template <class R>
__device__ __forceinline__ R limiterQuotient(R x, R y);
template <>
__device__ __forceinline__ float limiterQuotient<float>(float x, float y)
{
    return __fdividef(x, y);
}

// Central moments to populations: the backward transform in x, then y, then z
// (K17CompressibleNavierStokes.h:525-557)
template <class R>
__device__ __forceinline__ void momentsToPopulations(R* f, R vvx, R vvy, R vvz)
{
    {
        const Sweep<R> w(vvx);
        bwd(f[dMMM], f[d0MM], f[dPMM], w, typename ScalarOf<R>::type(1));
        bwd(f[dM0M], f[d00M], f[dP0M], w, typename ScalarOf<R>::type(0));
        bwd(f[dMPM], f[d0PM], f[dPPM], w, cst<typename ScalarOf<R>::type>(1, 3));
        bwd(f[dMM0], f[d0M0], f[dPM0], w, typename ScalarOf<R>::type(0));
        bwd(f[dM00], f[d000], f[dP00], w, typename ScalarOf<R>::type(0));
        bwd(f[dMP0], f[d0P0], f[dPP0], w, typename ScalarOf<R>::type(0));
        bwd(f[dMMP], f[d0MP], f[dPMP], w, cst<typename ScalarOf<R>::type>(1, 3));
        bwd(f[dM0P], f[d00P], f[dP0P], w, typename ScalarOf<R>::type(0));
        bwd(f[dMPP], f[d0PP], f[dPPP], w, cst<typename ScalarOf<R>::type>(1, 9));
    }
    {
        const Sweep<R> w(vvy);
        bwd(f[dMMM], f[dM0M], f[dMPM], w, cst<typename ScalarOf<R>::type>(1, 6));
        bwd(f[dMM0], f[dM00], f[dMP0], w, typename ScalarOf<R>::type(0));
        bwd(f[dMMP], f[dM0P], f[dMPP], w, cst<typename ScalarOf<R>::type>(1, 18));
        bwd(f[d0MM], f[d00M], f[d0PM], w, cst<typename ScalarOf<R>::type>(2, 3));
        bwd(f[d0M0], f[d000], f[d0P0], w, typename ScalarOf<R>::type(0));
        bwd(f[d0MP], f[d00P], f[d0PP], w, cst<typename ScalarOf<R>::type>(2, 9));
        bwd(f[dPMM], f[dP0M], f[dPPM], w, cst<typename ScalarOf<R>::type>(1, 6));
        bwd(f[dPM0], f[dP00], f[dPP0], w, typename ScalarOf<R>::type(0));
        bwd(f[dPMP], f[dP0P], f[dPPP], w, cst<typename ScalarOf<R>::type>(1, 18));
    }
    {
        const Sweep<R> w(vvz);
        bwd(f[dMMM], f[dMM0], f[dMMP], w, cst<typename ScalarOf<R>::type>(1, 36));
        bwd(f[dM0M], f[dM00], f[dM0P], w, cst<typename ScalarOf<R>::type>(1, 9));
        bwd(f[dMPM], f[dMP0], f[dMPP], w, cst<typename ScalarOf<R>::type>(1, 36));
        bwd(f[d0MM], f[d0M0], f[d0MP], w, cst<typename ScalarOf<R>::type>(1, 9));
        bwd(f[d00M], f[d000], f[d00P], w, cst<typename ScalarOf<R>::type>(4, 9));
        bwd(f[d0PM], f[d0P0], f[d0PP], w, cst<typename ScalarOf<R>::type>(1, 9));
        bwd(f[dPMM], f[dPM0], f[dPMP], w, cst<typename ScalarOf<R>::type>(1, 36));
        bwd(f[dP0M], f[dP00], f[dP0P], w, cst<typename ScalarOf<R>::type>(1, 9));
        bwd(f[dPPM], f[dPP0], f[dPPP], w, cst<typename ScalarOf<R>::type>(1, 36));
    }
}

// One K17 collision on f[27] (pre-collision in, post-collision out).  (fx, fy, fz)
// is half the acceleration already scaled by the level factor
// (RunCollision.cuh:111-113).  Returns drho and the force-shifted velocity.
template <class R>
__device__ __forceinline__ void k17Collide(R* f, const Rates<R>& r, R fx, R fy, R fz, R& drho_out,
                                                    R& vx_out, R& vy_out, R& vz_out)
{
    // sums over the nine z lines (x, y fixed): s = a + b + c, m2 = a + c, d = c - a
#define VFB_ZLINE(XY, A, B, C)                                                                                         \
    const R m2_##XY = f[A] + f[C];                                                                                     \
    const R d_##XY = f[C] - f[A];                                                                                      \
    const R s_##XY = m2_##XY + f[B];
    VFB_ZLINE(MM, dMMM, dMM0, dMMP)
    VFB_ZLINE(M0, dM0M, dM00, dM0P)
    VFB_ZLINE(MP, dMPM, dMP0, dMPP)
    VFB_ZLINE(0M, d0MM, d0M0, d0MP)
    VFB_ZLINE(00, d00M, d000, d00P)
    VFB_ZLINE(0P, d0PM, d0P0, d0PP)
    VFB_ZLINE(PM, dPMM, dPM0, dPMP)
    VFB_ZLINE(P0, dP0M, dP00, dP0P)
    VFB_ZLINE(PP, dPPM, dPP0, dPPP)
#undef VFB_ZLINE
    const R drho = (((s_MM + s_PP) + (s_MP + s_PM)) + ((s_M0 + s_P0) + (s_0M + s_0P))) + s_00;
    const R jx = ((s_PM + s_PP) - (s_MM + s_MP)) + (s_P0 - s_M0);
    const R jy = ((s_MP + s_PP) - (s_MM + s_PM)) + (s_0P - s_0M);
    const R jz = (((d_MM + d_PP) + (d_MP + d_PM)) + ((d_M0 + d_P0) + (d_0M + d_0P))) + d_00;
    const R oneOverRho = R(1) / (drho + R(1));
    const R vvx = fma(jx, oneOverRho, fx);
    const R vvy = fma(jy, oneOverRho, fy);
    const R vvz = fma(jz, oneOverRho, fz);
    const R vx2 = vvx * vvx, vy2 = vvy * vvy, vz2 = vvz * vvz;

    // forward chimera in z (:190-199) from the line sums
    {
        const Sweep<R> w(vvz);
#define VFB_ZFWD(XY, A, B, C, K)                                                                                       \
    {                                                                                                                  \
        const R m0K = s_##XY + (K);                                                                                    \
        f[A] = s_##XY;                                                                                                 \
        f[B] = fma(w.nvv, m0K, d_##XY);                                                                                \
        f[C] = fma(w.v2, m0K, fma(w.n2vv, d_##XY, m2_##XY));                                                           \
    }
        VFB_ZFWD(MM, dMMM, dMM0, dMMP, cst<R>(1, 36))
        VFB_ZFWD(M0, dM0M, dM00, dM0P, cst<R>(1, 9))
        VFB_ZFWD(MP, dMPM, dMP0, dMPP, cst<R>(1, 36))
        VFB_ZFWD(0M, d0MM, d0M0, d0MP, cst<R>(1, 9))
        VFB_ZFWD(00, d00M, d000, d00P, cst<R>(4, 9))
        VFB_ZFWD(0P, d0PM, d0P0, d0PP, cst<R>(1, 9))
        VFB_ZFWD(PM, dPMM, dPM0, dPMP, cst<R>(1, 36))
        VFB_ZFWD(P0, dP0M, dP00, dP0P, cst<R>(1, 9))
        VFB_ZFWD(PP, dPPM, dPP0, dPPP, cst<R>(1, 36))
#undef VFB_ZFWD
    }
    // y (:202-210)
    {
        const Sweep<R> w(vvy);
        fwd(f[dMMM], f[dM0M], f[dMPM], w, cst<typename ScalarOf<R>::type>(1, 6));
        fwd(f[dMM0], f[dM00], f[dMP0], w, typename ScalarOf<R>::type(0));
        fwd(f[dMMP], f[dM0P], f[dMPP], w, cst<typename ScalarOf<R>::type>(1, 18));
        fwd(f[d0MM], f[d00M], f[d0PM], w, cst<typename ScalarOf<R>::type>(2, 3));
        fwd(f[d0M0], f[d000], f[d0P0], w, typename ScalarOf<R>::type(0));
        fwd(f[d0MP], f[d00P], f[d0PP], w, cst<typename ScalarOf<R>::type>(2, 9));
        fwd(f[dPMM], f[dP0M], f[dPPM], w, cst<typename ScalarOf<R>::type>(1, 6));
        fwd(f[dPM0], f[dP00], f[dPP0], w, typename ScalarOf<R>::type(0));
        fwd(f[dPMP], f[dP0P], f[dPPP], w, cst<typename ScalarOf<R>::type>(1, 18));
    }
    // x (:213-222)
    {
        const Sweep<R> w(vvx);
        fwd(f[dMMM], f[d0MM], f[dPMM], w, typename ScalarOf<R>::type(1));
        fwd(f[dM0M], f[d00M], f[dP0M], w, typename ScalarOf<R>::type(0));
        fwd(f[dMPM], f[d0PM], f[dPPM], w, cst<typename ScalarOf<R>::type>(1, 3));
        fwd(f[dMM0], f[d0M0], f[dPM0], w, typename ScalarOf<R>::type(0));
        fwd(f[dM00], f[d000], f[dP00], w, typename ScalarOf<R>::type(0));
        fwd(f[dMP0], f[d0P0], f[dPP0], w, typename ScalarOf<R>::type(0));
        fwd(f[dMMP], f[d0MP], f[dPMP], w, cst<typename ScalarOf<R>::type>(1, 3));
        fwd(f[dM0P], f[d00P], f[dP0P], w, typename ScalarOf<R>::type(0));
        fwdThird(f[dMPP], f[d0PP], f[dPPP], w);
    }

    // moment names: m_abc is stored in the slot of direction (a-1, b-1, c-1)
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

    // second and third order combinations (:329-346)
    R mxxPyyPzz = m200 + m020 + m002;
    R mxxMyy = m200 - m020;
    R mxxMzz = m200 - m002;
    R mxxyPyzz = m210 + m012;
    R mxxyMyzz = m210 - m012;
    R mxxzPyyz = m201 + m021;
    R mxxzMyyz = m201 - m021;
    R mxyyPxzz = m120 + m102;
    R mxyyMxzz = m120 - m102;

    // velocity gradients (:357-362), OxxPyyPzz = 1; the mixed ones (from the
    // second-order moments before relaxation) enter only the fourth-order
    // terms, through fourthB
    const R cm112 = r.fourthB * m110;
    const R cm121 = r.fourthB * m101;
    const R cm211 = r.fourthB * m011;
    const R dxux = r.halfMinusOmega * (mxxMyy + mxxMzz) + R(0.5) * (m000 - mxxPyyPzz);
    const R dyuy = dxux + r.omegaThreeHalves * mxxMyy;
    const R dzuz = dxux + r.omegaThreeHalves * mxxMzz;

    // second order relaxation with correction (:387-389)
    mxxPyyPzz += (m000 - mxxPyyPzz) - R(1.5) * (vx2 * dxux + vy2 * dyuy + vz2 * dzuz);
    mxxMyy += r.minusOmega * mxxMyy - r.secondOrderCorrection * (vx2 * dxux - vy2 * dyuy);
    mxxMzz += r.minusOmega * mxxMzz - r.secondOrderCorrection * (vx2 * dxux - vz2 * dzuz);
    m011 = fma(r.minusOmega, m011, m011);
    m101 = fma(r.minusOmega, m101, m101);
    m110 = fma(r.minusOmega, m110, m110);

    // third order with quartic limiter (:404-417); x - w x rounded once (as a
    // rounded product subtracted from x it stores other codes)
    R w;
    w = fma(r.oneMinusOxyz, limiterQuotient(fabs(m111), fabs(m111) + r.qlD), r.Oxyz);
    m111 = fma(-w, m111, m111);
    w = fma(r.oneMinusOxyyPxzz, limiterQuotient(fabs(mxxyPyzz), fabs(mxxyPyzz) + r.qlP), r.OxyyPxzz);
    mxxyPyzz = fma(-w, mxxyPyzz, mxxyPyzz);
    w = fma(r.oneMinusOxyyMxzz, limiterQuotient(fabs(mxxyMyzz), fabs(mxxyMyzz) + r.qlM), r.OxyyMxzz);
    mxxyMyzz = fma(-w, mxxyMyzz, mxxyMyzz);
    w = fma(r.oneMinusOxyyPxzz, limiterQuotient(fabs(mxxzPyyz), fabs(mxxzPyyz) + r.qlP), r.OxyyPxzz);
    mxxzPyyz = fma(-w, mxxzPyyz, mxxzPyyz);
    w = fma(r.oneMinusOxyyMxzz, limiterQuotient(fabs(mxxzMyyz), fabs(mxxzMyyz) + r.qlM), r.OxyyMxzz);
    mxxzMyyz = fma(-w, mxxzMyyz, mxxzMyyz);
    w = fma(r.oneMinusOxyyPxzz, limiterQuotient(fabs(mxyyPxzz), fabs(mxyyPxzz) + r.qlP), r.OxyyPxzz);
    mxyyPxzz = fma(-w, mxyyPxzz, mxyyPxzz);
    w = fma(r.oneMinusOxyyMxzz, limiterQuotient(fabs(mxyyMxzz), fabs(mxyyMxzz) + r.qlM), r.OxyyMxzz);
    mxyyMxzz = fma(-w, mxyyMxzz, mxyyMxzz);

    // back to single moments (:431-441)
    // (1/3)(-2 a + b + c) = (1/3)(a + b + c) - a, likewise for m002
    m200 = cst<R>(1, 3) * (mxxMyy + mxxMzz + mxxPyyPzz);
    m020 = m200 - mxxMyy;
    m002 = m200 - mxxMzz;
    m210 = (mxxyMyzz + mxxyPyzz) * R(0.5);
    m012 = (-mxxyMyzz + mxxyPyzz) * R(0.5);
    m201 = (mxxzMyyz + mxxzPyyz) * R(0.5);
    m021 = (-mxxzMyyz + mxxzPyyz) * R(0.5);
    m120 = (mxyyMxzz + mxyyPxzz) * R(0.5);
    m102 = (-mxyyMxzz + mxyyPxzz) * R(0.5);

    // fourth order to the modified equilibrium (:452-457); orders 5 and 6
    // relax to zero (:463-471)
    const R cm022 = r.fourthA * (dyuy + dzuz);
    const R cm202 = r.fourthA * (dxux + dzuz);
    const R cm220 = r.fourthA * (dyuy + dxux);

    // cumulants back to central moments (:478-505)
    // (the reference's (1/3) X / rho and (9 P + 3 S) / (9 rho) - drho / (9 rho)
    // regrouped as X (1/(3 rho)) and P / rho + S / (3 rho) - drho / (9 rho))
    const R oor3 = oneOverRho * cst<R>(1, 3);
    const R dr9 = drho * oneOverRho * cst<R>(1, 9);
    m211 = fma(fma(fma(R(3), m200, R(1)), m011, R(6) * (m110 * m101)), oor3, cm211);
    m121 = fma(fma(fma(R(3), m020, R(1)), m101, R(6) * (m110 * m011)), oor3, cm121);
    m112 = fma(fma(fma(R(3), m002, R(1)), m110, R(6) * (m101 * m011)), oor3, cm112);
    m220 = fma(fma(m200, m020, R(2) * (m110 * m110)), oneOverRho, fma(m200 + m020, oor3, cm220 - dr9));
    m202 = fma(fma(m200, m002, R(2) * (m101 * m101)), oneOverRho, fma(m200 + m002, oor3, cm202 - dr9));
    m022 = fma(fma(m002, m020, R(2) * (m011 * m011)), oneOverRho, fma(m002 + m020, oor3, cm022 - dr9));
    m122 = fma(fma(m002, m120, fma(m020, m102, fma(R(4) * m011, m111, R(2) * fma(m101, m021, m110 * m012)))),
               oneOverRho, (m120 + m102) * oor3);
    m212 = fma(fma(m002, m210, fma(m200, m012, fma(R(4) * m101, m111, R(2) * fma(m011, m201, m110 * m102)))),
               oneOverRho, (m210 + m012) * oor3);
    m221 = fma(fma(m200, m021, fma(m020, m201, fma(R(4) * m110, m111, R(2) * fma(m101, m120, m011 * m210)))),
               oneOverRho, (m021 + m201) * oor3);
    m222 = -c222Term(m111, m200, m020, m002, m022, m202, m220, m011, m101, m110, m211, m121, m112, m120, m102, m210,
                     m012, m201, m021, oneOverRho, drho);

    // first moments change sign (force, :512-514)
    m100 = -m100;
    m010 = -m010;
    m001 = -m001;

    // backward chimera, x then y then z (:525-557)
    momentsToPopulations(f, vvx, vvy, vvz);

    drho_out = drho;
    vx_out = vvx;
    vy_out = vvy;
    vz_out = vvz;
}
} // namespace termwise

// the K17 operator of a storage: Rates<R>, make(omega, qlP, qlM, qlD) and
// collide(f, rates, fx, fy, fz, drho, vx, vy, vz, forced)
template <class S, bool TERMWISE = sizeof(S) == 2>
struct K17Of {
    template <class R>
    using Rates = K17Rates<R>;
    template <class R>
    static Rates<R> make(R omega, R qlP, R qlM, R qlD)
    {
        return makeK17Rates<R>(omega, qlP, qlM, qlD);
    }
    template <class R>
    __device__ __forceinline__ static void collide(R* f, const Rates<R>& r, R fx, R fy, R fz, R& drho, R& vx, R& vy,
                                                   R& vz, bool forced)
    {
        k17Collide<R>(f, r, fx, fy, fz, drho, vx, vy, vz, forced);
    }
};
template <class S>
struct K17Of<S, true> {
    template <class R>
    using Rates = termwise::Rates<R>;
    template <class R>
    static Rates<R> make(R omega, R qlP, R qlM, R qlD)
    {
        return termwise::makeRates(omega, qlP, qlM, qlD);
    }
    template <class R>
    __device__ __forceinline__ static void collide(R* f, const Rates<R>& r, R fx, R fy, R fz, R& drho, R& vx, R& vy,
                                                   R& vz, bool)
    {
        termwise::k17Collide<R>(f, r, fx, fy, fz, drho, vx, vy, vz);
    }
};
} // namespace vfb
