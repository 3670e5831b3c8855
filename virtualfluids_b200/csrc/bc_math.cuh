// bc_math.cuh -- per-node formulas of the post-collision boundary conditions,
// shared by the BC kernels (bc.cu) and their adjoints (adjoint.cu) so that
// both run the same arithmetic.  Formulas: KernelUtilities.h:171-195 and the
// macroscopic sums of NoSlipInterpolatedCompressible.cu:144-160.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "collision_math.cuh"
#include "d3q27.cuh"

namespace vfb
{

// directions in the order the reference's BC kernels visit them
__host__ __device__ constexpr int qOrder(int j)
{
    constexpr int t[26] = { dP00, dM00, d0P0, d0M0, d00P, d00M, dPP0, dMM0, dPM0, dMP0, dP0P, dM0M, dP0M,
                            dM0P, d0PP, d0MM, d0PM, d0MP, dPPP, dMMM, dPPM, dMMP, dPMP, dMPM, dPMM, dMPP };
    return t[j];
}

template <class R>
struct BcLattice {
    unsigned long long N;
    const uint32_t* __restrict__ nX;
    const uint32_t* __restrict__ nY;
    const uint32_t* __restrict__ nZ;
    R omega;
};

// drho and velocity from post-collision populations (g[d] moves in direction
// d): the sums of NoSlipInterpolatedCompressible.cu:144-160 as trees, since a
// short list's launch lasts as long as one entry's dependent chain
template <class R>
__device__ __forceinline__ void bcMacros(const R* g, R& drho, R& vx1, R& vx2, R& vx3)
{
    drho = pyramidDensity(g);
    const R oneOverRho = reciprocal(R(1) + drho);
    vx1 = pyramidJx(g) * oneOverRho;
    vx2 = pyramidJy(g) * oneOverRho;
    vx3 = pyramidJz(g) * oneOverRho;
}

// KernelUtilities.h:171-174
template <class R>
__device__ __forceinline__ R feqBC(R drho, R vel, R cuSq, R w)
{
    return w * (drho + R(9) / R(2) * vel * vel * (R(1) + drho) - cuSq);
}

// The relaxation of the interpolated links: 2 omega and 1 / (1 - omega)
template <class R>
struct LinkRates {
    R twoOmega, inverse;
    __device__ __forceinline__ explicit LinkRates(R omega) : twoOmega(R(2) * omega), inverse(R(1) / (R(1) - omega)) {}
};

// KernelUtilities.h:176-195: the interpolated bounce-back of a link with wall
// distance q, over the common denominator 1 + q (one reciprocal a link, by
// Newton-Raphson steps, where the formula as written has three divisions; those
// were most of an FP64 list's time, and the chain that a short list waits for):
//   [ (1 - q) / 2 (f - finv + (f + finv - 2 omega feq) / (1 - omega)) + q (f + finv) - moving ] / (1 + q)
// moving: 6 w c.u of a moving wall, 0 of one at rest
template <class R>
__device__ __forceinline__ R interpolatedLink(R q, R f, R finv, R feq, const LinkRates<R>& r, R moving)
{
    const R s = f + finv;
    const R t = fma(fma(-r.twoOmega, feq, s), r.inverse, f - finv);
    return fma(fma(R(-0.5), q, R(0.5)), t, fma(q, s, -moving)) * reciprocal(R(1) + q);
}

template <class R>
__device__ __forceinline__ R interpNoSlip(R q, R f, R finv, R feq, const LinkRates<R>& r)
{
    return interpolatedLink(q, f, finv, feq, r, R(0));
}

template <class R>
__device__ __forceinline__ R interpVelocity(R q, R f, R finv, R feq, const LinkRates<R>& r, R vel, R w)
{
    return interpolatedLink(q, f, finv, feq, r, R(6) * w * vel);
}

// KernelUtilities.h:199-206 (the interpolated no-slip value minus w drho)
template <class R>
__device__ __forceinline__ R interpNoSlipPressure(R q, R f, R finv, R feq, const LinkRates<R>& r, R drho, R w)
{
    return interpNoSlip(q, f, finv, feq, r) - w * drho;
}

// PressureNonEquilibriumCompressible.cu:75-309: populations f of the
// neighbour with their equilibrium moved from its density to 1 + drhoBC at the
// same velocity: f_d + w_d (drhoBC - drho) (1 + 3 c.u + 9/2 (c.u)^2 - 3/2 u^2),
// the reference's subtraction and addition of two equilibria in one term
template <class R>
__device__ __forceinline__ void pressureShift(R* f, R drhoBC)
{
    const R drho = pyramidDensity(f);
    const R oneOverRho = reciprocal(drho + R(1));
    const R vx1 = pyramidJx(f) * oneOverRho;
    const R vx2 = pyramidJy(f) * oneOverRho;
    const R vx3 = pyramidJz(f) * oneOverRho;
    const R keep = R(1) - R(3) / R(2) * (vx1 * vx1 + vx2 * vx2 + vx3 * vx3);
    const R delta = drhoBC - drho;
    f[d000] = fma(R(8) / R(27) * delta, keep, f[d000]);
#pragma unroll
    for (int d = 1; d < 27; ++d) {
        const R cu = cdot<R>(d, vx1, vx2, vx3);
        f[d] = fma(weight<R>(d) * delta, fma(fma(R(9) / R(2), cu, R(3)), cu, keep), f[d]);
    }
}

// The wall model's clip (iMEM.cuh:131-136): -3 F forceFactor formed in
// double (the reference's literal 3.0 promotes it), bounded by +-clip with
// the NaN-ignoring double min / max.
template <class R>
__device__ __forceinline__ R imemClip(R clip, R F, R forceFactor)
{
    const double t = -3.0 * (double)F * (double)forceFactor;
    return (R)(clip > -clip ? fmin((double)clip, fmax((double)-clip, t)) : fmax((double)clip, fmin((double)-clip, t)));
}

// one step of a temporal filter, eps v + (1 - eps) mean with the second
// product in double as the reference writes it (iMEM.cuh:78-90)
template <class R>
__device__ __forceinline__ R imemFilter(R eps, R v, R mean)
{
    return (R)((double)(eps * v) + (1.0 - (double)eps) * (double)mean);
}

// The iMEM wall model of one BC entry (iMEM.cuh:57-137, Asmuth et al. 2021):
// the filtered velocities at the sampling node (el, in/out) and at the wall
// node (wm, in/out), the friction velocity u* = kappa |u_el,t| / ln(z / z0)
// at z = samplingOffset + q, the wall shear stress u*^2 along the wall node's
// tangential velocity over the filtered one's magnitude, minus the tangential
// momentum the bounce-back exchanged with the wall at rest (mom), and the wall
// velocity -3 F forceFactor clipped to twice the filtered tangential velocity.
template <class R>
__device__ __forceinline__ void imemWallVelocity(const R n[3], R el[3], R wm[3], const R vw[3], R rho, R z, R z0,
                                                 R forceFactor, const R mom[3], R& uStar, R V[3])
{
    const R dEl = el[0] * n[0] + el[1] * n[1] + el[2] * n[2];
    R t[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        t[a] = el[a] - dEl * n[a];
    const R magEl = sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
    const R dWm = wm[0] * n[0] + wm[1] * n[1] + wm[2] * n[2];
    R tm[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        tm[a] = wm[a] - dWm * n[a];
    const R magWm = sqrt(tm[0] * tm[0] + tm[1] * tm[1] + tm[2] * tm[2]);
    const R dW = vw[0] * n[0] + vw[1] * n[1] + vw[2] * n[2];
    uStar = magEl * R(0.4) / log(z / z0);
    const R tauW = uStar * uStar;
    const R dM = mom[0] * n[0] + mom[1] * n[1] + mom[2] * n[2];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const R Fw = (tauW * R(1)) * ((vw[a] - dW * n[a]) / magWm);
        const R F = Fw - (mom[a] - dM * n[a]) / rho;
        V[a] = imemClip(R(2) * t[a], F, forceFactor);
    }
}

} // namespace vfb
