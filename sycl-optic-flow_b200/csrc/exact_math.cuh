// Exactly rounded single-precision helpers shared by host and device code.
// Each function returns bit-for-bit what the reference's x86 build computes
// for the same expression (IEEE single/double, no contraction), but with
// cheaper instruction sequences on the GPU.  They are compiled on the host as
// well, so tests can check them against the plain expressions on the CPU.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

namespace oflow {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ float __int_as_float_hd(int i) { return __int_as_float(i); }
__device__ __forceinline__ int __float_as_int_hd(float f) { return __float_as_int(f); }
#else
inline float __int_as_float_hd(int i) { float f; memcpy(&f, &i, 4); return f; }
inline int __float_as_int_hd(float f) { int i; memcpy(&i, &f, 4); return i; }
#endif

// Single-precision hypot exactly as glibc's hypotf: the squares are exact in
// double, one rounding for the sum, one for the square root, one to single.
// On the GPU this runs on the double-precision pipe (two conversions in, the
// IEEE double square root, one conversion out), which measured cheaper than
// a single-precision candidate with a residual test around the rounding
// midpoints.
__host__ __device__ __forceinline__ float hypot_ref(float a, float b) {
    const double da = a, db = b;
    return (float)sqrt(da * da + db * db);
}

#ifdef __CUDACC__
// hypot_ref for 1 + c*hypot without the IEEE square root: one third-order
// Householder step from the hardware estimate of the reciprocal square root
// (rsqrt.approx; its relative error is below 2^-20 on every upper word, the
// only one the unit reads, which leaves 2^-58 after the step) and Ziv's
// rounding test.  The double result r is within kHypotUnits units of its last
// place of the root (measured: within 1, on every upper word of the sums' exponents
// with three lower words each; oflow_selftest_math), so it rounds to single precision as hypot_ref does unless
// it lies that close to the midpoint of two neighbouring floats (one sum in
// 2^25).  `near` is the distance above the lower end of that interval, of the
// 29 bits below a float's last, modulo 2^32: the result stands if it is above
// kHypotNear.  2^-400 added to the sum keeps zero off the estimate's pole and
// is far below a unit of any other; a root below 2^-100 may round differently
// from hypot_ref's, which 1 + c*hypot does not show.  Infinities give NaN.
constexpr unsigned kHypotUnits = 8, kHypotNear = 2 * 8 * kHypotUnits;
__device__ __forceinline__ double hypot_root(double s, double &y) {  // of s; y: the estimate
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    const double h = __dmul_rn(s, y);
    const double e = __fma_rn(-h, y, 1.0);  // s y^2 = 1 - e
    return __fma_rn(__dmul_rn(h, e), __fma_rn(e, 0.375, 0.5), h);
}
__device__ __forceinline__ float hypot_fast(float a, float b, unsigned &near) {
    const double da = a, db = b;
    double y;
    const double r = hypot_root(__fma_rn(da, da, __fma_rn(db, db, 0x1p-400)), y);
    near = (unsigned)__double2loint(r) * 8u + (8u * kHypotUnits - 0x80000000u);
    return (float)r;
}
#endif

#ifdef __CUDA_ARCH__
#define OF_FMAF(a, b, c) __fmaf_rn(a, b, c)
#define OF_RCP(x) __frcp_rn(x)
#else
#define OF_FMAF(a, b, c) fmaf(a, b, c)
#define OF_RCP(x) (1.0f / (x))
#endif

// Hardware reciprocal estimate (PTX rcp.approx), refined below by one Newton
// step.  On the host the refined form is the plain correctly rounded
// reciprocal, which satisfies the same contract.
#ifdef __CUDACC__
__device__ __forceinline__ float rcp_est(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
#endif

// RN(1/g) for g in [kRcpLo, kRcpHi): the reciprocal estimate r, then one
// Newton step r + r(1 - g r) with the residual formed exactly by a fused
// multiply-add.  The device tests check every float of the range against the
// correctly rounded reciprocal; rcp_in_range says whether g lies in it.
constexpr float kRcpLo = 0x1p-40f, kRcpHi = 0x1p24f;
__host__ __device__ __forceinline__ bool rcp_in_range(float g) { return g >= kRcpLo && g < kRcpHi; }
__host__ __device__ __forceinline__ float rcp_near_rn(float g) {
#ifdef __CUDA_ARCH__
    const float r = rcp_est(g);
    const float e = __fmaf_rn(-g, r, 1.0f);
    return __fmaf_rn(r, e, r);
#else
    return 1.0f / g;
#endif
}

// p / g correctly rounded (IEEE division) from y = RN(1/g): q0 = RN(p*y),
// r = q0*g - p (exact by FMA), q = RN(q0 - r*y) (Markstein).  Valid while
// neither the quotient nor p underflows: |p| > 2^-100 with g < 2^24 keeps the
// quotient above 2^-124; and for p = +0 or -0 (the residual's sign is chosen
// so that the quotient keeps p's).  markstein_safe says so for p (it sends -0
// to the plain division, which agrees); other p take the plain division.
__host__ __device__ __forceinline__ float markstein(float p, float g, float y) {
    const float q0 = p * y;
    const float r = OF_FMAF(q0, g, -p);
    return OF_FMAF(-r, y, q0);
}

// p / g correctly rounded for every finite p but zeros, from y = RN(1/g) with g in
// [2^-40, 2^24): Newton's step for the reciprocal and Markstein's correction of the
// quotient, both in double, where neither p nor the quotient underflows.  That
// leaves 2^-52 of the quotient; two 24-bit numbers' quotient is a rounding midpoint
// of single precision (normal or not) or 2^-49 of itself away from any, so the last
// rounding is that of p / g.
__host__ __device__ __forceinline__ float div_in_double(float p, float g, float y) {
    const double G = g, P = p, Y0 = y;
    const double Y = fma(Y0, fma(-G, Y0, 1.0), Y0);
    const double q = P * Y;
    return (float)fma(fma(-q, G, P), Y, q);
}

// For a running minimum over numerators: every one is zero or above 2^-100 in
// magnitude exactly when the minimum of markstein_key is at least kMarksteinKey.
constexpr unsigned kMarksteinKey = 2u * 0x0d800000u;  // 2^-100
__host__ __device__ __forceinline__ unsigned markstein_key(float p) {
    return 2u * (unsigned)__float_as_int_hd(p) - 1u;
}

__host__ __device__ __forceinline__ bool markstein_safe(float p) {
    return fabsf(p) > 0x1p-100f || __float_as_int_hd(p) == 0;
}

__host__ __device__ __forceinline__ float div_by_rcp(float p, float g, float y) {
    if (markstein_safe(p)) return markstein(p, g, y);
    return p / g;
}

}  // namespace oflow
