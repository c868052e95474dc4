// Device checks of the approximation behind the exact fast forms of
// exact_math.cuh.  rcp_near_rn starts from the hardware's estimate
// instruction, whose rounding the host cannot reproduce, so its contract is
// checked on the device: exhaustively over its range of float bit patterns
// (which 1), and through the Markstein quotient on seeded pseudo-random
// operands (which 3).  hypot_fast starts from the estimate of the reciprocal
// square root: its root against the IEEE square root for every upper word (which
// 4), and its results, where it vouches for them, against hypot_ref (which 5).
// oflow_selftest_math returns the number of operands that break the contract.
#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "internal.hpp"

namespace oflow {
namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {  // splitmix64 finaliser
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// a float with a uniformly drawn exponent in [emin, emax], random mantissa and sign
__device__ __forceinline__ float draw(uint64_t h, int emin, int emax, bool sign) {
    const int e = emin + (int)((h >> 40) % (uint64_t)(emax - emin + 1));
    const uint32_t m = (uint32_t)h & 0x7fffffu;
    uint32_t bits = ((uint32_t)(e + 127) << 23) | m;
    if (sign && (h >> 63)) bits |= 0x80000000u;
    return __uint_as_float(bits);
}

__device__ __forceinline__ bool same_bits(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

// One thread's operands of which 4: upper word i (bits 0-20: mantissa and the
// exponent's parity, above them the exponent, from 2^-400 on), three lower words.
// The estimate's relative error is within 2^-20, and the root within `units` of its
// last place of the IEEE square root.
__device__ unsigned long long root_far(uint32_t i, uint64_t units) {
    unsigned long long bad = 0;
    for (int k = 0; k < 3; k++) {
        const uint32_t low = k == 0 ? 0u : k == 1 ? 0xffffffffu : (uint32_t)mix64(i);
        const uint32_t up = (uint32_t)(1023 - 400 + 2 * (int)(i >> 21)) * 0x100000u + (i & 0x1fffffu);
        const double s = __hiloint2double((int)up, (int)low);
        double y;
        const double r = hypot_root(s, y);
        const bool est = fabs(__fma_rn(-__dmul_rn(s, y), y, 1.0)) <= 0x1p-19;  // s y^2 = (1 + error)^2
        const long long d = __double_as_longlong(r) - __double_as_longlong(__dsqrt_rn(s));
        bad += !est || (uint64_t)(d < 0 ? -d : d) > units;
    }
    return bad;
}

// Operands of which 5, by the low bits of i: any two floats; two whose hypotenuse is
// the midpoint of two floats (a Pythagorean triple with an odd 25-bit hypotenuse), or
// a unit of one leg away; one next to a midpoint (a small leg beside a large one).
// Whether hypot_fast vouches for a result that is not hypot_ref's.  Roots below 2^-100
// are not its business.
__device__ bool hypot_off(uint32_t i, uint64_t seed) {
    const uint64_t h = mix64(seed ^ ((uint64_t)i << 1)), h2 = mix64(h);
    float a = draw(h, -90, 60, true), b = draw(h2, -140 + 27, 60, true);
    if ((i & 3) == 1) {
        const uint64_t m = 2900 + h % 2900, k = 1 + (h >> 24) % (m - 1);
        const int sc = (int)(h2 % 60) - 40;
        a = ldexpf((float)(m * m - k * k), sc);
        b = ldexpf((float)(2 * m * k), sc);
        if (h2 >> 63) a = __uint_as_float(__float_as_uint(a) + (uint32_t)((h2 >> 60) & 3) - 1);
    } else if ((i & 3) == 2) {
        a = draw(h, -40, 40, true);
        const float ulp = __uint_as_float(__float_as_uint(fabsf(a)) + 1) - fabsf(a);
        const float odd = (float)(2 * (int)((h2 >> 8) % 4) + 1);
        b = sqrtf(fabsf(a) * ulp * odd);  // the root is odd/2 units above a
        b = __uint_as_float(__float_as_uint(b) + (uint32_t)(h2 & 15) - 8);
    }
    const float ref = hypot_ref(a, b);
    unsigned near;
    const float r = hypot_fast(a, b, near);
    return ref >= 0x1p-100f && near > kHypotNear && !same_bits(r, ref);
}

__global__ void k_selftest(int which, uint32_t lo, uint32_t hi, uint64_t seed,
                           unsigned long long *count) {
    unsigned long long bad = 0;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = lo + blockIdx.x * blockDim.x + threadIdx.x; i < hi && i >= lo; i += stride) {
        if (which == 1) {  // rcp_near_rn is the correctly rounded reciprocal
            const float g = __uint_as_float(i);
            bad += !same_bits(rcp_near_rn(g), __frcp_rn(g));
        } else if (which == 4) {
            bad += root_far(i, seed ? seed - 1 : kHypotUnits);
        } else if (which == 5) {
            bad += hypot_off(i, seed);
        } else {  // Markstein quotient from rcp_near_rn equals IEEE division
            const uint64_t h = mix64(seed ^ ((uint64_t)i << 1)), h2 = mix64(h);
            const float g = (i & 1) ? draw(h, -40, 23, false) : 1.0f + draw(h, -20, 22, false);
            const float p = (i & 2) ? draw(h2, -99, 30, true) : draw(h2, -20, 20, true);
            if (rcp_in_range(g) && markstein_safe(p))
                bad += !same_bits(markstein(p, g, rcp_near_rn(g)), __fdiv_rn(p, g));
        }
    }
    for (int o = 16; o > 0; o >>= 1) bad += __shfl_down_sync(0xffffffffu, bad, o);
    if ((threadIdx.x & 31) == 0 && bad) atomicAdd(count, bad);
}

}  // namespace
}  // namespace oflow

extern "C" oflow_status oflow_selftest_math(int which, uint32_t lo, uint32_t hi,
                                            unsigned long long seed, unsigned long long *mismatches) {
    if (!mismatches || (which != 1 && which != 3 && which != 4 && which != 5) || hi < lo) return OFLOW_ERR_BAD_ARG;
    unsigned long long *d = nullptr;
    if (cudaMalloc(&d, sizeof(*d)) != cudaSuccess) {
        cudaGetLastError();
        return OFLOW_ERR_CUDA;
    }
    cudaError_t e = cudaMemset(d, 0, sizeof(*d));
    if (e == cudaSuccess) {
        oflow::k_selftest<<<oflow::kNumSMs * 8, 256>>>(which, lo, hi, seed, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(mismatches, d, sizeof(*d), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return OFLOW_ERR_CUDA;
    }
    return OFLOW_OK;
}
