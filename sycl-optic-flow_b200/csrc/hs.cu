// Horn-Schunck on B200: kernels and the batched plan.  Restates
// src/hs/cuda/flow.cu:112-208 and src/hs/cuda/kernels/*.cuh with the
// semantics those kernels are written for (bilinear clamp-to-edge warp and
// upscale, clamped derivative taps, every pixel written); the arithmetic
// contract is in common.cuh.
//
// Layout per pair b (N = w*h at the finest level, levels packed):
//   raw[b][2] staged frames, pyr_l[b][2] float pyramid (finest = nlevels-1),
//   D float2 planes (Ix, Iy) and (Iz, Ix^2+Iy^2+alpha) of all pairs, dU0/dU1[b]
//   float2 ping-pong increments, Ua/Ub[b] float2 flow (alternating per level),
//   out[2][b].
// All ping-pong parities are known on the host, so the schedule is static and
// captured into one CUDA graph.
//
// The Jacobi sweeps are temporally blocked: one launch runs up to K sweeps on
// a tile held in registers with a K-pixel halo; what is exact shrinks by one
// pixel per sweep, so after K sweeps the owned tile is exact (clamped
// neighbours at the image border are exact at every sweep).
#include <cudaTypedefs.h>

#include <cstring>
#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"
#include "hs.hpp"
#include "pairio.hpp"
#include "internal.hpp"
#include "ptx.cuh"
#include "tvl1.hpp"

namespace oflow {


// 2x2 box average (downscaleKernel.cuh:27-29), every output pixel written.
__global__ void k_hs_downscale(const float *__restrict__ src, size_t sstride, int w, int h,
                               float *dst, size_t dstride) {
    const int nw = w / 2, nh = h / 2;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= nw || y >= nh) return;
    const float *s = src + (size_t)blockIdx.z * sstride + (size_t)(2 * y) * w + 2 * x;
    dst[(size_t)blockIdx.z * dstride + (size_t)y * nw + x] = 0.25f * (s[0] + s[w] + s[1] + s[w + 1]);
}

__device__ __forceinline__ float hs_deriv5(float m2, float m1, float p1, float p2) {
    float t = m2;
    t -= m1 * 8.0f;
    t += p1 * 8.0f;
    t -= p2;
    t /= 12.0f;
    return t;
}

// Fused warp + derivatives (warpingKernel.cuh:28-44, derivativesKernel.cuh:
// 29-73).  The tile plus a 2-pixel halo is filled with values at clamped
// image coordinates, so a derivative tap at offset k reads the clamped
// neighbour directly.
constexpr int kDTW = 32, kDTH = 8;
__global__ void __launch_bounds__(kDTW *kDTH) k_hs_warp_deriv(
    const float *__restrict__ pyr, size_t lp, int w, int h, const float2 *__restrict__ U,
    size_t ustride, int zero_flow, float alpha, float2 *D, size_t plane, size_t dstride) {
    constexpr int RW = kDTW + 4, RH = kDTH + 4;
    __shared__ float s0[RH * RW], s1[RH * RW];
    const int b = blockIdx.z;
    const float *I0 = pyr + (size_t)(2 * b) * lp;
    const float *I1 = pyr + (size_t)(2 * b + 1) * lp;
    const float2 *Ub = U + (size_t)b * ustride;
    const int x0 = blockIdx.x * kDTW - 2, y0 = blockIdx.y * kDTH - 2;
    const int tid = threadIdx.y * kDTW + threadIdx.x;
    for (int i = tid; i < RW * RH; i += kDTW * kDTH) {
        const int cx = imin(imax(x0 + i % RW, 0), w - 1);
        const int cy = imin(imax(y0 + i / RW, 0), h - 1);
        const size_t p = (size_t)cy * w + cx;
        s0[i] = __ldg(I0 + p);
        const float2 u = zero_flow ? make_float2(0.f, 0.f) : Ub[p];
        s1[i] = bilinear_clamped(I1, w, h, (float)cx + u.x, (float)cy + u.y);
    }
    __syncthreads();
    const int x = blockIdx.x * kDTW + threadIdx.x, y = blockIdx.y * kDTH + threadIdx.y;
    if (x >= w || y >= h) return;
    const int c = (threadIdx.y + 2) * RW + threadIdx.x + 2;
    float t0 = hs_deriv5(s0[c - 2], s0[c - 1], s0[c + 1], s0[c + 2]);
    float t1 = hs_deriv5(s1[c - 2], s1[c - 1], s1[c + 1], s1[c + 2]);
    const float Ix = (t0 + t1) * 0.5f;
    const float Iz = s1[c] - s0[c];
    t0 = hs_deriv5(s0[c - 2 * RW], s0[c - RW], s0[c + RW], s0[c + 2 * RW]);
    t1 = hs_deriv5(s1[c - 2 * RW], s1[c - RW], s1[c + RW], s1[c + 2 * RW]);
    const float Iy = (t0 + t1) * 0.5f;
    const float den = Ix * Ix + Iy * Iy + alpha;
    const size_t q = (size_t)b * dstride + (size_t)y * w + x;
    D[q] = make_float2(Ix, Iy);
    D[plane + q] = make_float2(Iz, den);
}

// Jacobi tiles: the region is 64 pixels wide and V*NW high, a warp owns V rows
// and a lane two adjacent columns of them, with the increments and D in
// registers for all sweeps of the launch.  Left and right neighbours come by
// shuffle, upper and lower ones from the thread's own registers, and only the
// first and last row of a warp goes through shared memory.  A sweep is 33
// instructions a pixel (19 of them the arithmetic, two shuffles, two the
// division's guard) and issue-bound while it runs.  64 pairs of 320x240, 200
// sweeps: 3.73 ms with D and the increments in shared memory (seven accesses a
// pixel), 2.52 ms here with 48x48 tiles and 8 sweeps a launch; without the
// fetch of the next tile's data during the sweeps 3.1 ms, with border tests in
// every pixel of a border region 2.7 ms.
//
// The division by Ix^2+Iy^2+alpha is Markstein's correction from the
// reciprocal, formed once per launch.  What that takes for granted (numerators
// zero or above 2^-100, denominators in [2^-40, 2^24); or, for frames of 16 bits,
// above 2^-76 and in [2^24, 2^48)) is kept as a running
// minimum; a block that breaks it runs its tile again from the untouched input,
// CAREFUL: looking at each numerator.  Where a part of the frames stands still the
// increments fall off from what moves by about 1/4 a pixel, and there are such
// numerators in every sweep; so the tile's next launch is careful at once
// (HsJacobiArgs::hint) until a launch meets none.  64 pairs of 320x240 with one moving
// disc each, 200 sweeps: 12.4 ms without the hint and with IEEE divisions for all of
// a tile, 4.3 ms here, and 2.6 where everything moves.  (Looking at a warp's
// numerators once a sweep, before its quotients, needs no second run; it costs
// frames without any 15 %.)
template <int V_, int NW_, int K_> struct HsTile {
    static constexpr int V = V_, NW = NW_, K = K_, NT = 32 * NW;
    static constexpr int RW = 64, RH = V * NW, TW = RW - 2 * K, TH = RH - 2 * K;
};

template <int V> struct HsState {
    float2 a[V][2];           // increments
    float ix[V][2], iy[V][2], iz[V][2], den[V][2], rcp[V][2];
};

struct HsJacobiArgs {
    const float2 *D;
    size_t plane, dstride;    // elements between D's planes, between pairs
    const float2 *in;         // increments before (ignored when first), after
    float2 *out, *U;          // U: the flow, updated by the last launch
    size_t stride;
    int w, h, sweeps, first, last;
    int vec;                  // two neighbouring pixels are 16-byte aligned
    int tiles_x, tiles_y, tiles;  // tiles: of all pairs
    int tma;                  // the maps below describe the level
    int *hint;                // per tile: its last launch met a numerator or denominator out of range
    int *err;                 // set when a bounded wait gives up
    CUtensorMap m0, m1, mi;   // D's planes, the increments: (w, h, pair), 8-byte elements
};

// Where a region meets the image border (all but odd and the lanes' x are
// uniform over the warp).  The first image row is the first of a warp (the halo
// is whole warps), so it only replaces the row from the warp above.
struct HsEdge {
    bool left, right, odd;  // this lane's column 0 is the first, column 1 the last; column 0 is the last (odd widths)
    int bottom;             // the warp's row that is the last of the image (else out of its rows)
};

// Denominators whose reciprocal rcp_near_rn rounds correctly (the device tests check
// every float of the range), and the least key of a numerator whose quotient by one
// below den markstein forms: either way quotients stay above 2^-124.
constexpr float kHsDenHi = 0x1p48f;
constexpr unsigned kMarksteinKeyFar = 2u * 0x19800000u;  // 2^-76
__device__ __forceinline__ bool hs_den_in_range(float den) { return den >= kRcpLo && den < kHsDenHi; }
__device__ __forceinline__ unsigned hs_least_key(float den) {
    return den < kRcpHi ? kMarksteinKey : kMarksteinKeyFar;
}

// p / den: Markstein's correction where it holds, in double where p is too small
// for it, the IEEE division where den is out of range.
__device__ __forceinline__ float hs_quotient(float p, float den, float rcp) {
    float q = markstein(p, den, rcp);
    if (markstein_key(p) < hs_least_key(den) || !hs_den_in_range(den))
        q = hs_den_in_range(den) ? div_in_double(p, den, rcp) : p / den;
    return q;
}

// The largest of the thread's denominators.
template <int V> __device__ __forceinline__ float hs_den_most(const HsState<V> &s) {
    float m = s.den[0][0];
#pragma unroll
    for (int v = 0; v < V; v++) m = fmaxf(m, fmaxf(s.den[v][0], s.den[v][1]));
    return m;
}

// One sweep (solverKernel.cuh:41-153): neighbour mean of the increments
// (clamped at the image border), frac = (Ix*su + Iy*sv + Iz) / den and the
// update, in the reference's order.  above / below: the neighbouring warps'
// rows; broken: a denominator of the thread is out of range.  CAREFUL: a warp
// with a numerator out of range looks at each.
// EDGE: 0 the region lies inside the image; 1 it meets its top, left or (at an
// even width) right border; 2 any border.
template <typename T, int EDGE, bool CAREFUL>
__device__ __forceinline__ void hs_sweep(HsState<T::V> &s, float4 above, float4 below, const HsEdge &e,
                                         bool broken, unsigned &key) {
    constexpr int V = T::V;
    float2 dn[2] = {make_float2(above.x, above.y), make_float2(above.z, above.w)};  // y - 1, before the sweep
    float num[V][2];  // CAREFUL: the numerators
    unsigned now = ~0u;
#pragma unroll
    for (int v = 0; v < V; v++) {
        const float2 c0 = s.a[v][0], c1 = s.a[v][1];
        float2 l, r, m = c1;  // left of column 0, right of column 1, right of column 0
        l.x = __shfl_up_sync(0xffffffffu, c1.x, 1);
        l.y = __shfl_up_sync(0xffffffffu, c1.y, 1);
        r.x = __shfl_down_sync(0xffffffffu, c0.x, 1);
        r.y = __shfl_down_sync(0xffffffffu, c0.y, 1);
        float2 up0 = v + 1 < V ? s.a[v + 1 < V ? v + 1 : v][0] : make_float2(below.x, below.y);
        float2 up1 = v + 1 < V ? s.a[v + 1 < V ? v + 1 : v][1] : make_float2(below.z, below.w);
        if (EDGE) {
            if (e.left) l = c0;
            if (e.right) r = c1;
        }
        if (EDGE == 2) {
            if (e.odd) m = c0;
            if (e.bottom == v) {
                up0 = c0;
                up1 = c1;
            }
        }
        float p[2];
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const float2 al = c ? c0 : l, ar = c ? r : m, au = c ? up1 : up0, ad = dn[c];
            const float su = (al.x + ar.x + au.x + ad.x) * 0.25f;
            const float sv = (al.y + ar.y + au.y + ad.y) * 0.25f;
            p[c] = s.ix[v][c] * su + s.iy[v][c] * sv + s.iz[v][c];
            if (CAREFUL) {
                num[v][c] = p[c];
                s.a[v][c] = make_float2(su, sv);
            } else {
                const float frac = markstein(p[c], s.den[v][c], s.rcp[v][c]);
                s.a[v][c] = make_float2(su - s.ix[v][c] * frac, sv - s.iy[v][c] * frac);
            }
        }
        unsigned &least = CAREFUL ? now : key;
        least = umin(umin(least, markstein_key(p[0])), markstein_key(p[1]));
        dn[0] = c0;
        dn[1] = c1;
    }
    if (CAREFUL) {
        const bool look = __any_sync(0xffffffffu, broken || now < hs_least_key(hs_den_most(s)));
        key = umin(key, now);
#pragma unroll
        for (int v = 0; v < V; v++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const float2 m = s.a[v][c];
                float frac = markstein(num[v][c], s.den[v][c], s.rcp[v][c]);
                if (look) frac = hs_quotient(num[v][c], s.den[v][c], s.rcp[v][c]);
                s.a[v][c] = make_float2(m.x - s.ix[v][c] * frac, m.y - s.iy[v][c] * frac);
            }
    }
}

// Sweep j of a tile: the warps' first and last rows exchanged through
// alternating buffers (one barrier a sweep), then the sweep.
template <typename T, int EDGE, bool CAREFUL, typename F>
__device__ __forceinline__ void hs_step(HsState<T::V> &s, int j, float4 (*sRow)[2][T::NW][32], bool top,
                                        const HsEdge &e, bool broken, unsigned &key, F &&taken) {
    constexpr int V = T::V, NW = T::NW;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float4(*row)[NW][32] = sRow[j & 1];
    const float4 first = make_float4(s.a[0][0].x, s.a[0][0].y, s.a[0][1].x, s.a[0][1].y);
    row[0][wid][lane] = first;
    row[1][wid][lane] = make_float4(s.a[V - 1][0].x, s.a[V - 1][0].y, s.a[V - 1][1].x, s.a[V - 1][1].y);
    __syncthreads();
    if (j == 0) taken();
    float4 above = row[1][wid > 0 ? wid - 1 : 0][lane];
    const float4 below = row[0][wid + 1 < NW ? wid + 1 : wid][lane];
    if (EDGE && top) above = first;
    hs_sweep<T, EDGE, CAREFUL>(s, above, below, e, broken, key);
}

// Pair, region origin and the thread's first pixel of a tile.
struct HsAt {
    int b, ox, oy, x, y0;
};
template <typename T> __device__ __forceinline__ HsAt hs_at(const HsJacobiArgs &a, int tile) {
    HsAt t;
    const int row = tile / a.tiles_x;
    t.b = row / a.tiles_y;
    t.ox = (tile - row * a.tiles_x) * T::TW - T::K;
    t.oy = (row - t.b * a.tiles_y) * T::TH - T::K;
    t.x = t.ox + 2 * (threadIdx.x & 31);
    t.y0 = t.oy + (threadIdx.x >> 5) * T::V;
    return t;
}

// A tile's data in shared memory: D's planes and the increments of the region.
template <typename T> struct HsSmem {
    float2 d0[T::RH][T::RW], d1[T::RH][T::RW], in[T::RH][T::RW];
};

// Brings a tile's region into shared memory (zeros outside the level): by one
// thread's TMA boxes, completing on `bar`, or by every thread's cp.async of two
// pixels (one, where rows don't start on 16 bytes), waited for by wait_all.
template <typename T>
__device__ __forceinline__ void hs_fetch_tma(const HsJacobiArgs &a, int tile, HsSmem<T> &sm, uint32_t bar) {
    const HsAt t = hs_at<T>(a, tile);
    mbar_arrive_expect_tx(bar, (uint32_t)(T::RH * T::RW * 8) * (a.first ? 2u : 3u));
    tma_load_3d(smem_u32(&sm.d0), &a.m0, t.ox, t.oy, t.b, bar);
    tma_load_3d(smem_u32(&sm.d1), &a.m1, t.ox, t.oy, t.b, bar);
    if (!a.first) tma_load_3d(smem_u32(&sm.in), &a.mi, t.ox, t.oy, t.b, bar);
}
template <typename T>
__device__ __forceinline__ void hs_fetch(const HsJacobiArgs &a, int tile, HsSmem<T> &sm) {
    const HsAt t = hs_at<T>(a, tile);
    const float2 *D0 = a.D + (size_t)t.b * a.dstride, *D1 = D0 + a.plane, *In = a.in + (size_t)t.b * a.stride;
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int ry = threadIdx.x >> 5; ry < T::RH; ry += T::NW) {
        const int y = t.oy + ry;
        const bool iy = y >= 0 && y < a.h;
        if (a.vec) {
            const int rx = 2 * lane, x = t.ox + rx;
            const bool in = iy && x >= 0 && x < a.w;
            const size_t q = in ? (size_t)y * a.w + x : 0;
            cp_async16(smem_u32(&sm.d0[ry][rx]), D0 + q, in);
            cp_async16(smem_u32(&sm.d1[ry][rx]), D1 + q, in);
            if (!a.first) cp_async16(smem_u32(&sm.in[ry][rx]), In + q, in);
        } else {
#pragma unroll
            for (int rx = lane; rx < T::RW; rx += 32) {
                const int x = t.ox + rx;
                const bool in = iy && x >= 0 && x < a.w;
                const size_t q = in ? (size_t)y * a.w + x : 0;
                cp_async8(smem_u32(&sm.d0[ry][rx]), D0 + q, in);
                cp_async8(smem_u32(&sm.d1[ry][rx]), D1 + q, in);
                if (!a.first) cp_async8(smem_u32(&sm.in[ry][rx]), In + q, in);
            }
        }
    }
}

// Up to K sweeps of one tile whose data is in shared memory; once every thread
// has taken its share into registers, `taken` runs.  first: increments start at 0
// (flow.cu:168-171); last: add the increment to the flow (AddKernel,
// addKernel.cuh:28-36) instead of storing it.  Returns whether the guard broke
// (nothing is stored then, unless CAREFUL).
template <typename T, bool CAREFUL, typename F>
__device__ __forceinline__ bool hs_tile(const HsJacobiArgs &a, int tile, const HsSmem<T> &sm,
                                        float4 (*sRow)[2][T::NW][32], F &&taken) {
    constexpr int V = T::V, K = T::K, NW = T::NW, U = K < 8 ? K : 8;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, w = a.w, h = a.h;
    const HsAt t = hs_at<T>(a, tile);
    const int x = t.x, y0 = t.y0;
    HsState<V> s;
    unsigned key = ~0u;
    const bool in0 = x >= 0 && x < w, in1 = x + 1 >= 0 && x + 1 < w;
    bool broken = false;
#pragma unroll
    for (int v = 0; v < V; v++) {
        const bool iy = y0 + v >= 0 && y0 + v < h;
        const int r = wid * V + v;
        const float4 d0 = *reinterpret_cast<const float4 *>(&sm.d0[r][2 * lane]);
        const float4 d1 = *reinterpret_cast<const float4 *>(&sm.d1[r][2 * lane]);
        const float4 u = a.first ? make_float4(0.f, 0.f, 0.f, 0.f)
                                 : *reinterpret_cast<const float4 *>(&sm.in[r][2 * lane]);
        s.a[v][0] = make_float2(u.x, u.y);
        s.a[v][1] = make_float2(u.z, u.w);
        s.ix[v][0] = d0.x; s.iy[v][0] = d0.y; s.iz[v][0] = d1.x; s.den[v][0] = iy && in0 ? d1.y : 1.0f;
        s.ix[v][1] = d0.z; s.iy[v][1] = d0.w; s.iz[v][1] = d1.z; s.den[v][1] = iy && in1 ? d1.w : 1.0f;
    }
#pragma unroll
    for (int v = 0; v < V; v++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
            s.rcp[v][c] = rcp_near_rn(s.den[v][c]);
            broken |= !hs_den_in_range(s.den[v][c]);
        }
    const bool interior = t.ox >= 1 && t.oy >= 1 && t.ox + T::RW <= w - 1 && t.oy + T::RH <= h - 1;
    const HsEdge e{x == 0, x + 1 == w - 1, x == w - 1, h - 1 - y0};
    const bool top = y0 == 0;
    if (CAREFUL) {
#pragma unroll 1
        for (int j = 0; j < a.sweeps; j++) hs_step<T, 2, true>(s, j, sRow, top, e, broken, key, taken);
    } else if (a.sweeps != K) {
#pragma unroll 1
        for (int j = 0; j < a.sweeps; j++) hs_step<T, 2, false>(s, j, sRow, top, e, broken, key, taken);
    } else if (interior) {
        // unrolled, so that old and new increments swap registers instead of being copied
        // (64 pairs of 320x240, 200 sweeps: 2.61 ms, with 4 and 2 sweeps here and below 2.70)
#pragma unroll U
        for (int j = 0; j < K; j++) hs_step<T, 0, false>(s, j, sRow, top, e, broken, key, taken);
    } else if (t.oy + T::RH <= h - 1 && (w & 1) == 0) {
#pragma unroll U
        for (int j = 0; j < K; j++) hs_step<T, 1, false>(s, j, sRow, top, e, broken, key, taken);
    } else {
#pragma unroll 2
        for (int j = 0; j < K; j++) hs_step<T, 2, false>(s, j, sRow, top, e, broken, key, taken);
    }
    // (also: every warp has read the rows before the next tile writes them)
    const bool bad = __syncthreads_or(broken || key < hs_least_key(hs_den_most(s)));
    if (!CAREFUL && bad) return true;
    if (lane < K / 2 || lane >= 32 - K / 2 || wid < K / V || wid >= NW - K / V || x >= w) return bad;
    float2 *Out = (a.last ? a.U : a.out) + (size_t)t.b * a.stride;
#pragma unroll
    for (int v = 0; v < V; v++) {
        if (y0 + v >= h) break;
        const size_t q = (size_t)(y0 + v) * w + x;
        float2 r0 = s.a[v][0], r1 = s.a[v][1];
        if (a.last) {
            const float4 u = ld_two(Out, q, a.vec, true, in1);
            r0 = make_float2(u.x + r0.x, u.y + r0.y);
            r1 = make_float2(u.z + r1.x, u.w + r1.y);
        }
        if (a.vec) {
            *reinterpret_cast<float4 *>(Out + q) = make_float4(r0.x, r0.y, r1.x, r1.y);
        } else {
            Out[q] = r0;
            if (in1) Out[q + 1] = r1;
        }
    }
    return bad;
}

// Resident blocks walk the tiles of all pairs; a tile's data is brought to
// shared memory (TMA, where the level's strides allow it and there is a flag for
// its bounded wait) while the block's previous tile is in the registers.  Without
// TMA the copies take every thread's instructions: 48 pairs of 321x241, 104 sweeps,
// 1.55 ms (of 320x240 1.13); loading a tile between two barriers, with nothing else to
// run on the SM meanwhile, 2.55.
template <typename T, int MINB, bool TMA>
__global__ void __launch_bounds__(T::NT, MINB) k_hs_jacobi(const __grid_constant__ HsJacobiArgs a) {
    extern __shared__ __align__(128) char hs_dyn[];
    HsSmem<T> &sm = *reinterpret_cast<HsSmem<T> *>(hs_dyn);
    __shared__ float4 sRow[2][2][T::NW][32];
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ int s_hint;
    const uint32_t bar = smem_u32(&s_bar), hint = smem_u32(&s_hint);
    uint32_t parity = 0;
    if (threadIdx.x == 0) {
        if (TMA) {
            mbar_init(bar, 1);
            fence_mbar_init();
            hs_fetch_tma<T>(a, blockIdx.x, sm, bar);
        }
        cp_async4(hint, a.hint + blockIdx.x);
    }
    if (!TMA) hs_fetch<T>(a, blockIdx.x, sm);
    __syncthreads();  // the barrier is initialised before anyone waits on it
    for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
        const int next = tile + gridDim.x;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        if (TMA) {
            const bool ok = mbar_wait_bounded(bar, parity);
            parity ^= 1u;
            if (__syncthreads_or(!ok)) {
                // report, let the copies land (bounded), leave; the host drops
                // the plan's results
                if (threadIdx.x == 0) atomicExch(a.err, 1);
                mbar_wait_bounded(bar, parity ^ 1u);
                return;
            }
        } else {
            __syncthreads();
        }
        const bool careful = !a.first && s_hint != 0;  // (the first launch writes every tile's hint)
        const auto fetch_next = [&] {
            if (next >= a.tiles) return;
            if (!TMA) {
                hs_fetch<T>(a, next, sm);
            } else if (threadIdx.x == 0) {
                fence_async_smem();  // the block's reads of this tile, then the copies of the next
                hs_fetch_tma<T>(a, next, sm, bar);
            }
            if (threadIdx.x == 0) cp_async4(hint, a.hint + next);  // (nobody waits for it before the tile's data)
        };
        bool bad = careful;
        if (!careful && hs_tile<T, false>(a, tile, sm, sRow, fetch_next)) {
            bad = true;
            // again from the untouched input, then the next tile's copies again
            if (TMA && next < a.tiles) {
                const bool ok = mbar_wait_bounded(bar, parity);
                parity ^= 1u;
                if (__syncthreads_or(!ok)) {
                    if (threadIdx.x == 0) atomicExch(a.err, 1);
                    mbar_wait_bounded(bar, parity ^ 1u);
                    return;
                }
            }
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();
            hs_fetch<T>(a, tile, sm);
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();
        }
        if (bad) bad = hs_tile<T, true>(a, tile, sm, sRow, fetch_next);
        if (threadIdx.x == 0 && (a.first || bad != careful)) a.hint[tile] = bad;
    }
}

// All sweeps of a warp of a small level in one launch: a cluster of blocks holds a
// pair's level, a tile each, in the registers of k_hs_jacobi's sweeps.  Every K
// sweeps the blocks lay the pixels they own in shared memory, meet at the cluster's
// barrier and take their halos from the owners' (two buffers, so that one barrier
// is enough).  A launch per 8 sweeps waits for its own start and its tile's data:
// 152 sweeps of a level take (19 launches without the gaps between them, and here)
//   40x30 103 and 68 us, 80x60 102 and 70, 160x120 109 and 87; 9 pairs of 160x120
//   173 and 135, 16 pairs of 80x60 112 and 115, 37 pairs 176 and 178.
// One block an SM instead of two saves the spills (160x120 83 us) and costs batches
// more (9 pairs 166).  The barriers of the block and the cluster bound it.
//
// The guard is looked at once, at the end: where any block of the cluster broke it,
// all of them run the warp again, CAREFUL.  150 sweeps of 160x120 take 102 us, and
// 248 where a part of the frames stands still (start of one disc moving; 464 with an
// IEEE division in every pixel of the second run); 9 pairs 172 and 405 us.  Looking
// at the end of every exchange, and going on from there, takes 173 us where frames
// stand still, but 106 and 184 where they don't.
template <typename T> struct HsRes {
    float2 own[2][T::TH][T::TW];
};

// The thread's D, its reciprocals, and whether a denominator is out of range.
template <typename T>
__device__ __forceinline__ bool hs_res_load(const HsJacobiArgs &a, const HsAt &t, HsState<T::V> &s) {
    constexpr int V = T::V;
    const float2 *D0 = a.D + (size_t)t.b * a.dstride, *D1 = D0 + a.plane;
    const int x = t.x, y0 = t.y0, w = a.w, h = a.h;
    const bool in0 = x >= 0 && x < w, in1 = x + 1 >= 0 && x + 1 < w;
#pragma unroll
    for (int v = 0; v < V; v++) {
        const bool iy = y0 + v >= 0 && y0 + v < h;
        const size_t q = iy && in0 ? (size_t)(y0 + v) * w + x : 0;
        const float4 d0 = ld_two(D0, q, a.vec, iy && in0, iy && in0 && in1);
        const float4 d1 = ld_two(D1, q, a.vec, iy && in0, iy && in0 && in1);
        s.ix[v][0] = d0.x; s.iy[v][0] = d0.y; s.iz[v][0] = d1.x; s.den[v][0] = iy && in0 ? d1.y : 1.0f;
        s.ix[v][1] = d0.z; s.iy[v][1] = d0.w; s.iz[v][1] = d1.z; s.den[v][1] = iy && in0 && in1 ? d1.w : 1.0f;
    }
    bool broken = false;
#pragma unroll
    for (int v = 0; v < V; v++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
            s.rcp[v][c] = rcp_near_rn(s.den[v][c]);
            broken |= !hs_den_in_range(s.den[v][c]);
        }
    return broken;
}

// The increments that the blocks laid in buffer buf: a thread's own pixels, or its
// halo from the owners (zeros beyond an odd width are the owner's).
template <typename T>
__device__ __forceinline__ void hs_res_take(const HsJacobiArgs &a, const HsAt &t, const HsRes<T> &sm, int buf,
                                            HsState<T::V> &s) {
#pragma unroll
    for (int v = 0; v < T::V; v++) {
        const int x = t.x, y = t.y0 + v;
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
        if (x >= 0 && x < a.w && y >= 0 && y < a.h) {
            const int tx = x / T::TW, ty = y / T::TH;
            u = cluster_ld4(smem_u32(&sm.own[buf][y - ty * T::TH][x - tx * T::TW]), ty * a.tiles_x + tx);
        }
        s.a[v][0] = make_float2(u.x, u.y);
        s.a[v][1] = make_float2(u.z, u.w);
    }
}

// Lays the thread's pixels in buffer buf (zeros outside the level).
template <typename T>
__device__ __forceinline__ void hs_res_lay(const HsJacobiArgs &a, const HsAt &t, HsRes<T> &sm, int buf,
                                           HsState<T::V> &s) {
    constexpr int V = T::V, K = T::K;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int v = 0; v < V; v++) {
        const bool iy = t.y0 + v < a.h;
        if (!iy || t.x >= a.w) s.a[v][0] = make_float2(0.f, 0.f);
        if (!iy || t.x + 1 >= a.w) s.a[v][1] = make_float2(0.f, 0.f);
        *reinterpret_cast<float4 *>(&sm.own[buf][wid * V + v - K][2 * lane - K]) =
            make_float4(s.a[v][0].x, s.a[v][0].y, s.a[v][1].x, s.a[v][1].y);
    }
}

// Whether the thread's pixels are the block's own.
template <typename T> __device__ __forceinline__ bool hs_own() {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    return lane >= T::K / 2 && lane < 32 - T::K / 2 && wid >= T::K / T::V && wid < T::NW - T::K / T::V;
}

// All sweeps again, CAREFUL.  Returns the buffer that holds the last increments.
template <typename T>
__device__ __forceinline__ int hs_res_careful(const HsJacobiArgs &a, HsRes<T> &sm, float4 (*sRow)[2][T::NW][32]) {
    constexpr int K = T::K;
    const HsAt t = hs_at<T>(a, blockIdx.x);
    const HsEdge e{t.x == 0, t.x + 1 == a.w - 1, t.x == a.w - 1, a.h - 1 - t.y0};
    HsState<T::V> s;
    const bool broken = hs_res_load<T>(a, t, s);
#pragma unroll
    for (int v = 0; v < T::V; v++) s.a[v][0] = s.a[v][1] = make_float2(0.f, 0.f);
    unsigned key = ~0u;
    int buf = 0;
#pragma unroll 1
    for (int done = 0; done < a.sweeps; done += K, buf ^= 1) {
        if (done > 0) hs_res_take<T>(a, t, sm, buf ^ 1, s);
        const int n = imin(K, a.sweeps - done);
#pragma unroll 1
        for (int j = 0; j < n; j++) hs_step<T, 2, true>(s, j, sRow, t.y0 == 0, e, broken, key, [] {});
        if (hs_own<T>()) hs_res_lay<T>(a, t, sm, buf, s);
        cluster_barrier();
    }
    return buf ^ 1;
}

template <typename T>
__global__ void __launch_bounds__(T::NT, 2) k_hs_res(const __grid_constant__ HsJacobiArgs a) {
    constexpr int V = T::V, K = T::K, NW = T::NW;
    static_assert(K % V == 0 && K % 2 == 0, "owned pixels are whole threads");
    extern __shared__ __align__(128) char hs_dyn[];
    HsRes<T> &sm = *reinterpret_cast<HsRes<T> *>(hs_dyn);
    __shared__ float4 sRow[2][2][NW][32];
    const int w = a.w, h = a.h;
    const HsAt t = hs_at<T>(a, blockIdx.x);
    const int x = t.x, y0 = t.y0;
    const bool own = hs_own<T>();
    HsState<V> s;
    const bool broken = hs_res_load<T>(a, t, s);
    const bool interior = t.ox >= 1 && t.oy >= 1 && t.ox + T::RW <= w - 1 && t.oy + T::RH <= h - 1;
    const bool plain = t.oy + T::RH <= h - 1 && (w & 1) == 0;
    const HsEdge e{x == 0, x + 1 == w - 1, x == w - 1, h - 1 - y0};
    const bool top = y0 == 0;
    const auto taken = [] {};

    // whether a block of the cluster met anything out of range (told by the block itself
    // before the last meeting)
    __shared__ int s_bad;
    if (threadIdx.x == 0) s_bad = 0;
    unsigned key = ~0u;
#pragma unroll
    for (int v = 0; v < V; v++) s.a[v][0] = s.a[v][1] = make_float2(0.f, 0.f);
    int buf = 0;
#pragma unroll 1
    for (int done = 0;; done += K, buf ^= 1) {
        const int n = imin(K, a.sweeps - done);
        if (n != K) {
#pragma unroll 1
            for (int j = 0; j < n; j++) hs_step<T, 2, false>(s, j, sRow, top, e, broken, key, taken);
        } else if (interior) {
#pragma unroll 2
            for (int j = 0; j < K; j++) hs_step<T, 0, false>(s, j, sRow, top, e, broken, key, taken);
        } else if (plain) {
#pragma unroll 2
            for (int j = 0; j < K; j++) hs_step<T, 1, false>(s, j, sRow, top, e, broken, key, taken);
        } else {
#pragma unroll 2
            for (int j = 0; j < K; j++) hs_step<T, 2, false>(s, j, sRow, top, e, broken, key, taken);
        }
        if (done + K >= a.sweeps) break;
        if (own) hs_res_lay<T>(a, t, sm, buf, s);
        cluster_barrier();
        if (!own) hs_res_take<T>(a, t, sm, buf, s);
    }
    if (a.sweeps <= K) cluster_barrier();  // (every block runs before its memory is written)
    if (broken || key < hs_least_key(hs_den_most(s)))
        for (int k = 0; k < a.tiles_x * a.tiles_y; k++) cluster_st1(smem_u32(&s_bad), k, 1);
    cluster_barrier();
    const bool bad = s_bad != 0;
    if (bad) buf = hs_res_careful<T>(a, sm, sRow);
    if (bad && own) hs_res_take<T>(a, t, sm, buf, s);
    // (nobody reads another block's shared memory after the last meeting)
    if (!own || x >= w) return;
    const bool in1 = x + 1 < w;
    float2 *Out = (a.last ? a.U : a.out) + (size_t)t.b * a.stride;
#pragma unroll
    for (int v = 0; v < V; v++) {
        if (y0 + v >= h) break;
        const size_t q = (size_t)(y0 + v) * w + x;
        float2 r0 = s.a[v][0], r1 = s.a[v][1];
        if (a.last) {
            const float4 u = ld_two(Out, q, a.vec, true, in1);
            r0 = make_float2(u.x + r0.x, u.y + r0.y);
            r1 = make_float2(u.z + r1.x, u.w + r1.y);
        }
        if (a.vec) {
            *reinterpret_cast<float4 *>(Out + q) = make_float4(r0.x, r0.y, r1.x, r1.y);
        } else {
            Out[q] = r0;
            if (in1) Out[q + 1] = r1;
        }
    }
}

// Flow prolongation (upscaleKernel.cuh:26-40 as a filtering upscale):
// bilinear, clamp-to-edge, centre-aligned, component-wise scale.
__device__ __forceinline__ float2 bilinear2(const float2 *__restrict__ src, int w, int h,
                                            float xf, float yf) {
    xf = fminf(fmaxf(xf, -1.0f), (float)w);
    yf = fminf(fmaxf(yf, -1.0f), (float)h);
    const float x0f = floorf(xf), y0f = floorf(yf);
    const float fx = xf - x0f, fy = yf - y0f;
    const int x0 = (int)x0f, y0 = (int)y0f;
    const int xa = imin(imax(x0, 0), w - 1), xb = imin(imax(x0 + 1, 0), w - 1);
    const int ya = imin(imax(y0, 0), h - 1), yb = imin(imax(y0 + 1, 0), h - 1);
    const float2 v00 = src[(size_t)ya * w + xa], v10 = src[(size_t)ya * w + xb];
    const float2 v01 = src[(size_t)yb * w + xa], v11 = src[(size_t)yb * w + xb];
    const float gx = 1.0f - fx, gy = 1.0f - fy;
    float2 r;
    float top = gx * v00.x + fx * v10.x, bot = gx * v01.x + fx * v11.x;
    r.x = gy * top + fy * bot;
    top = gx * v00.y + fx * v10.y;
    bot = gx * v01.y + fx * v11.y;
    r.y = gy * top + fy * bot;
    return r;
}

// Two pixels of a row a thread; rx = w/nw and ry = h/nh come from the host
// (one IEEE division either way).
__global__ void k_upscale2(const float2 *__restrict__ src, size_t sstride, int w, int h,
                           float2 *dst, size_t dstride, int nw, int nh, float sx, float sy, float rx, float ry) {
    const int x = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= nw || y >= nh) return;
    const float2 *s = src + (size_t)blockIdx.z * sstride;
    float2 *d = dst + (size_t)blockIdx.z * dstride + (size_t)y * nw + x;
    const float fy = ((float)y + 0.5f) * ry - 0.5f;
    const float2 a = bilinear2(s, w, h, ((float)x + 0.5f) * rx - 0.5f, fy);
    const float2 ra = make_float2(a.x * sx, a.y * sy);
    if (x + 1 >= nw) {
        d[0] = ra;
        return;
    }
    const float2 b = bilinear2(s, w, h, ((float)(x + 1) + 0.5f) * rx - 0.5f, fy);
    const float2 rb = make_float2(b.x * sx, b.y * sy);
    if (reinterpret_cast<uintptr_t>(d) % 16 == 0) {
        *reinterpret_cast<float4 *>(d) = make_float4(ra.x, ra.y, rb.x, rb.y);
    } else {
        d[0] = ra;
        d[1] = rb;
    }
}

__global__ void k_split2(const float2 *__restrict__ U, size_t stride, int N, float *ou, float *ov,
                         int B) {
    const int b = blockIdx.y;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const float2 u = U[(size_t)b * stride + i];
        ou[(size_t)b * N + i] = u.x;  // ov already points at the v planes
        ov[(size_t)b * N + i] = u.y;
    }
}

void launch_upscale2(const float2 *src, size_t sstride, int w, int h, float2 *dst,
                     size_t dstride, int nw, int nh, float sx, float sy, int B,
                     cudaStream_t st) {
    dim3 blk(32, 8), g(div_up(nw, 64), div_up(nh, 8), B);
    k_upscale2<<<g, blk, 0, st>>>(src, sstride, w, h, dst, dstride, nw, nh, sx, sy, (float)w / (float)nw,
                                  (float)h / (float)nh);
}

// Each thread converts four consecutive pixels of a row; rows whose source and destination allow it move them as one vector.
constexpr int kTabPx = 4;
template <typename T>
__global__ void k_ingest_tab(const FrameRef *__restrict__ frames, int w, int h, float *dst,
                             size_t N) {
    const int x = (blockIdx.x * blockDim.x + threadIdx.x) * kTabPx;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const FrameRef f = frames[blockIdx.z];
    const T *src = static_cast<const T *>(f.p) + (size_t)y * f.pitch + x;
    float *d = dst + (size_t)blockIdx.z * N + (size_t)y * w + x;
    const bool vec = x + kTabPx <= w && reinterpret_cast<uintptr_t>(d) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(src) % (kTabPx * sizeof(T)) == 0;
    if (vec) {
        float4 v;
        if (sizeof(T) == 4) {
            v = __ldg(reinterpret_cast<const float4 *>(src));
        } else {
            const uchar4 c = __ldg(reinterpret_cast<const uchar4 *>(src));
            v = make_float4((float)c.x, (float)c.y, (float)c.z, (float)c.w);
        }
        *reinterpret_cast<float4 *>(d) = v;
        return;
    }
    for (int k = 0; k < kTabPx && x + k < w; k++) d[k] = (float)__ldg(src + k);
}

void launch_ingest_tab(const FrameRef *frames, int dtype, int w, int h, float *dst, size_t N,
                       int planes, cudaStream_t st) {
    dim3 blk(32, 8), g(div_up(w, 32 * kTabPx), div_up(h, 8), planes);
    if (dtype == OFLOW_U8)
        k_ingest_tab<uint8_t><<<g, blk, 0, st>>>(frames, w, h, dst, N);
    else
        k_ingest_tab<float><<<g, blk, 0, st>>>(frames, w, h, dst, N);
}

__global__ void k_split_tab(const float2 *__restrict__ U, size_t stride, int w, int h,
                            const OutRef *__restrict__ outs) {
    const int x = (blockIdx.x * blockDim.x + threadIdx.x) * kTabPx;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const OutRef o = outs[blockIdx.z];
    const float2 *s = U + (size_t)blockIdx.z * stride + (size_t)y * w + x;
    float *du = o.u + (size_t)y * o.pitch + x, *dv = o.v + (size_t)y * o.pitch + x;
    const bool vec = x + kTabPx <= w &&
                     ((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(du) |
                       reinterpret_cast<uintptr_t>(dv)) % 16 == 0);
    if (vec) {
        const float4 a = reinterpret_cast<const float4 *>(s)[0];
        const float4 b = reinterpret_cast<const float4 *>(s)[1];
        *reinterpret_cast<float4 *>(du) = make_float4(a.x, a.z, b.x, b.z);
        *reinterpret_cast<float4 *>(dv) = make_float4(a.y, a.w, b.y, b.w);
        return;
    }
    for (int k = 0; k < kTabPx && x + k < w; k++) {
        const float2 u = s[k];
        du[k] = u.x;
        dv[k] = u.y;
    }
}

void launch_split_tab(const float2 *U, size_t stride, int w, int h, const OutRef *outs, int B,
                      cudaStream_t st) {
    dim3 blk(32, 8), g(div_up(w, 32 * kTabPx), div_up(h, 8), B);
    k_split_tab<<<g, blk, 0, st>>>(U, stride, w, h, outs);
}

void launch_split2(const float2 *U, size_t stride, int N, float *out, int B, cudaStream_t st) {
    k_split2<<<dim3(imin(div_up(N, 1024), 1024), B), 256, 0, st>>>(U, stride, N, out,
                                                                   out + (size_t)B * N, B);
}

// ================================================================ host plan
// Jacobi configurations: the region is 64 x v*nw pixels with a k-pixel halo, nw
// warps, mb blocks resident on an SM.
struct HsJCfg {
    int v, nw, k, mb;
};
constexpr HsJCfg kHsCfgs[] = {{4, 16, 4, 1}, {4, 8, 4, 2}, {4, 16, 8, 1}, {2, 12, 4, 2}, {4, 16, 16, 1}, {2, 16, 8, 2}};
constexpr int kHsNumCfgs = 6;
std::string hs_config_name(int c) {  // owned tile and sweeps a launch
    if (c < 0 || c >= kHsNumCfgs) return "";
    const HsJCfg &f = kHsCfgs[c];
    return std::to_string(64 - 2 * f.k) + "x" + std::to_string(f.v * f.nw - 2 * f.k) + "/" + std::to_string(f.k);
}

template <int C> using HsCfgTile = HsTile<kHsCfgs[C].v, kHsCfgs[C].nw, kHsCfgs[C].k>;

template <int C> constexpr int hs_smem() { return (int)sizeof(HsSmem<HsCfgTile<C>>); }

// cuTensorMapEncodeTiled, looked up in the driver once (null if unavailable).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// A tiled map of 8-byte elements, zero fill outside; dims innermost first,
// byte strides of dims 1..rank-1.
static bool encode_map8(CUtensorMap *m, void *base, int rank, const cuuint64_t *dims,
                 const cuuint64_t *strides, const cuuint32_t *box) {
    const PFN_cuTensorMapEncodeTiled_v12000 fn = tensor_map_encoder();
    if (!fn) return false;
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT64, (cuuint32_t)rank, base, dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor maps of the regions of configuration c.  TMA wants 16-byte strides
// (even w and pair stride); otherwise, or without err, the kernel loads the
// regions itself.
static void hs_maps(HsJacobiArgs &a, int c, int B, int *err) {
    a.err = err;
    a.tma = 0;
    if (!a.vec || !err) return;
    const cuuint32_t box[3] = {64, (cuuint32_t)(kHsCfgs[c].v * kHsCfgs[c].nw), 1};
    const cuuint64_t dims[3] = {(cuuint64_t)a.w, (cuuint64_t)a.h, (cuuint64_t)B};
    const cuuint64_t sd[2] = {8 * (cuuint64_t)a.w, 8 * (cuuint64_t)a.dstride};
    const cuuint64_t si[2] = {8 * (cuuint64_t)a.w, 8 * (cuuint64_t)a.stride};
    a.tma = encode_map8(&a.m0, const_cast<float2 *>(a.D), 3, dims, sd, box) &&
            encode_map8(&a.m1, const_cast<float2 *>(a.D + a.plane), 3, dims, sd, box) &&
            encode_map8(&a.mi, const_cast<float2 *>(a.in), 3, dims, si, box);
}

template <int C> static void hs_jacobi_launch(int B, cudaStream_t st, const HsJacobiArgs &a) {
    using T = HsCfgTile<C>;
    HsJacobiArgs t = a;
    t.tiles_x = div_up(a.w, T::TW);
    t.tiles_y = div_up(a.h, T::TH);
    t.tiles = t.tiles_x * t.tiles_y * B;
    const auto k = a.tma ? k_hs_jacobi<T, kHsCfgs[C].mb, true> : k_hs_jacobi<T, kHsCfgs[C].mb, false>;
    k<<<imin(t.tiles, kHsCfgs[C].mb * kNumSMs), T::NT, hs_smem<C>(), st>>>(t);
}

template <int C> static void hs_set_smem_attr() {
    OF_CUDA(cudaFuncSetAttribute(k_hs_jacobi<HsCfgTile<C>, kHsCfgs[C].mb, true>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, hs_smem<C>()));
    OF_CUDA(cudaFuncSetAttribute(k_hs_jacobi<HsCfgTile<C>, kHsCfgs[C].mb, false>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, hs_smem<C>()));
}
static void hs_jacobi_cfg(int c, int B, cudaStream_t st, const HsJacobiArgs &a) {
    switch (c) {
        case 1: hs_jacobi_launch<1>(B, st, a); break;
        case 2: hs_jacobi_launch<2>(B, st, a); break;
        case 3: hs_jacobi_launch<3>(B, st, a); break;
        case 4: hs_jacobi_launch<4>(B, st, a); break;
        case 5: hs_jacobi_launch<5>(B, st, a); break;
        default: hs_jacobi_launch<0>(B, st, a); break;
    }
}

// Resident levels: tiles of 48x16 with 8 sweeps between exchanges or, where those
// are more than a cluster's 16 blocks, of 56x24 with 4.
using HsRes8 = HsTile<2, 16, 8>;
using HsRes4 = HsTile<2, 16, 4>;
template <typename T> static bool hs_res_fits(int w, int h) { return div_up(w, T::TW) * div_up(h, T::TH) <= 16; }

// Launch configuration of n blocks in clusters of C; at: its cluster attribute.
template <typename T> static cudaLaunchConfig_t hs_res_config(int n, int C, cudaLaunchAttribute &at) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(n);
    lc.blockDim = dim3(T::NT);
    lc.dynamicSmemBytes = sizeof(HsRes<T>);
    at = cudaLaunchAttribute{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    lc.attrs = &at;
    lc.numAttrs = 1;
    return lc;
}

template <typename T> static void hs_res_launch(int B, cudaStream_t st, HsJacobiArgs a) {
    a.tiles_x = div_up(a.w, T::TW);
    a.tiles_y = div_up(a.h, T::TH);
    a.tiles = a.tiles_x * a.tiles_y * B;
    cudaLaunchAttribute at;
    cudaLaunchConfig_t lc = hs_res_config<T>(a.tiles, a.tiles_x * a.tiles_y, at);
    lc.stream = st;
    OF_CUDA(cudaLaunchKernelEx(&lc, k_hs_res<T>, a));
}

constexpr int kHsResAlone = 120 * 1024;  // shared memory that leaves a block its SM

template <typename T> static void hs_res_attrs() {
    OF_CUDA(cudaFuncSetAttribute(k_hs_res<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHsResAlone));
    OF_CUDA(cudaFuncSetAttribute(k_hs_res<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

// Clusters of C blocks that run at the same time, two blocks on an SM or (alone) one
// (0: the device takes none).
template <typename T> static int hs_res_active(int C, bool alone) {
    static std::mutex mu;
    static std::map<std::tuple<int, int, bool>, int> seen;
    int dev = 0;
    OF_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(dev, C, alone);
    const auto it = seen.find(key);
    if (it != seen.end()) return it->second;
    cudaLaunchAttribute at;
    cudaLaunchConfig_t lc = hs_res_config<T>(C, C, at);
    if (alone) lc.dynamicSmemBytes = kHsResAlone;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_hs_res<T>, &lc) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    return seen[key] = n;
}

// Microseconds of K sweeps and an exchange: alone on the SMs, and two blocks an SM.
template <typename T> static float hs_res_form_time(int w, int h, int B, int sweeps, float alone, float shared) {
    const int C = div_up(w, T::TW) * div_up(h, T::TH), most = hs_res_active<T>(C, false);
    if (most <= 0) return 1e30f;
    const int waves = (B - 1) / most, rest = B - waves * most;
    const float t = (float)waves * shared + (rest <= hs_res_active<T>(C, true) ? alone : shared);
    return t * (float)div_up(sweeps, T::K);
}
// Microseconds of the sweeps of B pairs in resident levels (1e30: not possible).
// OFLOW_HS_RES=0: as on a device that takes no clusters (used to test it).
static float hs_res_time(int w, int h, int B, int sweeps) {
    if (const char *e = getenv("OFLOW_HS_RES"))
        if (!atoi(e)) return 1e30f;
    if (hs_res_fits<HsRes8>(w, h)) return hs_res_form_time<HsRes8>(w, h, B, sweeps, 3.8f, 7.2f);
    if (hs_res_fits<HsRes4>(w, h)) return hs_res_form_time<HsRes4>(w, h, B, sweeps, 2.3f, 4.0f);
    return 1e30f;
}

// Microseconds of the sweeps in launches of a configuration, by TMA or without: what
// a launch takes with one tile an SM, and what each further tile of the busiest SM
// adds.  Fitted to 40x30 to 1280x720, 1 to 64 pairs, 52 to 200 sweeps.
constexpr float kHsAlone[2][kHsNumCfgs] = {{6.8f, 4.4f, 9.3f, 4.05f, 13.9f, 6.55f}, {5.9f, 4.1f, 8.5f, 3.85f, 13.2f, 6.2f}};
constexpr float kHsMore[2][kHsNumCfgs] = {{5.5f, 2.5f, 7.7f, 2.2f, 11.4f, 4.4f}, {4.1f, 1.9f, 6.25f, 1.75f, 10.0f, 3.45f}};
static float hs_tiles_time(int c, int w, int h, int B, int sweeps, bool tma) {
    const HsJCfg &f = kHsCfgs[c];
    const long long tiles = (long long)div_up(w, 64 - 2 * f.k) * div_up(h, f.v * f.nw - 2 * f.k) * B;
    return (float)div_up(sweeps, f.k) * (kHsAlone[tma][c] + (float)((tiles - 1) / kNumSMs) * kHsMore[tma][c]);
}

static void hs_set_smem_attrs() {
    hs_set_smem_attr<0>();
    hs_set_smem_attr<1>();
    hs_set_smem_attr<2>();
    hs_set_smem_attr<3>();
    hs_set_smem_attr<4>();
    hs_set_smem_attr<5>();
    hs_res_attrs<HsRes8>();
    hs_res_attrs<HsRes4>();
}

// All sweeps of one warp: from zero increments to the flow updated.  Configuration 5
// runs resident where a cluster holds the level and that is the faster way.
static void hs_sweeps(int cfg, int B, cudaStream_t st, const float2 *D, size_t plane, float2 *const dU[2],
                      float2 *U, size_t stride, int w, int h, int sweeps, bool update, int *hint, int *err) {
    const int K = kHsCfgs[cfg].k;
    const bool vec = (w & 1) == 0 && (stride & 1) == 0;  // and so by TMA, if there is a flag for its wait
    if (cfg == 5 && sweeps > 0 && hs_res_time(w, h, B, sweeps) < hs_tiles_time(5, w, h, B, sweeps, vec && err)) {
        HsJacobiArgs a;
        memset(&a, 0, sizeof(a));
        a.D = D;
        a.plane = plane;
        a.dstride = a.stride = stride;
        a.out = dU[1];
        a.U = U;
        a.w = w;
        a.h = h;
        a.sweeps = sweeps;
        a.last = update;
        a.vec = vec;
        if (hs_res_fits<HsRes8>(w, h)) hs_res_launch<HsRes8>(B, st, a);
        else hs_res_launch<HsRes4>(B, st, a);
        return;
    }
    for (int done = 0, cur = 0; done < sweeps; cur ^= 1) {
        const int k = imin(K, sweeps - done);
        HsJacobiArgs a;
        memset(&a, 0, sizeof(a));
        a.D = D;
        a.plane = plane;
        a.dstride = a.stride = stride;
        a.in = dU[cur];
        a.out = dU[cur ^ 1];
        a.U = U;
        a.hint = hint;
        a.w = w;
        a.h = h;
        a.sweeps = k;
        a.first = done == 0;
        a.last = update && done + k == sweeps;
        a.vec = vec;
        hs_maps(a, cfg, B, err);
        hs_jacobi_cfg(cfg, B, st, a);
        done += k;
    }
}

// The configuration of a level, the one with the least estimated time; OFLOW_HS_CFG
// forces one (used to test and time them), and a plan's tuning table comes before it.
// 104 sweeps of B pairs, here and by two forms alone (resident or 48x16 tiles up to
// 296 of them, else 48x48 tiles), both with tiles fetched ahead:
//   101x99, 20 pairs 168 and 265 us; 145x97, 13: 143 and 254; 160x120, 13: 134 and 224;
//   193x145, 8: 201 and 247; 337x170, 5: 199 and 243; 400x300, 1: 102 and 139
static int hs_pick(int w, int h, int B, int sweeps, bool tma) {
    if (const char *e = getenv("OFLOW_HS_CFG")) {
        const int c = atoi(e);
        if (c >= 0 && c < kHsNumCfgs) return c;
    }
    int best = 5;
    float best_t = hs_res_time(w, h, B, sweeps);
    for (int c = 0; c < kHsNumCfgs; c++) {
        const float t = hs_tiles_time(c, w, h, B, sweeps, tma);
        if (t < best_t) {
            best_t = t;
            best = c;
        }
    }
    return best;
}

HsPlan::HsPlan(int w, int h, int B, int dtype, const oflow_hs_params &prm, const TuneTable *tuned)
    : w_(w), h_(h), B_(B), dtype_(dtype), prm_(prm) {
    OF_CHECK(B >= 1, "hs: empty batch");
    OF_CHECK(prm.nlevels >= 1 && prm.nlevels <= 16, "hs: nlevels out of range");
    OF_CHECK(prm.nwarp >= 0 && prm.nsolver >= 0, "hs: negative iteration count");
    L_ = prm.nlevels;
    W_[L_ - 1] = w;
    H_[L_ - 1] = h;
    for (int l = L_ - 1; l > 0; l--) {
        W_[l - 1] = W_[l] / 2;
        H_[l - 1] = H_[l] / 2;
    }
    OF_CHECK(W_[0] >= 1 && H_[0] >= 1, "hs: too many levels for the frame size");
    N_ = (size_t)w * h;
    size_t acc = 0;
    for (int l = 0; l < L_; l++) {
        pyr_off_[l] = acc;
        acc += (size_t)2 * B * W_[l] * H_[l];
    }
    const size_t esz = dtype == OFLOW_U8 ? 1 : 4;
    o_raw_ = ar_.reserve(2 * B * N_ * esz);
    o_pyr_ = ar_.reserve(acc * 4);
    o_D_ = ar_.reserve(B * N_ * 16);
    o_dU0_ = ar_.reserve(B * N_ * 8);
    o_dU1_ = ar_.reserve(B * N_ * 8);
    o_Ua_ = ar_.reserve(B * N_ * 8);
    o_Ub_ = ar_.reserve(B * N_ * 8);
    o_out_ = ar_.reserve(2 * B * N_ * 4);
    o_hint_ = ar_.reserve((size_t)B * div_up(w, 32) * div_up(h, 16) * 4);  // the smallest tiles are 32x32, 48x16
    o_ftab_ = ar_.reserve(sizeof(FrameRef) * 2 * B);
    o_otab_ = ar_.reserve(sizeof(OutRef) * B);
    ar_.commit();
    io_.init(ar_.at<FrameRef>(o_ftab_), ar_.at<OutRef>(o_otab_), B);
    for (int b = 0; b < B; b++) {
        bind_raw(b, 0);
        bind_raw(b, 1);
        bind_own_out(b);
    }
    // the default tables are valid for schedules recorded into a caller's graph
    io_.upload(nullptr);
    OF_CUDA(cudaStreamSynchronize(nullptr));
    hs_set_smem_attrs();
    for (int l = 0; l < L_; l++) {
        const auto it = tuned ? tuned->find(tune_key(W_[l], H_[l], B, kTuneHs)) : TuneTable::const_iterator();
        const bool ok = tuned && it != tuned->end() && it->second >= 0 && it->second < kHsNumCfgs;
        jcfg_[l] = ok ? it->second
                      : hs_pick(W_[l], H_[l], B, prm.nsolver, (W_[l] & 1) == 0 && (N_ & 1) == 0);
    }
}

void *HsPlan::raw_input(int b, int k) const {
    const size_t esz = dtype_ == OFLOW_U8 ? 1 : 4;
    return ar_.at<char>(o_raw_) + (size_t)(2 * b + k) * N_ * esz;
}
const float *HsPlan::out_u(int b) const { return ar_.at<float>(o_out_) + (size_t)b * N_; }
const float *HsPlan::out_v(int b) const { return ar_.at<float>(o_out_) + (size_t)(B_ + b) * N_; }
void HsPlan::bind_frame(int b, int k, const void *p, int pitch) { io_.set_frame(b, k, p, pitch ? pitch : w_); }
void HsPlan::bind_raw(int b, int k) { io_.set_frame(b, k, raw_input(b, k), w_); }
void HsPlan::bind_out(int b, float *u, float *v, int pitch) { io_.set_out(b, u, v, pitch ? pitch : w_); }
void HsPlan::bind_own_out(int b) {
    float *o = ar_.at<float>(o_out_);
    io_.set_out(b, o + (size_t)b * N_, o + (size_t)(B_ + b) * N_, w_);
}

void HsPlan::record(cudaStream_t st) {
    const int B = B_;
    float *pyr = ar_.at<float>(o_pyr_);
    float2 *D = ar_.at<float2>(o_D_);
    float2 *dU[2] = {ar_.at<float2>(o_dU0_), ar_.at<float2>(o_dU1_)};
    float2 *Ubuf[2] = {ar_.at<float2>(o_Ua_), ar_.at<float2>(o_Ub_)};
    const int top = L_ - 1;
    {
        // frames through the frame table (the caller's device frames in place,
        // or this plan's staging buffers)
        launch_ingest_tab(io_.frames(), dtype_, w_, h_, pyr + pyr_off_[top], N_, 2 * B, st);
    }
    for (int l = top; l > 0; l--) {
        dim3 blk(32, 8), g(div_up(W_[l - 1], 32), div_up(H_[l - 1], 8), 2 * B);
        k_hs_downscale<<<g, blk, 0, st>>>(pyr + pyr_off_[l], (size_t)W_[l] * H_[l], W_[l], H_[l],
                                          pyr + pyr_off_[l - 1], (size_t)W_[l - 1] * H_[l - 1]);
    }
    int ub = 0;  // Ubuf index holding the flow of the current level
    OF_CUDA(cudaMemsetAsync(Ubuf[ub], 0, B * N_ * 8, st));
    for (int l = 0; l < L_; l++) {
        const int lw = W_[l], lh = H_[l];
        const size_t lp = (size_t)lw * lh;
        for (int wi = 0; wi < prm_.nwarp; wi++) {
            dim3 dg(div_up(lw, kDTW), div_up(lh, kDTH), B);
            k_hs_warp_deriv<<<dg, dim3(kDTW, kDTH), 0, st>>>(pyr + pyr_off_[l], lp, lw, lh,
                                                             Ubuf[ub], N_, 0, prm_.alpha, D, B * N_, N_);
            // with no sweeps du = 0: the flow is unchanged
            hs_sweeps(jcfg_[l], B, st, D, B * N_, dU, Ubuf[ub], N_, lw, lh, prm_.nsolver, true,
                      ar_.at<int>(o_hint_), err_.device());
        }
        if (l != top) {
            const float sx = (float)W_[l + 1] / (float)lw;
            const float sy = (float)H_[l + 1] / (float)lh;
            launch_upscale2(Ubuf[ub], N_, lw, lh, Ubuf[ub ^ 1], N_, W_[l + 1], H_[l + 1], sx, sy, B,
                            st);
            ub ^= 1;
        }
    }
    launch_split_tab(Ubuf[ub], N_, w_, h_, io_.outs(), B, st);
    OF_CUDA(cudaGetLastError());
}

void HsPlan::run(cudaStream_t st) {
    io_.upload(st);
    if (!graph_.ready()) graph_.capture(st, [&](cudaStream_t s) { record(s); });
    graph_.launch(st);
}

// Best of `reps` timed runs of 48 sweeps (in launches of the configuration's
// depth) per configuration and level.  The sweep has no data-dependent control
// flow, so the derivative buffer the last solve left is fine input at every
// level size; the runs write only the du scratch, never the flow or outputs.
void HsPlan::autotune(cudaStream_t st, TuneTable *table, int reps) {
    float2 *D = ar_.at<float2>(o_D_);
    float2 *dU[2] = {ar_.at<float2>(o_dU0_), ar_.at<float2>(o_dU1_)};
    float2 *U = ar_.at<float2>(o_Ua_);
    cudaEvent_t e0, e1;
    OF_CUDA(cudaEventCreate(&e0));
    OF_CUDA(cudaEventCreate(&e1));
    constexpr int kSweeps = 48;
    try {
        for (int l = 0; l < L_; l++) {
            const int lw = W_[l], lh = H_[l];
            float best = 1e30f;
            int best_c = jcfg_[l];
            for (int c = 0; c < kHsNumCfgs; c++) {
                float ms_min = 1e30f;
                for (int r = 0; r <= reps; r++) {  // the first round warms up
                    OF_CUDA(cudaEventRecord(e0, st));
                    hs_sweeps(c, B_, st, D, B_ * N_, dU, U, N_, lw, lh, kSweeps, false, ar_.at<int>(o_hint_),
                              err_.device());
                    OF_CUDA(cudaEventRecord(e1, st));
                    OF_CUDA(cudaEventSynchronize(e1));
                    float ms = 0.0f;
                    OF_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                    if (r > 0) ms_min = ms < ms_min ? ms : ms_min;
                }
                if (ms_min < best) {
                    best = ms_min;
                    best_c = c;
                }
            }
            jcfg_[l] = best_c;
            if (table) (*table)[tune_key(lw, lh, B_, kTuneHs)] = best_c;
        }
    } catch (...) {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    graph_.reset();  // the next run captures the new configurations
}

void HsPlan::check_device_error() {
    if (err_.take()) throw Error(OFLOW_ERR_TIMEOUT, "hs: a Jacobi tile's TMA load gave up its bounded wait");
}

// ================================================================ caller scratch
// The Horn-Schunck schedule of HsPlan::record for one pair, enqueued on
// scratch the caller provides (no allocation here).  Frames and flows are
// device float planes with row pitches in elements.
static size_t hs_carve(size_t &off, size_t bytes) {
    const size_t at = (off + 255) & ~size_t(255);
    off = at + bytes;
    return at;
}

size_t hs_scratch_bytes(int w, int h, int nlevels) {
    if (w < 1 || h < 1 || nlevels < 1 || nlevels > 16) return 0;
    int W = w, H = h;
    size_t pyr = 0;
    for (int l = nlevels - 1; l >= 0; l--) {
        if (W < 1 || H < 1) return 0;
        pyr += (size_t)2 * W * H;
        W /= 2;
        H /= 2;
    }
    const size_t N = (size_t)w * h;
    size_t off = 0;
    hs_carve(off, pyr * 4);   // pyramid
    hs_carve(off, N * 16);    // D
    hs_carve(off, N * 8);     // dU0
    hs_carve(off, N * 8);     // dU1
    hs_carve(off, N * 8);     // Ua
    hs_carve(off, N * 8);     // Ub
    hs_carve(off, 2 * N * 4); // u | v; before them the sweeps' hints (a tile has a pixel)
    return off;
}

void hs_enqueue_into(void *scratch, const float *I0, const float *I1, int w, int h, int pitch,
                     const oflow_hs_params &prm, float *u, float *v, int out_pitch,
                     cudaStream_t st) {
    hs_set_smem_attrs();
    const int L = prm.nlevels;
    int Wl[16], Hl[16];
    Wl[L - 1] = w;
    Hl[L - 1] = h;
    for (int l = L - 1; l > 0; l--) {
        Wl[l - 1] = Wl[l] / 2;
        Hl[l - 1] = Hl[l] / 2;
    }
    size_t pyr_off[16], acc = 0;
    for (int l = 0; l < L; l++) {
        pyr_off[l] = acc;
        acc += (size_t)2 * Wl[l] * Hl[l];
    }
    const size_t N = (size_t)w * h;
    size_t off = 0;
    char *base = static_cast<char *>(scratch);
    float *pyr = reinterpret_cast<float *>(base + hs_carve(off, acc * 4));
    float2 *D = reinterpret_cast<float2 *>(base + hs_carve(off, N * 16));
    float2 *dU[2];
    dU[0] = reinterpret_cast<float2 *>(base + hs_carve(off, N * 8));
    dU[1] = reinterpret_cast<float2 *>(base + hs_carve(off, N * 8));
    float2 *Ubuf[2];
    Ubuf[0] = reinterpret_cast<float2 *>(base + hs_carve(off, N * 8));
    Ubuf[1] = reinterpret_cast<float2 *>(base + hs_carve(off, N * 8));
    float *out = reinterpret_cast<float *>(base + hs_carve(off, 2 * N * 4));
    const int top = L - 1;
    const size_t rowb = (size_t)w * 4, pb = (size_t)(pitch ? pitch : w) * 4;
    OF_CUDA(cudaMemcpy2DAsync(pyr + pyr_off[top], rowb, I0, pb, rowb, h, cudaMemcpyDeviceToDevice, st));
    OF_CUDA(cudaMemcpy2DAsync(pyr + pyr_off[top] + N, rowb, I1, pb, rowb, h,
                              cudaMemcpyDeviceToDevice, st));
    for (int l = top; l > 0; l--) {
        dim3 blk(32, 8), g(div_up(Wl[l - 1], 32), div_up(Hl[l - 1], 8), 2);
        k_hs_downscale<<<g, blk, 0, st>>>(pyr + pyr_off[l], (size_t)Wl[l] * Hl[l], Wl[l], Hl[l],
                                          pyr + pyr_off[l - 1], (size_t)Wl[l - 1] * Hl[l - 1]);
    }
    int ub = 0;
    OF_CUDA(cudaMemsetAsync(Ubuf[ub], 0, N * 8, st));  // the flow starts at zero
    for (int l = 0; l < L; l++) {
        const int lw = Wl[l], lh = Hl[l];
        const size_t lp = (size_t)lw * lh;
        for (int wi = 0; wi < prm.nwarp; wi++) {
            dim3 dg(div_up(lw, kDTW), div_up(lh, kDTH), 1);
            k_hs_warp_deriv<<<dg, dim3(kDTW, kDTH), 0, st>>>(pyr + pyr_off[l], lp, lw, lh,
                                                             Ubuf[ub], N, 0, prm.alpha, D, N, N);
            hs_sweeps(hs_pick(lw, lh, 1, prm.nsolver, false), 1, st, D, N, dU, Ubuf[ub], N, lw, lh, prm.nsolver, true,
                      reinterpret_cast<int *>(out), nullptr);
        }
        if (l != top) {
            const float sx = (float)Wl[l + 1] / (float)lw;
            const float sy = (float)Hl[l + 1] / (float)lh;
            launch_upscale2(Ubuf[ub], N, lw, lh, Ubuf[ub ^ 1], N, Wl[l + 1], Hl[l + 1], sx, sy, 1, st);
            ub ^= 1;
        }
    }
    launch_split2(Ubuf[ub], N, (int)N, out, 1, st);
    OF_CUDA(cudaGetLastError());
    const size_t ob = (size_t)(out_pitch ? out_pitch : w) * 4;
    OF_CUDA(cudaMemcpy2DAsync(u, ob, out, rowb, rowb, h, cudaMemcpyDeviceToDevice, st));
    OF_CUDA(cudaMemcpy2DAsync(v, ob, out + N, rowb, rowb, h, cudaMemcpyDeviceToDevice, st));
}

}  // namespace oflow
