// Forward 3x3 convolution (pad 1, stride 1 or 2) of the warm-start network on
// the 5th-generation tensor cores: an implicit GEMM with tcgen05.mma (BF16 in,
// FP32 accumulate in tensor memory).
//
//   out[m][k] = bias[k] + sum_{tap, c} x[n][p*st+r-1][q*st+s-1][c] * w[k][tap][c]
//   m = (n, p, q) (NHWC), tap = 3r + s
//
// A CTA owns a rectangle of output pixels, NACC accumulators of 128 of them
// (8 columns x 16 rows each), and all NP (= K padded to a multiple of 16)
// output channels.  The input pixels of all taps, with their halo, are copied
// to shared memory once (16-byte cp.async, zero-filled outside the image), as
// planes of 8 channels: 16 bytes a pixel, pixels of a row next to each other.
// Eight neighbouring pixels of a plane are then one 8-row x 16-byte core matrix
// of the no-swizzle K-major layout wherever they start, rows of the image are
// the descriptor's stride (SBO), planes its other stride (LBO), and a tap is
// an offset of the descriptor's start address.  Only the weights stream.  They
// are packed once (conv_pack_weights) to the order in which the stages of one
// tap x 8 kcs channels take them, so that a stage is one bulk copy; the copies
// run as many stages ahead as there are buffers.  One thread issues the MMAs of
// 128 x NP x 16 of a stage and commits them to the mbarrier that frees its buffer.
// Taps come in order and channels in order within a tap, whatever the tile; where the
// channels come in several regions (C above some 500), all taps of a region first.
//
//   stride 1    the region is the tile and one pixel around it
//   stride 2    even and odd columns of a region row lie apart, so that a tap's
//               every second pixel are neighbours; every second row is the SBO
//   dilated     (backward-data of stride 2) the four parities of an output pixel
//               are the four accumulators; a tap has whole sources in exactly one
//
// Gathering every tap of 128 flat pixels anew moved nine times the input, and the
// weights once per 128 pixels, through L1 and L2 with the tensor pipe idle, and the
// dilated form multiplied 36 taps by zeros for its 9.  16 images, on the device:
//
//   128x55  160 -> 64    204 -> 52 us       128x55   64 -> 64    92 -> 23 us
//   256x109  32 -> 32     84 -> 31 us       64x28   224 -> 96    73 -> 30 us
//   512x218  16 -> 32 s2  50 -> 38 us       256x109  32 -> 64 s2 47 -> 24 us
//
// What is left: an MMA with N = 64 reads 6 KB of shared memory (48 cycles, three
// times its multiplication), and a CTA loads, multiplies and stores one after the
// other, covered only by the other CTAs of the SM.
//
// The epilogue reads the accumulators back with tcgen05.ld (warp w holds TMEM
// lanes 32 (w % 4) ..., one pixel per thread), adds the bias, applies the ReLU
// and stores bf16 or f32.
//
// Every wait on an mbarrier is bounded (kWaitNs of %globaltimer); when one
// gives up, the kernel sets *err, waits (bounded) for its own copies, frees
// its tensor memory and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "cnn.cuh"
#include "common.cuh"
#include "internal.hpp"
#include "ptx.cuh"

namespace oflow {
namespace {

constexpr int kUmBM = 128;       // rows of a tile (UMMA M)

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}

// Shared-memory matrix descriptor, no swizzle, K-major: start address, LBO =
// byte distance between core matrices along K, SBO = byte distance between
// 8-row groups along M/N (all in 16-byte units), version 1 (bits 46-47).
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::f16: D f32 (bits 4-5 = 1), A and B bf16
// (bits 7-9 = 1, 10-12 = 1), both K-major, N/8 at bit 17, M/16 at bit 24.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                     bar)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
        "[%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// tensor-memory columns of N accumulator columns (a power of two, at least 32)
template <int N> __host__ __device__ constexpr uint32_t tmem_cols() {
    return N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : N <= 256 ? 256 : 512;
}

// True in one thread of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(p));
    return p != 0;
}

enum UmMode { kUmStride1 = 0, kUmStride2 = 1, kUmDilated = 2 };

// Geometry of a CTA's tile: NACC accumulators of 128 pixels, output rectangle
// TW x TH, input region RW x RH (stored RW pixels a row, a plane of PX pixels;
// PX is odd so that the planes of one pixel fall into different banks), SBO in
// pixels.
template <int MODE, int MT> struct UmTile {
    static constexpr int NACC = MODE == kUmDilated ? 4 : MT;
    static constexpr int TW = MODE == kUmDilated ? 16 : 8 * MT, TH = MODE == kUmDilated ? 32 : 16;
    static constexpr int RW = MODE == kUmStride1 ? 8 * MT + 2 : MODE == kUmStride2 ? 16 * MT + 1 : 9;
    static constexpr int RH = MODE == kUmStride1 ? 18 : MODE == kUmStride2 ? 33 : 17;
    static constexpr int PX = (RW * RH) | 1;
    static constexpr int ROW = MODE == kUmStride2 ? 2 * RW : RW;
    static constexpr int NT = NACC == 1 ? 128 : 256;
};

constexpr int kUmMaxBufs = 16;  // weight buffers of the forward kernel at most

// Bytes of one weight stage: kcs planes of 8 channels, NP rows of 16 bytes.
__host__ __device__ constexpr int um_wstage(int np, int kcs) { return kcs * np * 16; }

// The MMAs of one weight stage for accumulators t0 .. t1 - 1 (t0 + 1 when
// DILATED); straight code, since a loop with addresses to compute issues one in
// 110 cycles.
template <int NP, int NACC, bool DILATED, int PX, int KCS>
__device__ __forceinline__ void um_issue(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, int t0, int nacc,
                                         bool first) {
#pragma unroll
    for (int t = 0; t < (DILATED ? 1 : NACC); t++) {
        if (!DILATED && t >= nacc) break;
        const uint32_t acc = tmem + (uint32_t)((DILATED ? t0 : t) * NP);
#pragma unroll
        for (int j = 0; j < KCS / 2; j++)
            umma_bf16(acc, ad + (uint32_t)(8 * t + 2 * j * PX), bd + (uint32_t)(2 * j * NP), idesc,
                      j == 0 && first ? 0u : 1u);
    }
}

// w: packed weights.  kcs: planes of 8 channels a weight stage (2, 4 or 8);
// bufs: weight buffers; cr: channels of the region held at a time (all of them
// unless they don't fit); 8 kcs divides cr and C.
template <int NP, int MODE, int MT>
__global__ void __launch_bounds__(UmTile<MODE, MT>::NT)
    k_conv_fwd_umma(ConvDims d, const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
                    const float *__restrict__ bias, void *y, int flags, int ldy, int kcs, int bufs, int cr, int *err) {
    static_assert(NP % 16 == 0 && NP >= 16 && NP <= 128, "UMMA M=128 needs N a multiple of 16");
    using T = UmTile<MODE, MT>;
    constexpr int NT = T::NT, RW = T::RW, PX = T::PX;
    constexpr uint32_t TCOLS = tmem_cols<T::NACC * NP>();
    constexpr uint32_t IDESC = umma_idesc_bf16(kUmBM, NP);
    extern __shared__ __align__(1024) uint8_t um_smem[];
    __shared__ __align__(8) uint64_t mbar[2 * kUmMaxBufs + 2];  // landed, freed; the region has landed, is done with
    __shared__ uint32_t tmem_base;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    const int gx = div_up(d.Q, T::TW), gy = div_up(d.P, T::TH);
    const int q0 = (blockIdx.x % gx) * T::TW, p0 = (blockIdx.x / gx) % gy * T::TH, n = blockIdx.x / (gx * gy);
    const int wstage = um_wstage(NP, kcs);
    const uint32_t sreg = smem_u32(um_smem), sring = sreg + (uint32_t)(cr / 8) * (PX * 16);
    const int nst = 9 * (d.C / 8 / kcs), per_reg = 9 * (cr / 8 / kcs);
    // accumulators with a column inside the image
    const int nacc = MODE == kUmDilated ? 4 : imin(MT, div_up(d.Q - q0, 8));
    const uint32_t full = smem_u32(mbar), freed = full + 8 * kUmMaxBufs, regbar = freed + 8 * kUmMaxBufs,
                   regdone = regbar + 8;

    // first input row and column of the region
    const int y0 = MODE == kUmStride1 ? p0 - 1 : MODE == kUmStride2 ? 2 * p0 - 1 : p0 / 2;
    const int x0 = MODE == kUmStride1 ? q0 - 1 : MODE == kUmStride2 ? 2 * q0 - 1 : q0 / 2;
    const __nv_bfloat16 *xn = x + (size_t)n * d.H * d.W * d.C;
    // lanes run over the channel planes of a pixel first: whole sectors
    auto load_region = [&](int c0) {
        const int nk = cr / 8;
        const uint32_t magic = 0xFFFFFFFFu / (uint32_t)nk + 1u;  // exact quotients below 2^16
        for (int e = tid - 32; e < RW * T::RH * nk; e += NT - 32) {
            const int px = (int)__umulhi((uint32_t)e, magic), kc = e - px * nk;
            const int ry = px / RW, rx = px % RW, yy = y0 + ry, xx = x0 + rx;
            const bool ok = (unsigned)yy < (unsigned)d.H && (unsigned)xx < (unsigned)d.W;
            const int pos = MODE == kUmStride2 ? ry * RW + (rx >> 1) + (rx & 1 ? 8 * MT + 1 : 0) : px;
            cp_async16_l1(sreg + (uint32_t)(kc * PX + pos) * 16,
                       ok ? xn + ((size_t)yy * d.W + xx) * d.C + c0 + kc * 8 : x, ok);
        }
    };

    if (warp > 0) load_region(0);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_u32(&tmem_base)),
                     "r"(TCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < bufs; i++) {
            mbar_init(full + 8 * i, 1);
            mbar_init(freed + 8 * i, 1);
        }
        mbar_init(regbar, NT - 32);
        mbar_init(regdone, 1);
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    bool timed_out = false;

    if (warp > 0) {
        // thread 32 fetches the weights: stages follow one another by channels of
        // the region, taps, regions (counters, since a division a stage would cost
        // more than its MMAs)
        int issued = 0, fbuf = 0, fkc = 0, ftap = 0;
        const __nv_bfloat16 *src = w, *reg0 = w;
        auto fetch = [&]() {
            mbar_arrive_expect_tx(full + 8 * fbuf, (uint32_t)wstage);
            bulk_load(sring + (uint32_t)(fbuf * wstage), src, (uint32_t)wstage, full + 8 * fbuf);
            issued++;
            if (++fbuf == bufs) fbuf = 0;
            src += wstage / 2;
            fkc += kcs;
            if (fkc == cr / 8) {
                fkc = 0;
                src += (size_t)(d.C - cr) * NP;
                if (++ftap == 9) {
                    ftap = 0;
                    src = reg0 += (size_t)cr * NP;
                }
            }
        };
        if (tid == 32)
            while (issued < imin(bufs, nst)) fetch();
        cp_async_commit();
        cp_async_wait<0>();
        fence_async_smem();
        mbar_arrive(regbar);
        // The next region replaces one whose MMAs are done.  Thread 32 knows that
        // from the last stage's buffer and tells the others, on a barrier that can't
        // pass them (thread 32's next arrival needs theirs on regbar), which the
        // buffers' could: those are freed once a stage, and tell two phases apart.
        int buf = 0, ph = 0, left = per_reg, c0 = 0;  // stage s: its buffer is freed for the (ph + 1)-th time
        if (tid == 32 || per_reg < nst)
#pragma unroll 1
            for (int s = 0, rph = 0; s < nst; s++) {
                if (tid == 32 && !mbar_wait_bounded(freed + 8 * buf, ph)) {
                    timed_out = true;
                    break;
                }
                if (tid == 32 && issued < nst) fetch();
                if (--left == 0 && s + 1 < nst) {  // the next channels
                    if (tid == 32) {
                        mbar_arrive(regdone);
                    } else if (!mbar_wait_bounded(regdone, rph)) {
                        timed_out = true;
                        break;
                    }
                    rph ^= 1;
                    left = per_reg;
                    load_region(c0 += cr);
                    cp_async_commit();
                    cp_async_wait<0>();
                    fence_async_smem();
                    mbar_arrive(regbar);
                }
                if (++buf == bufs) {
                    buf = 0;
                    ph ^= 1;
                }
            }
        if (timed_out && tid == 32)  // its own copies in flight
            for (int s = imax(0, issued - bufs); s < issued; s++)
                mbar_wait_bounded(full + 8 * (s % bufs), (uint32_t)(s / bufs) & 1u);
    } else {
        // the whole warp follows the stages, so that addresses and descriptors are
        // uniform; one thread issues
        const bool issuer = elect_one();
        const uint64_t adesc = umma_desc(0, PX * 16, T::ROW * 16), bdesc = umma_desc(0, NP * 16, 128);
        int tap = 0, kc0 = 0, buf = 0, ph = 0;
#pragma unroll 1
        for (int s = 0; s < nst; s++) {
            if ((tap == 0 && kc0 == 0 && !mbar_wait_bounded(regbar, (uint32_t)(s / per_reg) & 1u)) ||
                !mbar_wait_bounded(full + 8 * buf, ph)) {
                timed_out = true;
                break;
            }
            tc_fence_after();
            const int r = tap / 3, sx = tap % 3;
            // the tap's first pixel in the region, its accumulator, and whether
            // that holds anything yet
            int off, t0 = 0;
            bool first = s == 0;
            if (MODE == kUmStride1) {
                off = r * RW + sx;
            } else if (MODE == kUmStride2) {
                off = r * RW + (sx == 1 ? 8 * MT + 1 : sx >> 1);
            } else {
                off = (r >> 1) * RW + (sx >> 1);
                t0 = (r != 1 ? 2 : 0) + (sx != 1 ? 1 : 0);
                first = s < per_reg && kc0 == 0 && r < 2 && sx < 2;
            }
            const uint64_t ad = adesc + ((sreg >> 4) + (uint32_t)(kc0 * PX + off));
            const uint64_t bd = bdesc + ((sring + (uint32_t)(buf * wstage)) >> 4);
            if (issuer) {
                constexpr bool DIL = MODE == kUmDilated;
                switch (kcs) {
                    case 2: um_issue<NP, T::NACC, DIL, PX, 2>(tmem, ad, bd, IDESC, t0, nacc, first); break;
                    case 4: um_issue<NP, T::NACC, DIL, PX, 4>(tmem, ad, bd, IDESC, t0, nacc, first); break;
                    case 6: um_issue<NP, T::NACC, DIL, PX, 6>(tmem, ad, bd, IDESC, t0, nacc, first); break;
                    case 8: um_issue<NP, T::NACC, DIL, PX, 8>(tmem, ad, bd, IDESC, t0, nacc, first); break;
                    case 10: um_issue<NP, T::NACC, DIL, PX, 10>(tmem, ad, bd, IDESC, t0, nacc, first); break;
                    default: um_issue<NP, T::NACC, DIL, PX, 14>(tmem, ad, bd, IDESC, t0, nacc, first); break;
                }
                umma_commit(freed + 8 * buf);
            }
            __syncwarp();
            kc0 += kcs;
            if (kc0 == cr / 8) {
                kc0 = 0;
                if (++tap == 9) tap = 0;
            }
            // the last commit tracks every MMA of this CTA
            if (s == nst - 1 && !mbar_wait_bounded(freed + 8 * buf, ph)) timed_out = true;
            if (++buf == bufs) {
                buf = 0;
                ph ^= 1;
            }
        }
    }
    // block-uniform from here: tcgen05.ld is warp-collective
    timed_out = __syncthreads_or(timed_out);
    if (timed_out && tid == 0) atomicOr(err, 1);
    tc_fence_after();
    if (!timed_out) {
        const int row = (warp & 3) * 32 + lane;
        const bool relu = flags & 1, f32 = flags & 2, accum = flags & 4;
        const int ld = ldy > 0 ? ldy : d.K;  // elements between output rows
        const bool vec = d.K % 8 == 0 && ld % 8 == 0;  // rows of y start on 16-byte boundaries
#pragma unroll 1
        for (int t = warp >> 2; t < nacc; t += NT / 128) {
            int p = p0 + (row >> 3), q = q0 + 8 * t + (row & 7);
            if (MODE == kUmDilated) {
                p = p0 + 2 * (row >> 3) + (t >> 1);
                q = q0 + 2 * (row & 7) + (t & 1);
            }
            const bool inside = p < d.P && q < d.Q;
            const size_t mo = ((size_t)n * d.P + p) * d.Q + q;
#pragma unroll 1
            for (int c0 = 0; c0 < NP; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(t * NP + c0), r);
                if (!inside) continue;
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int col = c0 + j;
                    float f = __uint_as_float(r[j]) + ((bias && col < d.K) ? bias[col] : 0.0f);
                    v[j] = relu ? fmaxf(f, 0.0f) : f;
                }
                if (f32) {
                    float *o = static_cast<float *>(y) + mo * ld + c0;
#pragma unroll
                    for (int j = 0; j < 16; j += 4)
                        if (vec && c0 + j + 3 < d.K) {
                            float4 *o4 = reinterpret_cast<float4 *>(o + j);
                            float4 f = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                            if (accum) {  // each output element belongs to one thread
                                const float4 g = *o4;
                                f = make_float4(g.x + f.x, g.y + f.y, g.z + f.z, g.w + f.w);
                            }
                            *o4 = f;
                        } else {
                            for (int e = 0; e < 4; e++)
                                if (c0 + j + e < d.K) o[j + e] = accum ? o[j + e] + v[j + e] : v[j + e];
                        }
                } else {
                    __nv_bfloat16 *o = static_cast<__nv_bfloat16 *>(y) + mo * ld + c0;
#pragma unroll
                    for (int j = 0; j < 16; j += 8) {
                        if (vec && c0 + j + 7 < d.K) {
                            uint4 pk;
                            __nv_bfloat162 h0 = __floats2bfloat162_rn(v[j], v[j + 1]);
                            __nv_bfloat162 h1 = __floats2bfloat162_rn(v[j + 2], v[j + 3]);
                            __nv_bfloat162 h2 = __floats2bfloat162_rn(v[j + 4], v[j + 5]);
                            __nv_bfloat162 h3 = __floats2bfloat162_rn(v[j + 6], v[j + 7]);
                            pk.x = *reinterpret_cast<uint32_t *>(&h0);
                            pk.y = *reinterpret_cast<uint32_t *>(&h1);
                            pk.z = *reinterpret_cast<uint32_t *>(&h2);
                            pk.w = *reinterpret_cast<uint32_t *>(&h3);
                            *reinterpret_cast<uint4 *>(o + j) = pk;
                        } else {
                            for (int e = 0; e < 8; e++)
                                if (c0 + j + e < d.K) o[j + e] = __float2bfloat16(v[j + e]);
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TCOLS)
                     : "memory");
}

// What one forward launch gets.
struct UmCall {
    const ConvDims &d;
    const __nv_bfloat16 *x, *w;
    const float *bias;
    void *y;
    int flags, ldy, *err;
    cudaStream_t st;
};

// Planes of 8 channels a weight stage, and its buffers: the deepest stage of at
// most 12 KB, and 16 KB of buffers or two.  Stages of 4 KB take 61 us where those of
// 10 take 52 (16 x 128x55, 160 -> 64 channels), and 32 KB of buffers cost resident
// CTAs (35 us for 30.5 at 32 -> 32).
int um_kcs(int C, int np) {
    int kcs = 2;
    for (int k : {4, 6, 8, 10, 14})
        if (C / 8 % k == 0 && um_wstage(np, k) <= 12 * 1024) kcs = k;
    return kcs;
}
int um_bufs(int C, int np) { return imax(2, imin(kUmMaxBufs, 16 * 1024 / um_wstage(np, um_kcs(C, np)))); }

// Dynamic shared memory of a CTA at most.  Kernels are allowed all of it at every
// launch: the attribute belongs to the process, and one set to a launch's own need
// could be lowered by another thread before the launch.
constexpr int kUmSmemMax = 227 * 1024 - 1024;

template <int MODE, int MT> int um_tiles(const ConvDims &d) {
    using T = UmTile<MODE, MT>;
    return div_up(d.Q, T::TW) * div_up(d.P, T::TH) * d.N;
}

template <int MODE, int MT> int um_smem(int np, int C, int cr) {
    return cr / 8 * UmTile<MODE, MT>::PX * 16 + um_bufs(C, np) * um_wstage(np, um_kcs(C, np));
}

template <int NP, int MODE, int MT> void launch_um(const UmCall &c) {
    const int kcs = um_kcs(c.d.C, NP), nk = c.d.C / 8;
    int cr = c.d.C;  // fewer channels a region where it would not fit
    while (um_smem<MODE, MT>(NP, c.d.C, cr) > kUmSmemMax) {
        cr -= 8 * kcs;
        while (nk % (cr / 8) != 0) cr -= 8 * kcs;
    }
    const int smem = um_smem<MODE, MT>(NP, c.d.C, cr);
    OF_CUDA(cudaFuncSetAttribute(k_conv_fwd_umma<NP, MODE, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kUmSmemMax));
    k_conv_fwd_umma<NP, MODE, MT><<<um_tiles<MODE, MT>(c.d), UmTile<MODE, MT>::NT, smem, c.st>>>(
        c.d, c.x, c.w, c.bias, c.y, c.flags, c.ldy, kcs, um_bufs(c.d.C, NP), cr, c.err);
}

// Wide tiles (half or less of a narrow one's halo) where the layer has few output
// channels, so that the region and not the multiplication takes the time, and
// tiles enough for two CTAs an SM that leave room for each other: 16 images of
// 256x109, 32 -> 32 channels, 30.5 us with four accumulators and 36.2 with one;
// 512x218 to half size, 16 -> 32, 38 and 41 with two and one.  With 64 output
// channels narrow tiles, of which more fit an SM, are the faster ones: 16 x 128x55,
// 64 -> 64, 26.3 us with two accumulators and 23.3 with one.
template <int NP, int MODE, int MT> bool um_wide(const ConvDims &d) {
    return um_smem<MODE, MT>(NP, d.C, d.C) <= 113 * 1024 && um_tiles<MODE, MT>(d) >= 2 * kNumSMs;
}

template <int NP> void launch_umma(const UmCall &c) {
    if (c.d.stride == 1) {
        if constexpr (NP <= 32)
            if (um_wide<NP, kUmStride1, 4>(c.d)) return launch_um<NP, kUmStride1, 4>(c);
        launch_um<NP, kUmStride1, 1>(c);
    } else if (c.d.stride == 2) {
        if constexpr (NP <= 32)
            if (um_wide<NP, kUmStride2, 2>(c.d)) return launch_um<NP, kUmStride2, 2>(c);
        launch_um<NP, kUmStride2, 1>(c);
    } else {
        launch_um<NP, kUmDilated, 1>(c);
    }
}

bool dispatch_np(int np, const UmCall &c) {
    switch (np) {
        case 16: launch_umma<16>(c); return true;
        case 32: launch_umma<32>(c); return true;
        case 48: launch_umma<48>(c); return true;
        case 64: launch_umma<64>(c); return true;
        case 96: launch_umma<96>(c); return true;
        case 128: launch_umma<128>(c); return true;
        default: return false;
    }
}

// Backward-weight product on the tensor cores:
//   gw[k][tap][c] = sum_m x[pixel(m, tap)][c] * g[m][k]
// as D = A B with rows of D (tap column, c), one accumulator per tap row, columns
// the output channels k (K rounded up to 16 = KP), and the reduction over output
// pixels m in tiles of 8 columns x 16 rows.  Both operands stay in the layout they
// have in memory, MN-major (no swizzle): a core matrix is 8 reduction rows (8
// neighbouring pixels) of 16 bytes (8 channels).  A tile of x is kept as planes of
// 16 bytes a pixel, one per 8 channels and tap column -- the columns' planes hold
// the same image shifted, so that planes are the M groups at one distance (SBO) and
// image rows the reduction groups at another (LBO) -- and a tap row is an offset
// of the start address: three times the image in shared memory for nine taps.
//
// A CTA takes the three tap columns of at most 5 channel groups (15 of the 16 M
// groups; the rest of the 128 rows is read from whatever follows and ignored)
// and every gridDim.y-th pixel tile, and adds its rows to gw with atomics.  Warps
// 1 to 7 load tiles (16-byte cp.async, zeros outside) into two or three buffers; a
// thread of warp 0 issues a tile's 24 MMAs and commits them to the mbarrier that
// frees the buffer.  Bounded waits as in the forward kernel.
//
// Gathering each of the nine taps on its own, behind a block barrier per 32 pixels,
// took 181 us for 160 -> 64 channels of 16 images of 128x55 where this takes 57;
// 78 and 37 us for 32 -> 32 of 256x109, 59 and 41 for 224 -> 96 of 64x28, 48 and 38
// for 16 -> 32 of 512x218 to half size.  What is left is the tiles' way from L2
// (some 50 KB a tile and CTA, 4 TB/s).
constexpr int kWgNT = 256;
constexpr int kWgGroups = 5;  // channel groups of 8 a CTA at most

// Geometry: input rows of a tile, pixels of a plane of x and of g (one more than
// they hold, so that planes fall into different banks).
template <int STRIDE> struct WgTile {
    static constexpr int RH = STRIDE == 1 ? 18 : 33;
    static constexpr int PXA = RH * 8 + 1, PXB = 129;
};

template <int KP, int STRIDE>
__global__ void __launch_bounds__(kWgNT) k_conv_wgrad_mn(ConvDims d, const __nv_bfloat16 *__restrict__ gb,
                                                         const __nv_bfloat16 *__restrict__ x, float *gw, int groups,
                                                         int bufs, int *err) {
    static_assert(KP % 16 == 0 && KP >= 16 && KP <= 128, "N = 16..128, step 16");
    using T = WgTile<STRIDE>;
    constexpr uint32_t IDESC = umma_idesc_bf16(kUmBM, KP) | (1u << 15) | (1u << 16);  // A, B MN-major
    constexpr uint32_t TCOLS = tmem_cols<3 * KP>();
    extern __shared__ __align__(1024) uint8_t um_smem[];
    __shared__ __align__(8) uint64_t mbar[6];  // landed, freed
    __shared__ uint32_t tmem_base;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    const int kc0 = blockIdx.x * groups, planes = 3 * imin(groups, d.C / 8 - kc0);
    const int gx = div_up(d.Q, 8), gy = div_up(d.P, 16), tiles = gx * gy * d.N;
    const int nt = div_up(tiles - (int)blockIdx.y, (int)gridDim.y);
    const uint32_t a_bytes = (uint32_t)(3 * groups * T::PXA * 16), stage = a_bytes + KP / 8 * T::PXB * 16;
    const uint32_t sbase = smem_u32(um_smem);
    const uint32_t full = smem_u32(mbar), freed = full + 24;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_u32(&tmem_base)),
                     "r"(TCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < bufs; i++) {
            mbar_init(full + 8 * i, kWgNT - 32);
            mbar_init(freed + 8 * i, 1);
        }
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    bool timed_out = false;

    if (warp > 0) {
        // a thread keeps its plane of x and its channels of g; lanes run over the
        // planes of a pixel first: the shifted ones share lines
        const int astep = (kWgNT - 32) / planes, pl = (tid - 32) % planes, apx = (tid - 32) / planes;
        const int kc = pl / 3, sx = pl - 3 * kc;
        constexpr int KG = KP / 8, BSTEP = (kWgNT - 32) / KG;
        const int kg = (tid - 32) % KG, bpx = (tid - 32) / KG;
        int buf = 0, ph = 1, abuf = 0;
#pragma unroll 1
        for (int i = 0; i < nt; i++) {
            if (i >= bufs && !mbar_wait_bounded(freed + 8 * buf, ph)) {
                timed_out = true;
                break;
            }
            const int t = blockIdx.y + i * gridDim.y;
            const int q0 = t % gx * 8, p0 = t / gx % gy * 16, n = t / (gx * gy);
            const uint32_t a = sbase + (uint32_t)buf * stage, b = a + a_bytes;
            const __nv_bfloat16 *xn = x + (size_t)n * d.H * d.W * d.C + (kc0 + kc) * 8;
            if (apx < astep)
#pragma unroll 4
                for (int px = apx; px < T::RH * 8; px += astep) {
                    const int yy = STRIDE * p0 - 1 + (px >> 3), xx = STRIDE * (q0 + (px & 7)) + sx - 1;
                    const bool ok = (unsigned)yy < (unsigned)d.H && (unsigned)xx < (unsigned)d.W;
                    cp_async16_l1(a + (uint32_t)(pl * T::PXA + px) * 16, ok ? xn + ((size_t)yy * d.W + xx) * d.C : x, ok);
                }
            const __nv_bfloat16 *gn = gb + (size_t)n * d.P * d.Q * d.K + kg * 8;
            if (bpx < BSTEP)
#pragma unroll 4
                for (int px = bpx; px < 128; px += BSTEP) {
                    const int p = p0 + (px >> 3), q = q0 + (px & 7);
                    const bool ok = p < d.P && q < d.Q && kg * 8 < d.K;
                    cp_async16_l1(b + (uint32_t)(kg * T::PXB + px) * 16, ok ? gn + ((size_t)p * d.Q + q) * d.K : gb, ok);
                }
            cp_async_commit();
            // the tile bufs - 1 loads ago has landed
            if (i >= bufs - 1) {
                if (bufs == 3) cp_async_wait<2>();
                else cp_async_wait<1>();
                fence_async_smem();
                mbar_arrive(full + 8 * abuf);
                if (++abuf == bufs) abuf = 0;
            }
            if (++buf == bufs) {
                buf = 0;
                ph ^= 1;
            }
        }
        cp_async_wait<0>();
        if (!timed_out) {
            fence_async_smem();
            for (int i = imax(0, nt - bufs + 1); i < nt; i++) {
                mbar_arrive(full + 8 * abuf);
                if (++abuf == bufs) abuf = 0;
            }
        }
    } else {
        const bool issuer = elect_one();
        const uint64_t adesc = umma_desc(0, STRIDE * 128, T::PXA * 16), bdesc = umma_desc(0, 128, T::PXB * 16);
        int buf = 0, ph = 0;
#pragma unroll 1
        for (int i = 0; i < nt; i++) {
            if (!mbar_wait_bounded(full + 8 * buf, ph)) {
                timed_out = true;
                break;
            }
            tc_fence_after();
            const uint32_t a = sbase + (uint32_t)buf * stage;
            const uint64_t ad = adesc + (a >> 4), bd = bdesc + ((a + a_bytes) >> 4);
            if (issuer) {
#pragma unroll
                for (int r = 0; r < 3; r++)
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        umma_bf16(tmem + (uint32_t)(r * KP), ad + (uint32_t)(8 * r + 16 * STRIDE * j),
                                  bd + (uint32_t)(16 * j), IDESC, j == 0 && i == 0 ? 0u : 1u);
                umma_commit(freed + 8 * buf);
            }
            __syncwarp();
            // the last commit tracks every MMA of this CTA
            if (i == nt - 1 && !mbar_wait_bounded(freed + 8 * buf, ph)) timed_out = true;
            if (++buf == bufs) {
                buf = 0;
                ph ^= 1;
            }
        }
    }
    timed_out = __syncthreads_or(timed_out);
    if (timed_out && tid == 0) atomicOr(err, 1);
    tc_fence_after();
    if (!timed_out && nt > 0) {
        const int row = (warp & 3) * 32 + lane, pl = row >> 3;  // TMEM lane = row of D
        const int c = (kc0 + pl / 3) * 8 + (row & 7), sx = pl % 3;
#pragma unroll 1
        for (int h = warp >> 2; h < 3 * (KP / 16); h += 2) {
            const int r = h / (KP / 16), cc = h % (KP / 16) * 16;
            uint32_t v[16];
            tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(r * KP + cc), v);
            if (pl >= planes) continue;
#pragma unroll
            for (int e = 0; e < 16; e++)
                if (cc + e < d.K)
                    atomicAdd(gw + ((size_t)(cc + e) * 9 + 3 * r + sx) * d.C + c, __uint_as_float(v[e]));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TCOLS)
                     : "memory");
}

template <int KP, int STRIDE>
void launch_wgrad(const ConvDims &d, const __nv_bfloat16 *gb, const __nv_bfloat16 *x, float *gw,
                  int *err, cudaStream_t st) {
    using T = WgTile<STRIDE>;
    const int tiles = div_up(d.Q, 8) * div_up(d.P, 16) * d.N;
    if (tiles <= 0) return;
    const int mtiles = div_up(d.C / 8, kWgGroups), groups = div_up(d.C / 8, mtiles);
    const int a = 3 * groups * T::PXA * 16, stage = a + KP / 8 * T::PXB * 16;
    // the MMAs read 16 planes from the start of a buffer
    const auto bytes = [&](int bufs) { return bufs * stage + imax(0, 16 * T::PXA * 16 - stage); };
    const int tm = 512 / (int)tmem_cols<3 * KP>();  // CTAs an SM by tensor memory
    const int bufs = bytes(3) <= kUmSmemMax / tm ? 3 : 2;
    const int smem = bytes(bufs);
    OF_CUDA(cudaFuncSetAttribute(k_conv_wgrad_mn<KP, STRIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kUmSmemMax));
    // one wave of the CTAs that fit by shared and tensor memory
    const int occ = imax(1, imin(227 * 1024 / (smem + 1024), tm));
    const int splits = imin(tiles, imax(1, kNumSMs * occ / mtiles));
    k_conv_wgrad_mn<KP, STRIDE><<<dim3(mtiles, splits), kWgNT, smem, st>>>(d, gb, x, gw, groups, bufs, err);
}

template <int KP>
void launch_wgrad(const ConvDims &d, const __nv_bfloat16 *gb, const __nv_bfloat16 *x, float *gw,
                  int *err, cudaStream_t st) {
    if (d.stride == 1) launch_wgrad<KP, 1>(d, gb, x, gw, err, st);
    else launch_wgrad<KP, 2>(d, gb, x, gw, err, st);
}

// bf16 copy of the output gradient, zero where the layer's ReLU was inactive
// (the same masking and rounding the mma.sync backward applies on its gather)
__global__ void k_mask_bf16(const float *__restrict__ g, const __nv_bfloat16 *__restrict__ yact,
                            __nv_bfloat16 *out, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        float v = g[i];
        if (yact && !(__bfloat162float(yact[i]) > 0.0f)) v = 0.0f;
        out[i] = __float2bfloat16(v);
    }
}

// The same masked bf16 copy fused with the bias gradient's first stage, for
// K % 4 == 0 (K <= 128): block b covers the gradient rows (output pixels)
// [b * rpb, (b + 1) * rpb); a thread keeps four adjacent channels (one float4
// of a row) and walks R = 256 / (K / 4) rows apart, so each step of the block
// reads whole rows.  The per-thread sums then go, in a fixed order, to one
// partial sum per channel and block: partial[b * K + k].
constexpr int kBiasBlocks = 4 * kNumSMs;
constexpr int kBiasFinalNT = 256;

// Scratch of the backward products, in bytes from its start: the masked bf16
// gradient (rounded up to 64 elements), then the bias partial sums
// (kBiasBlocks x K floats).
size_t bwd_scratch_part(const ConvDims &d) {
    const size_t kp = (size_t)(d.K + 15) / 16 * 16;  // gradient channels padded to 16
    return ((size_t)d.N * d.P * d.Q * kp + 63) / 64 * 64 * sizeof(__nv_bfloat16);
}

__global__ void __launch_bounds__(256) k_mask_bias(const float *__restrict__ g,
                                                   const __nv_bfloat16 *__restrict__ yact,
                                                   __nv_bfloat16 *__restrict__ out, int M, int K,
                                                   int rpb, float *__restrict__ partial) {
    __shared__ float4 sh[256];
    const int Q = K >> 2, R = 256 / Q, t = threadIdx.x;
    const int q = t % Q, ro = t / Q;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (ro < R) {
        const int r0 = blockIdx.x * rpb, r1 = imin(r0 + rpb, M);
        for (int r = r0 + ro; r < r1; r += R) {
            const size_t i = (size_t)r * K + 4 * q;
            float4 v = __ldg(reinterpret_cast<const float4 *>(g + i));
            if (yact) {
                const uint2 a = __ldg(reinterpret_cast<const uint2 *>(yact + i));
                const __nv_bfloat162 a01 = *reinterpret_cast<const __nv_bfloat162 *>(&a.x);
                const __nv_bfloat162 a23 = *reinterpret_cast<const __nv_bfloat162 *>(&a.y);
                if (!(__low2float(a01) > 0.0f)) v.x = 0.0f;
                if (!(__high2float(a01) > 0.0f)) v.y = 0.0f;
                if (!(__low2float(a23) > 0.0f)) v.z = 0.0f;
                if (!(__high2float(a23) > 0.0f)) v.w = 0.0f;
            }
            s.x += v.x;
            s.y += v.y;
            s.z += v.z;
            s.w += v.w;
            const __nv_bfloat162 o01 = __floats2bfloat162_rn(v.x, v.y);
            const __nv_bfloat162 o23 = __floats2bfloat162_rn(v.z, v.w);
            uint2 o;
            o.x = *reinterpret_cast<const uint32_t *>(&o01);
            o.y = *reinterpret_cast<const uint32_t *>(&o23);
            *reinterpret_cast<uint2 *>(out + i) = o;
        }
    }
    sh[t] = s;
    __syncthreads();
    if (t < K) {
        const int qq = t >> 2, e = t & 3;
        float acc = 0.0f;
        for (int j = 0; j < R; j++) {
            const float4 w = sh[j * Q + qq];
            acc += e == 0 ? w.x : e == 1 ? w.y : e == 2 ? w.z : w.w;
        }
        partial[(size_t)blockIdx.x * K + t] = acc;
    }
}

// gb[k] = the sum of the nb partial sums of channel k, one block a channel:
// thread t adds blocks t, t + NT, ... in order, then a fixed tree adds the
// threads' sums.
__global__ void __launch_bounds__(kBiasFinalNT) k_bias_final(const float *__restrict__ partial,
                                                             int nb, int K, float *gb) {
    __shared__ double scratch[kBiasFinalNT / 32];
    const int k = blockIdx.x;
    float acc = 0.0f;
    for (int b = threadIdx.x; b < nb; b += kBiasFinalNT) acc += __ldg(partial + (size_t)b * K + k);
    const double r = block_sum_double<kBiasFinalNT>((double)acc, scratch);
    if (threadIdx.x == 0) gb[k] = (float)r;
}

// Weights in the order of the forward kernel's stages: one 16-byte unit a
// thread, dst[tap][plane of 8 input channels][output channel][8].  Forward:
// w[k][tap][c]; output channels padded to 16 (zeros).  Backward-data seen as a
// forward convolution: rotated taps, input and output channels exchanged, output
// channels in groups of at most 128 one after the other, input channels padded
// to 16 (zeros).
__global__ void k_pack_weights(const __grid_constant__ ConvPack a) {
    const ConvPack::Job &J = a.job[blockIdx.y];
    const int outs = J.backward ? J.C : (J.K + 15) / 16 * 16, planes = (J.backward ? (J.K + 15) / 16 * 16 : J.C) / 8;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < outs * planes * 9; i += gridDim.x * blockDim.x) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (J.backward) {
            const int g = i / (128 * 9 * planes), np = imin(128, outs - 128 * g), e = i - g * (128 * 9 * planes);
            const int c = 128 * g + e % np, pl = (e / np) % planes, tap = e / (np * planes);
            __align__(16) __nv_bfloat16 h[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int k = 8 * pl + q;
                h[q] = k < J.K ? J.w[((size_t)k * 9 + (8 - tap)) * J.C + c] : __float2bfloat16(0.0f);
            }
            v = *reinterpret_cast<const uint4 *>(h);
        } else {
            const int k = i % outs, pl = (i / outs) % planes, tap = i / (outs * planes);
            if (k < J.K) v = *reinterpret_cast<const uint4 *>(J.w + ((size_t)k * 9 + tap) * J.C + 8 * pl);
        }
        reinterpret_cast<uint4 *>(J.dst)[i] = v;
    }
}

// masked bf16 gradient with its K channels padded to Kp (zero): out[m][k]
__global__ void k_mask_pad_bf16(const float *__restrict__ g, const __nv_bfloat16 *__restrict__ yact,
                                int M, int K, int Kp, __nv_bfloat16 *out) {
    const size_t n = (size_t)M * Kp;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t m = i / Kp;
        const int k = (int)(i - m * Kp);
        float v = 0.0f;
        if (k < K) {
            v = g[m * K + k];
            if (yact && !(__bfloat162float(yact[m * K + k]) > 0.0f)) v = 0.0f;
        }
        out[i] = __float2bfloat16(v);
    }
}

}  // namespace

size_t conv_packed_size(int K, int C) { return (size_t)(K + 15) / 16 * 16 * 9 * C; }

void conv_pack_weights(const ConvPack &a, cudaStream_t st) {
    if (a.n > 0) k_pack_weights<<<dim3(32, a.n), 256, 0, st>>>(a);
}

bool conv_forward_umma(const ConvDims &d, const __nv_bfloat16 *x, const __nv_bfloat16 *w,
                       const float *bias, void *y, bool y_f32, bool relu, int *err, cudaStream_t st,
                       int ldy, bool accumulate) {
    if (d.C % 16 != 0 || d.K > 128 || d.K < 1) return false;
    if (accumulate && !y_f32) return false;
    // 16-byte cp.async sources and vector stores
    const auto a16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (!a16(x) || !a16(w) || !a16(y)) return false;
    const int np = (d.K + 15) / 16 * 16;
    const int flags = (relu ? 1 : 0) | (y_f32 ? 2 : 0) | (accumulate ? 4 : 0);
    return dispatch_np(np, UmCall{d, x, w, bias, y, flags, ldy, err, st});
}

bool conv_backward_weight_umma(const ConvDims &d, const float *g, const __nv_bfloat16 *y_act,
                               const __nv_bfloat16 *x, float *gw, float *gb, void *scratch,
                               int *err, cudaStream_t st) {
    if (d.K > 128 || d.K % 8 != 0 || d.C % 16 != 0) return false;
    if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0 || (reinterpret_cast<uintptr_t>(scratch) & 15u) != 0)
        return false;
    const size_t ng = (size_t)d.N * d.P * d.Q * d.K;
    __nv_bfloat16 *gbf = static_cast<__nv_bfloat16 *>(scratch);
    // the masked bf16 copy and the bias gradient in one pass over g where the
    // channels split into float4 quads
    const int M = d.N * d.P * d.Q;
    const bool fused = M > 0 && d.K % 4 == 0 && (reinterpret_cast<uintptr_t>(g) & 15u) == 0 &&
                       (y_act == nullptr || (reinterpret_cast<uintptr_t>(y_act) & 7u) == 0);
    if (fused) {
        const int R = 256 / (d.K / 4);
        const int rpb = div_up(div_up(M, imin(kBiasBlocks, imax(1, div_up(M, 4 * R)))), R) * R;
        const int nb = div_up(M, rpb);
        float *part = reinterpret_cast<float *>(static_cast<char *>(scratch) + bwd_scratch_part(d));
        k_mask_bias<<<nb, 256, 0, st>>>(g, y_act, gbf, M, d.K, rpb, part);
        k_bias_final<<<d.K, kBiasFinalNT, 0, st>>>(part, nb, d.K, gb);
    } else {
        k_mask_bf16<<<imin((int)((ng + 255) / 256), 4096), 256, 0, st>>>(g, y_act, gbf, ng);
    }
    OF_CUDA(cudaMemsetAsync(gw, 0, sizeof(float) * (size_t)d.K * 9 * d.C, st));
    switch ((d.K + 15) / 16 * 16) {
        case 16: launch_wgrad<16>(d, gbf, x, gw, err, st); break;
        case 32: launch_wgrad<32>(d, gbf, x, gw, err, st); break;
        case 48: launch_wgrad<48>(d, gbf, x, gw, err, st); break;
        case 64: launch_wgrad<64>(d, gbf, x, gw, err, st); break;
        case 80: launch_wgrad<80>(d, gbf, x, gw, err, st); break;
        case 96: launch_wgrad<96>(d, gbf, x, gw, err, st); break;
        case 112: launch_wgrad<112>(d, gbf, x, gw, err, st); break;
        default: launch_wgrad<128>(d, gbf, x, gw, err, st); break;
    }
    if (!fused) conv_bias_grad(d, g, y_act, gb, st);
    return true;
}

size_t conv_backward_data_umma_scratch(const ConvDims &d) {
    return bwd_scratch_part(d) + sizeof(float) * kBiasBlocks * (size_t)d.K;
}

bool conv_backward_data_umma(const ConvDims &d, const float *g, const __nv_bfloat16 *y_act,
                             const __nv_bfloat16 *w, float *gin, bool accumulate, void *scratch,
                             int *err, cudaStream_t st, bool g_masked) {
    if (d.K % 8 != 0 || d.C % 16 != 0) return false;
    if ((reinterpret_cast<uintptr_t>(gin) & 15u) != 0) return false;
    // the gradient's channels are the product's input channels: padded to a
    // multiple of 16 (zero channels, zero weights) where K is not one
    const int Kp = (d.K + 15) / 16 * 16;
    const int M = d.N * d.P * d.Q;
    const size_t ng = (size_t)M * Kp;
    __nv_bfloat16 *gb = static_cast<__nv_bfloat16 *>(scratch);
    if (Kp != d.K)
        k_mask_pad_bf16<<<imin((int)((ng + 255) / 256), 4096), 256, 0, st>>>(g, y_act, M, d.K, Kp, gb);
    else if (!g_masked)
        k_mask_bf16<<<imin((int)((ng + 255) / 256), 4096), 256, 0, st>>>(g, y_act, gb, ng);
    // the product as a forward convolution over the output gradient: input
    // (N, P, Q, Kp), output (N, H, W, C); stride 2 layers read a dilated input
    ConvDims t{d.N, d.P, d.Q, Kp, d.H, d.W, 0, d.stride == 1 ? 1 : -2};
    for (int c0 = 0; c0 < d.C; c0 += 128) {  // at most 128 output channels a launch
        t.K = imin(128, d.C - c0);
        if (!conv_forward_umma(t, gb, w + (size_t)c0 * 9 * Kp, nullptr, gin + c0, true, false, err,
                               st, d.C, accumulate))
            return false;
    }
    return true;
}

}  // namespace oflow
