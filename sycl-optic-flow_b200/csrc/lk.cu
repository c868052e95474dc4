// Lucas-Kanade on B200: the reference's single-step solver over a frame ring
// (src/lk/cuda/lucaskanade.cu:54-71, kernels/kernels.cu:14-181) as one fused
// kernel, and a pyramidal, iterated variant built from the same steps.  The
// arithmetic contract is in common.cuh.
//
// The five window sums are accumulated per pixel in the reference's order
// (window rows, then columns), read from shared memory; a prefix-sum or
// separable box filter would change the rounding of det(A) and with it the
// flow wherever the structure tensor is near singular.
#include "common.cuh"
#include "hs.hpp"
#include "internal.hpp"
#include "lk.hpp"
#include "tvl1.hpp"

namespace oflow {

constexpr int kLTile = 32;  // pixels a side of a block's tile
constexpr int kLMaxC = 4, kLMaxT = 9;

struct LkTaps {
    float fs[9];
    float ft[9];
    int ns, nt;
};

int lk_taps(int spac, int temp, float *fs, float *ft) {
    static const float s1[] = {1.0f};
    static const float s3[] = {-1.0f / 2.0f, 0.0f, 1.0f / 2.0f};
    static const float s5[] = {1.0f / 12.0f, -2.0f / 3.0f, 0.0f, 2.0f / 3.0f, -1.0f / 12.0f};
    static const float s7[] = {-1.0f / 60.0f, 3.0f / 20.0f, -3.0f / 4.0f, 0.0f,
                               3.0f / 4.0f,   -3.0f / 20.0f, 1.0f / 60.0f};
    static const float s9[] = {1.0f / 280.0f, -4.0f / 105.0f, 1.0f / 5.0f, -4.0f / 5.0f, 0.0f,
                               4.0f / 5.0f,   -1.0f / 5.0f,   4.0f / 105.0f, -1.0f / 280.0f};
    static const float t2[] = {-1.0f, 1.0f};
    // central-difference tables of src/lk/cuda/lucaskanade.cu:79-161
    const float *S = spac == 1 ? s1 : spac == 3 ? s3 : spac == 5 ? s5 : spac == 7 ? s7
                                                                                    : spac == 9 ? s9 : nullptr;
    const float *T = temp == 1 ? s1 : temp == 2 ? t2 : temp == 3 ? s3 : temp == 5 ? s5
                                                                                   : temp == 7 ? s7
                                                                                               : temp == 9 ? s9
                                                                                                           : nullptr;
    if (!S || !T) return -1;
    for (int i = 0; i < spac; i++) fs[i] = S[i];
    for (int i = 0; i < temp; i++) ft[i] = T[i];
    return 0;
}

// Window sums and the closed-form 2x2 solve (kernels.cu:150-179) of 2 x PY
// pixels: two columns from col (even), rows of centres from row.  gx/gy/gt are
// region planes of RW columns in shared memory, the window of pixel (0, 0)
// starting at (row, col).  Each window element is loaded and its five products
// formed once for all pixels whose window holds it; each pixel still adds them
// in the reference's row-major order.
//
// The additions are 5 (2C+1)^2 a pixel and cannot be shared (a prefix sum or a
// separable box would round differently); eight pixels a thread leave 30
// multiplications and 9 shared loads a pixel at C = 2, where four in one column
// took 50 and 30.
template <int C, int PY>
__device__ __forceinline__ void lk_window_solve(const float *gx, const float *gy, const float *gt, int RW,
                                                int row, int col, float (&vx)[PY][2], float (&vy)[PY][2]) {
    float sxx[PY][2], sxy[PY][2], syy[PY][2], sxt[PY][2], syt[PY][2];
#pragma unroll
    for (int k = 0; k < PY; k++)
#pragma unroll
        for (int m = 0; m < 2; m++) sxx[k][m] = sxy[k][m] = syy[k][m] = sxt[k][m] = syt[k][m] = 0.0f;
#pragma unroll
    for (int r = 0; r < 2 * C + PY; r++) {
        const int at = (row + r) * RW + col;
        float ix[2 * C + 2], iy[2 * C + 2], it[2 * C + 2];
#pragma unroll
        for (int j = 0; j < C + 1; j++) {
            const float2 a = *reinterpret_cast<const float2 *>(gx + at + 2 * j);
            const float2 b = *reinterpret_cast<const float2 *>(gy + at + 2 * j);
            const float2 t = *reinterpret_cast<const float2 *>(gt + at + 2 * j);
            ix[2 * j] = a.x; ix[2 * j + 1] = a.y;
            iy[2 * j] = b.x; iy[2 * j + 1] = b.y;
            it[2 * j] = t.x; it[2 * j + 1] = t.y;
        }
#pragma unroll
        for (int j = 0; j < 2 * C + 2; j++) {
            const float pxx = ix[j] * ix[j], pxy = ix[j] * iy[j], pyy = iy[j] * iy[j], pxt = ix[j] * it[j],
                        pyt = iy[j] * it[j];
#pragma unroll
            for (int k = 0; k < PY; k++)
#pragma unroll
                for (int m = 0; m < 2; m++)
                    if (r - k >= 0 && r - k <= 2 * C && j - m >= 0 && j - m <= 2 * C) {
                        sxx[k][m] += pxx;
                        sxy[k][m] += pxy;
                        syy[k][m] += pyy;
                        sxt[k][m] += pxt;
                        syt[k][m] += pyt;
                    }
        }
    }
#pragma unroll
    for (int k = 0; k < PY; k++)
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const float det = (sxx[k][m] * syy[k][m] - sxy[k][m] * sxy[k][m]);
            vx[k][m] = 0.0f;
            vy[k][m] = 0.0f;
            if (det != 0.0f) {
                const float inv = 1.0f / det;
                vx[k][m] = inv * (syy[k][m] * (-sxt[k][m]) + (-sxy[k][m]) * (-syt[k][m]));
                vy[k][m] = inv * ((-sxy[k][m]) * (-sxt[k][m]) + sxx[k][m] * (-syt[k][m]));
            }
        }
}

// Visits the RW x RH region with NT threads, rows by warps, without divisions
// for the first 32 columns.
template <int NT, int RW, int RH, typename F> __device__ __forceinline__ void for_region(F &&f) {
    constexpr int NWARP = NT / 32, X = RW - 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll 4
    for (int ry = wid; ry < RH; ry += NWARP) f(lane, ry);
    if (X > 0)
        for (int i = threadIdx.x; i < X * RH; i += NT) f(32 + i % imax(X, 1), i / imax(X, 1));
}

// Single step over T uint8 frames in temporal order (src[0] the oldest), read
// where they lie.  One kernel: spatial FIR of the oldest frame, temporal FIR,
// window sums and solve.  Pixels closer than the window radius to the border
// get 0.  The five frames of a 1280x720 step used to be copied into the plan and
// the flow out of it (31 of 96 us), and the sums ran one pixel a thread (65 us);
// with four pixels a thread the whole step takes 26.6 us (with eight 27.7, with
// fewer blocks in flight).
struct LkStep {
    const uint8_t *src[kLMaxT];
    long long pitch[kLMaxT];
    int T, nx, ny;
    LkTaps taps;
    float *u, *v;
    long long out_pitch;
};
template <int C, int NS, int PY>
__global__ void __launch_bounds__(kLTile *kLTile / (2 * PY)) k_lk_step(const __grid_constant__ LkStep a) {
    constexpr int NT = kLTile * kLTile / (2 * PY), F = (NS - 1) / 2;
    constexpr int RW = kLTile + 2 * C, FW = RW + 2 * F;
    __shared__ float sf[FW * FW];
    __shared__ __align__(8) float gx[RW * RW], gy[RW * RW], gt[RW * RW];
    const int nx = a.nx, ny = a.ny;
    const int x0 = blockIdx.x * kLTile - C, y0 = blockIdx.y * kLTile - C;
    const uint8_t *old = a.src[0];
    for_region<NT, FW, FW>([&](int rx, int ry) {
        const int x = x0 - F + rx, y = y0 - F + ry;
        sf[ry * FW + rx] = (x >= 0 && x < nx && y >= 0 && y < ny) ? (float)__ldg(old + (size_t)y * a.pitch[0] + x) : 0.0f;
    });
    __syncthreads();
    for_region<NT, RW, RW>([&](int rx, int ry) {
        const int x = x0 + rx, y = y0 + ry;
        if (x < 0 || x >= nx || y < 0 || y >= ny) {
            // read only by the sums of border pixels, whose results are not used
            gx[ry * RW + rx] = gy[ry * RW + rx] = gt[ry * RW + rx] = 0.0f;
            return;
        }
        const float *f = sf + (ry + F) * FW + rx + F;
        float ax = 0.0f, ay = 0.0f;
#pragma unroll
        for (int k = 0; k < NS; k++) {
            const int xx = x + k - F, yy = y + k - F;
            if (xx >= 0 && xx < nx) ax += f[k - F] * a.taps.fs[k];
            if (yy >= 0 && yy < ny) ay += f[(k - F) * FW] * a.taps.fs[k];
        }
        float at = 0.0f;
        for (int k = 0; k < a.T; k++) at += a.taps.ft[k] * (float)__ldg(a.src[k] + (size_t)y * a.pitch[k] + x);
        gx[ry * RW + rx] = ax;
        gy[ry * RW + rx] = ay;
        gt[ry * RW + rx] = at;
    });
    __syncthreads();
    const int tx = 2 * (threadIdx.x % (kLTile / 2)), ty = (threadIdx.x / (kLTile / 2)) * PY;
    const int x = blockIdx.x * kLTile + tx, yb = blockIdx.y * kLTile + ty;
    if (x >= nx || yb >= ny) return;
    float dx[PY][2], dy[PY][2];
    lk_window_solve<C, PY>(gx, gy, gt, RW, ty, tx, dx, dy);
#pragma unroll
    for (int k = 0; k < PY; k++)
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int xx = x + m, y = yb + k;
            if (xx >= nx || y >= ny) continue;
            const bool in = xx >= C && y >= C && xx < nx - C && y < ny - C;
            a.u[(size_t)y * a.out_pitch + xx] = in ? dx[k][m] : 0.0f;
            a.v[(size_t)y * a.out_pitch + xx] = in ? dy[k][m] : 0.0f;
        }
}

// Rows a thread in launches that fill the GPU: two where the windows are wide and
// the blocks' shared memory with them, else four, whose windows share more
// (1920x1080, 9x9: 69.6 us with two, 77.0 with four; 5x5: 32.4 and 31.4).
template <int C, int NS> static void lk_step_launch(const LkStep &a, cudaStream_t st) {
    constexpr int PY = C > 2 ? 2 : 4;
    const dim3 g(div_up(a.nx, kLTile), div_up(a.ny, kLTile));
    if ((size_t)g.x * g.y > 4 * (size_t)kNumSMs)
        k_lk_step<C, NS, PY><<<g, kLTile * kLTile / (2 * PY), 0, st>>>(a);
    else
        k_lk_step<C, NS, 1><<<g, kLTile * kLTile / 2, 0, st>>>(a);
}
template <int C> static void lk_step_launch_c(const LkStep &a, cudaStream_t st) {
    switch (a.taps.ns) {
        case 1: lk_step_launch<C, 1>(a, st); break;
        case 3: lk_step_launch<C, 3>(a, st); break;
        case 5: lk_step_launch<C, 5>(a, st); break;
        case 7: lk_step_launch<C, 7>(a, st); break;
        default: lk_step_launch<C, 9>(a, st); break;
    }
}

// Spatial FIR (zero padding by dropped taps) of a float plane -> float2 (Ix, Iy),
// NS taps at compile time (every tap added, the zero one too, as the
// reference does); pixels at least NS/2 from every border skip the tests.
template <int NS>
__global__ void k_lk_grad(const float *__restrict__ src, size_t sstride, int nx, int ny,
                          const __grid_constant__ LkTaps taps, float2 *G, size_t gstride) {
    constexpr int FC = (NS - 1) / 2;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= nx || y >= ny) return;
    const float *f = src + (size_t)blockIdx.z * sstride;
    float ax = 0.0f, ay = 0.0f;
    if (x >= FC && x < nx - FC && y >= FC && y < ny - FC) {
        const float *row = f + (size_t)y * nx + x - FC, *col = f + (size_t)(y - FC) * nx + x;
#pragma unroll
        for (int k = 0; k < NS; k++) {
            ax += __ldg(row + k) * taps.fs[k];
            ay += __ldg(col + (size_t)k * nx) * taps.fs[k];
        }
    } else {
#pragma unroll
        for (int k = 0; k < NS; k++) {
            const int xx = x + k - FC, yy = y + k - FC;
            if (xx >= 0 && xx < nx) ax += __ldg(f + (size_t)y * nx + xx) * taps.fs[k];
            if (yy >= 0 && yy < ny) ay += __ldg(f + (size_t)yy * nx + x) * taps.fs[k];
        }
    }
    G[(size_t)blockIdx.z * gstride + (size_t)y * nx + x] = make_float2(ax, ay);
}

// The same for rows of whole aligned quads: four pixels a thread, the vertical
// taps and the results as vectors (64 pairs of 640x480 and two coarser levels:
// 109 -> 67 us).  Quads whose taps leave the image take k_lk_grad's sums.
template <int NS>
__global__ void k_lk_grad4(const float *__restrict__ src, size_t sstride, int nx, int ny,
                           const __grid_constant__ LkTaps taps, float2 *G, size_t gstride) {
    constexpr int FC = (NS - 1) / 2;
    const int x = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= nx || y >= ny) return;
    const float *f = src + (size_t)blockIdx.z * sstride;
    float ax[4] = {0.0f, 0.0f, 0.0f, 0.0f}, ay[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (x >= FC && x + 3 < nx - FC && y >= FC && y < ny - FC) {
        const float *row = f + (size_t)y * nx + x - FC, *col = f + (size_t)(y - FC) * nx + x;
        float r[4 + 2 * FC];
#pragma unroll
        for (int k = 0; k < 4 + 2 * FC; k++) r[k] = __ldg(row + k);
#pragma unroll
        for (int k = 0; k < NS; k++) {
            const float4 c = __ldg(reinterpret_cast<const float4 *>(col + (size_t)k * nx));
            const float cc[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
            for (int m = 0; m < 4; m++) {
                ax[m] += r[m + k] * taps.fs[k];
                ay[m] += cc[m] * taps.fs[k];
            }
        }
    } else {
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int k = 0; k < NS; k++) {
                const int xx = x + m + k - FC, yy = y + k - FC;
                if (xx >= 0 && xx < nx) ax[m] += __ldg(f + (size_t)y * nx + xx) * taps.fs[k];
                if (yy >= 0 && yy < ny) ay[m] += __ldg(f + (size_t)yy * nx + x + m) * taps.fs[k];
            }
    }
    float4 *o = reinterpret_cast<float4 *>(G + (size_t)blockIdx.z * gstride + (size_t)y * nx + x);
    o[0] = make_float4(ax[0], ay[0], ax[1], ay[1]);
    o[1] = make_float4(ax[2], ay[2], ax[3], ay[3]);
}

static void launch_lk_grad(dim3 g, dim3 blk, cudaStream_t st, const float *src, size_t sstride,
                           int nx, int ny, const LkTaps &taps, float2 *G, size_t gstride) {
    // planes start at multiples of sstride / gstride elements of 256-byte aligned buffers
    if (nx % 4 == 0 && sstride % 4 == 0 && gstride % 2 == 0 && reinterpret_cast<uintptr_t>(src) % 16 == 0) {
        const dim3 g4(div_up(nx, 32 * 4), g.y, g.z);
        switch (taps.ns) {
            case 1: k_lk_grad4<1><<<g4, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
            case 3: k_lk_grad4<3><<<g4, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
            case 5: k_lk_grad4<5><<<g4, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
            case 7: k_lk_grad4<7><<<g4, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
            default: k_lk_grad4<9><<<g4, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
        }
        return;
    }
    switch (taps.ns) {
        case 1: k_lk_grad<1><<<g, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
        case 3: k_lk_grad<3><<<g, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
        case 5: k_lk_grad<5><<<g, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
        case 7: k_lk_grad<7><<<g, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
        default: k_lk_grad<9><<<g, blk, 0, st>>>(src, sstride, nx, ny, taps, G, gstride); break;
    }
}

// It, Ix, Iy of up to M pixels of a region into its shared planes: the flows of
// all of them are loaded first, then all their samples of I1 (bilinear,
// clamp-to-edge; the few whose taps leave the image go through
// bilinear_clamped afterwards), so that a thread's gathers are in flight
// together.  on[m] false: no such pixel.
template <int M>
__device__ __forceinline__ void lk_warp_pixels(const int (&rx)[M], const int (&ry)[M], const bool (&on)[M], int x0, int y0,
                                               int RW, const float *__restrict__ I0, const float *__restrict__ I1,
                                               const float2 *__restrict__ G, const float2 *__restrict__ U, int nx,
                                               int ny, float *gx, float *gy, float *gt) {
    unsigned q[M], base[M];  // (more pixels than these count don't fit the device's memory)
    bool in[M], easy[M];
    float2 u[M], g[M];
    float i0[M], xf[M], yf[M], v00[M], v10[M], v01[M], v11[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int x = x0 + rx[m], y = y0 + ry[m];
        in[m] = on[m] && x >= 0 && x < nx && y >= 0 && y < ny;
        q[m] = in[m] ? (unsigned)y * (unsigned)nx + (unsigned)x : 0;
        u[m] = U[q[m]];
        xf[m] = (float)x;
        yf[m] = (float)y;
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        g[m] = G[q[m]];
        i0[m] = __ldg(I0 + q[m]);
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        xf[m] += u[m].x;
        yf[m] += u[m].y;
        easy[m] = xf[m] >= 0.0f && yf[m] >= 0.0f && xf[m] < (float)(nx - 1) && yf[m] < (float)(ny - 1);
        base[m] = easy[m] ? (unsigned)yf[m] * (unsigned)nx + (unsigned)xf[m] : 0;  // (nonnegative: truncation is floor)
        const float *p = I1 + base[m];
        v00[m] = __ldg(p);
        v10[m] = __ldg(p + 1);
        v01[m] = __ldg(p + nx);
        v11[m] = __ldg(p + nx + 1);
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        const float fx = xf[m] - (float)(int)xf[m], fy = yf[m] - (float)(int)yf[m];
        const float ex = 1.0f - fx, ey = 1.0f - fy;
        const float top = ex * v00[m] + fx * v10[m];
        const float bot = ex * v01[m] + fx * v11[m];
        float w = ey * top + fy * bot;
        if (!easy[m]) w = bilinear_clamped(I1, nx, ny, xf[m], yf[m]);
        float it = 0.0f;
        it += -1.0f * i0[m];
        it += 1.0f * w;
        if (on[m]) {
            // outside the image: read only by the sums of border pixels, whose results are not used
            const int i = ry[m] * RW + rx[m];
            gx[i] = in[m] ? g[m].x : 0.0f;
            gy[i] = in[m] ? g[m].y : 0.0f;
            gt[i] = in[m] ? it : 0.0f;
        }
    }
}

// One refinement of pyramidal LK: warp I1 by the current flow (bilinear,
// clamp-to-edge), It = 0 + (-1)*I0 + 1*I1w, window solve, Uout = Uin + d.
// Tile 32 x 32 with the window radius C as halo; a thread solves two columns of
// PY rows (lk_window_solve): 4 when a launch has tiles enough to fill the GPU,
// else 1 (four times the threads).  64 pairs of 640x480, three levels of three
// refinements at C = 2: 1.05 ms of launches (1.24 with one pixel a thread and
// its gathers one after the other); issue slots 79 % used, the additions bound it.
template <int C, int PY>
__global__ void __launch_bounds__(kLTile *kLTile / (2 * PY)) k_pyrlk_iter(
    const float *__restrict__ pyr, size_t lp, const float2 *__restrict__ G, size_t gstride,
    const float2 *__restrict__ Uin, float2 *Uout, size_t ustride, int nx, int ny,
    const OutRef *__restrict__ outs) {
    constexpr int NT = kLTile * kLTile / (2 * PY), RW = kLTile + 2 * C;
    __shared__ __align__(8) float gx[RW * RW], gy[RW * RW], gt[RW * RW];
    const int b = blockIdx.z;
    const float *I0 = pyr + (size_t)(2 * b) * lp;
    const float *I1 = pyr + (size_t)(2 * b + 1) * lp;
    const float2 *Gb = G + (size_t)b * gstride;
    const float2 *Ub = Uin + (size_t)b * ustride;
    const int x0 = blockIdx.x * kLTile - C, y0 = blockIdx.y * kLTile - C;
    {
        // rows by warps, three at a time, then the columns beyond the 32nd
        constexpr int M = 3, NWARP = NT / 32, X = RW - 32;
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        int rx[M], ry[M];
        bool on[M];
#pragma unroll 1
        for (int r = wid; r < RW; r += M * NWARP) {
#pragma unroll
            for (int m = 0; m < M; m++) {
                rx[m] = lane;
                ry[m] = r + m * NWARP;
                on[m] = ry[m] < RW;
            }
            lk_warp_pixels<M>(rx, ry, on, x0, y0, RW, I0, I1, Gb, Ub, nx, ny, gx, gy, gt);
        }
        if (X > 0)
#pragma unroll 1
            for (int i = threadIdx.x; i < X * RW; i += M * NT) {
#pragma unroll
                for (int m = 0; m < M; m++) {
                    const int k = i + m * NT;
                    on[m] = k < X * RW;
                    rx[m] = 32 + k % imax(X, 1);
                    ry[m] = k / imax(X, 1);
                }
                lk_warp_pixels<M>(rx, ry, on, x0, y0, RW, I0, I1, Gb, Ub, nx, ny, gx, gy, gt);
            }
    }
    __syncthreads();
    const int tx = 2 * (threadIdx.x % (kLTile / 2)), ty = (threadIdx.x / (kLTile / 2)) * PY;
    const int x = blockIdx.x * kLTile + tx, yb = blockIdx.y * kLTile + ty;
    if (x >= nx || yb >= ny) return;
    float dx[PY][2], dy[PY][2];
    lk_window_solve<C, PY>(gx, gy, gt, RW, ty, tx, dx, dy);
    OutRef o{nullptr, nullptr, 0};
    if (outs) o = outs[b];
#pragma unroll
    for (int k = 0; k < PY; k++)
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int xx = x + m, y = yb + k;
            if (xx >= nx || y >= ny) continue;
            const bool in = xx >= C && y >= C && xx < nx - C && y < ny - C;
            const size_t q = (size_t)y * nx + xx;
            const float2 u = Ub[q];
            const float2 r = make_float2(u.x + (in ? dx[k][m] : 0.0f), u.y + (in ? dy[k][m] : 0.0f));
            if (outs) {  // the solve's last refinement writes the caller's planes
                o.u[(size_t)y * o.pitch + xx] = r.x;
                o.v[(size_t)y * o.pitch + xx] = r.y;
            } else {
                Uout[(size_t)b * ustride + q] = r;
            }
        }
}

static void launch_pyrlk_iter(int c, dim3 g, cudaStream_t st, const float *pyr, size_t lp,
                              const float2 *G, size_t gstride, const float2 *Uin, float2 *Uout,
                              size_t ustride, int nx, int ny, const OutRef *outs) {
    const bool wide = (size_t)g.x * g.y * g.z > 4 * (size_t)kNumSMs;
#define OF_PYRLK(C)                                                                                  \
    if (wide)                                                                                        \
        k_pyrlk_iter<C, 4><<<g, kLTile * kLTile / 8, 0, st>>>(pyr, lp, G, gstride, Uin, Uout, ustride, nx, ny, outs); \
    else                                                                                             \
        k_pyrlk_iter<C, 1><<<g, kLTile * kLTile / 2, 0, st>>>(pyr, lp, G, gstride, Uin, Uout, ustride, nx, ny, outs);
    switch (c) {
        case 0: OF_PYRLK(0) break;
        case 1: OF_PYRLK(1) break;
        case 2: OF_PYRLK(2) break;
        case 3: OF_PYRLK(3) break;
        default: OF_PYRLK(4) break;
    }
#undef OF_PYRLK
}

// ================================================================ host plans
static LkTaps make_lk_taps(int spac, int temp) {
    LkTaps t{};
    if (lk_taps(spac, temp, t.fs, t.ft) != 0) throw Error(OFLOW_ERR_BAD_ARG, "lk: filter size not supported");
    t.ns = spac;
    t.nt = temp;
    return t;
}

LkPlan::LkPlan(int w, int h, const oflow_lk_params &prm) : w_(w), h_(h), prm_(prm) {
    OF_CHECK(prm.window >= 1 && (prm.window & 1) && (prm.window - 1) / 2 <= kLMaxC,
             "lk: window must be odd and at most 9");
    OF_CHECK(prm.temp >= 1 && prm.temp <= kLMaxT, "lk: temporal filter size out of range");
    make_lk_taps(prm.spac, prm.temp);
    OF_CHECK(w >= prm.window && h >= prm.window && w >= prm.spac && h >= prm.spac,
             "lk: frame smaller than the window or filter");
    N_ = (size_t)w * h;
    o_ring_ = ar_.reserve((size_t)prm.temp * N_);
    o_out_ = ar_.reserve(2 * N_ * 4);
    ar_.commit();
}

uint8_t *LkPlan::ring_slot(int k) const { return ar_.at<uint8_t>(o_ring_) + (size_t)k * N_; }
float *LkPlan::out_u() const { return ar_.at<float>(o_out_); }
float *LkPlan::out_v() const { return ar_.at<float>(o_out_) + N_; }

void LkPlan::run(const FrameRef *ring, int iframe, const OutRef &out, cudaStream_t st) {
    LkStep a{};
    a.T = prm_.temp;
    for (int k = 0; k < a.T; k++) {  // temporal order: the slot after the newest frame's is the oldest
        const FrameRef &f = ring[(k + iframe + 1) % a.T];
        a.src[k] = static_cast<const uint8_t *>(f.p);
        a.pitch[k] = f.pitch;
    }
    a.nx = w_;
    a.ny = h_;
    a.taps = make_lk_taps(prm_.spac, prm_.temp);
    a.u = out.u;
    a.v = out.v;
    a.out_pitch = out.pitch;
    switch ((prm_.window - 1) / 2) {
        case 0: lk_step_launch_c<0>(a, st); break;
        case 1: lk_step_launch_c<1>(a, st); break;
        case 2: lk_step_launch_c<2>(a, st); break;
        case 3: lk_step_launch_c<3>(a, st); break;
        default: lk_step_launch_c<4>(a, st); break;
    }
    OF_CUDA(cudaGetLastError());
}

PyrLkPlan::PyrLkPlan(int w, int h, int B, int dtype, const oflow_lk_params &prm)
    : w_(w), h_(h), B_(B), dtype_(dtype), prm_(prm) {
    OF_CHECK(B >= 1, "pyrlk: empty batch");
    OF_CHECK(prm.window >= 1 && (prm.window & 1) && (prm.window - 1) / 2 <= kLMaxC,
             "pyrlk: window must be odd and at most 9");
    OF_CHECK(prm.levels >= 1 && prm.levels <= 16, "pyrlk: levels out of range");
    OF_CHECK(prm.iters >= 0, "pyrlk: iters < 0");
    make_lk_taps(prm.spac, 2);
    taps_ = make_zoom_taps(0.5f);
    L_ = prm.levels;
    W_[0] = w;
    H_[0] = h;
    for (int l = 1; l < L_; l++) tvl1_zoom_size(W_[l - 1], H_[l - 1], &W_[l], &H_[l], 0.5f);
    for (int l = 0; l + 1 < L_; l++)
        OF_CHECK(taps_.size <= W_[l] && taps_.size <= H_[l], "pyrlk: level smaller than the Gaussian window");
    for (int l = 0; l < L_; l++)
        OF_CHECK(W_[l] >= prm.window && H_[l] >= prm.window, "pyrlk: level smaller than the window");
    N_ = (size_t)w * h;
    size_t acc = 0;
    for (int l = 0; l < L_; l++) {
        pyr_off_[l] = acc;
        acc += (size_t)2 * B * W_[l] * H_[l];
    }
    const size_t esz = dtype == OFLOW_U8 ? 1 : 4;
    o_raw_ = ar_.reserve(2 * B * N_ * esz);
    o_T_ = ar_.reserve(2 * B * N_ * 4);
    o_pyr_ = ar_.reserve(acc * 4);
    o_G_ = ar_.reserve(B * N_ * 8);
    o_U0_ = ar_.reserve(B * N_ * 8);
    o_U1_ = ar_.reserve(B * N_ * 8);
    o_out_ = ar_.reserve(2 * B * N_ * 4);
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
}

void PyrLkPlan::bind_frame(int b, int k, const void *p, int pitch) { io_.set_frame(b, k, p, pitch ? pitch : w_); }
void PyrLkPlan::bind_raw(int b, int k) { io_.set_frame(b, k, raw_input(b, k), w_); }
void PyrLkPlan::bind_out(int b, float *u, float *v, int pitch) { io_.set_out(b, u, v, pitch ? pitch : w_); }
void PyrLkPlan::bind_own_out(int b) {
    float *o = ar_.at<float>(o_out_);
    io_.set_out(b, o + (size_t)b * N_, o + (size_t)(B_ + b) * N_, w_);
}

void *PyrLkPlan::raw_input(int b, int k) const {
    const size_t esz = dtype_ == OFLOW_U8 ? 1 : 4;
    return ar_.at<char>(o_raw_) + (size_t)(2 * b + k) * N_ * esz;
}
const float *PyrLkPlan::out_u(int b) const { return ar_.at<float>(o_out_) + (size_t)b * N_; }
const float *PyrLkPlan::out_v(int b) const { return ar_.at<float>(o_out_) + (size_t)(B_ + b) * N_; }

void PyrLkPlan::record(cudaStream_t st) {
    const int B = B_;
    float *pyr = ar_.at<float>(o_pyr_);
    float *T = ar_.at<float>(o_T_);
    float2 *G = ar_.at<float2>(o_G_);
    float2 *U[2] = {ar_.at<float2>(o_U0_), ar_.at<float2>(o_U1_)};
    const LkTaps taps = make_lk_taps(prm_.spac, 2);
    // frames through the frame table (device frames in place, or staged)
    launch_ingest_tab(io_.frames(), dtype_, w_, h_, pyr, N_, 2 * B, st);
    for (int l = 1; l < L_; l++) {
        const size_t sp = (size_t)W_[l - 1] * H_[l - 1], dp = (size_t)W_[l] * H_[l];
        launch_zoom_out(pyr + pyr_off_[l - 1], sp, W_[l - 1], H_[l - 1], T, pyr + pyr_off_[l], dp,
                        W_[l], H_[l], 0.5f, taps_, 2 * B, st);
    }
    int cur = 0;
    OF_CUDA(cudaMemsetAsync(U[cur], 0, B * N_ * 8, st));
    const int c = (prm_.window - 1) / 2;
    for (int l = L_ - 1; l >= 0; l--) {
        const int lw = W_[l], lh = H_[l];
        const size_t lp = (size_t)lw * lh;
        dim3 blk(32, 8), g(div_up(lw, 32), div_up(lh, 8), B);
        // Ix, Iy of I0: plane 2b of the level, so a stride of two planes
        launch_lk_grad(g, blk, st, pyr + pyr_off_[l], 2 * lp, lw, lh, taps, G, N_);
        dim3 ig(div_up(lw, kLTile), div_up(lh, kLTile), B);
        for (int r = 0; r < prm_.iters; r++) {
            const bool end = l == 0 && r + 1 == prm_.iters;
            launch_pyrlk_iter(c, ig, st, pyr + pyr_off_[l], lp, G, N_, U[cur], U[cur ^ 1], N_, lw, lh,
                              end ? io_.outs() : nullptr);
            cur ^= 1;
        }
        if (l > 0) {
            const float sx = (float)W_[l - 1] / (float)lw;
            const float sy = (float)H_[l - 1] / (float)lh;
            launch_upscale2(U[cur], N_, lw, lh, U[cur ^ 1], N_, W_[l - 1], H_[l - 1], sx, sy, B, st);
            cur ^= 1;
        }
    }
    if (prm_.iters == 0) launch_split_tab(U[cur], N_, w_, h_, io_.outs(), B, st);
    OF_CUDA(cudaGetLastError());
}

void PyrLkPlan::run(cudaStream_t st) {
    io_.upload(st);
    if (!graph_.ready()) graph_.capture(st, [&](cudaStream_t s) { record(s); });
    graph_.launch(st);
}

}  // namespace oflow
