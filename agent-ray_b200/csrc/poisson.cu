// Screened-Poisson reconstruction for the gradient-domain tracer
// (screened_poisson_reconstruct, src/integrators/gradient_domain_pt.rs:449-630).
//
// System per colour channel (5-point stencil, Neumann borders):
//   (alpha + N(x)) I(x) - sum_{n in N(x)} I(n) = alpha * primal(x) + div G(x)
// (the reference's sign; AR_GDPT_CONSISTENT_DIVERGENCE subtracts div G instead)
//
// Two solvers:
//   * red-black SOR, the reference method: each half sweep updates one colour
//     of the checkerboard, whose neighbours all have the other colour, so the
//     sweep is order independent and matches the sequential loop bit for bit
//     (this file is compiled with -fmad=false);
//   * FP32 conjugate gradient with FP64 iterative refinement: the residual
//     r = b - A x and all dot products are accumulated in FP64, the correction
//     A d = r is solved in FP32 CG, and x (FP64) += d until ||r|| / ||b|| <= tol.
// Buffers are interleaved RGB (W*H*3), like Film::to_hdr_vec.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <utility>
#include <vector>

#include "ar_render.hpp"

namespace ar {

namespace {

// Launches `kernel` so that it is set up while the kernel before it on the stream
// still drains; it begins with after_previous(), which returns once all earlier
// work of the stream is complete and visible.  A solve is a chain of short kernels
// (128 of 5 to 14 us for 64 iterations of conjugate gradient), and launch and ramp-up
// were up to a third of it.  Unchained -> chained: conjugate gradient to 1e-6, 256^2
// 919 -> 609 us, 511x513 1191 -> 889, 512^2 1148 -> 828, 1024^2 2124 -> 1832; 200
// iterations of SOR, 64^2 284 -> 234, 256^2 299 -> 259, 512^2 456 -> 370, 333x701
// 455 -> 359, 1024^2 1285 -> 1223.  No kernel lets its successor start before it ends: blocks that
// only wait took room from those that work (a trigger at the start of the conjugate
// gradient's kernels: 970 us for 512^2 and 2311 for 1024^2; for SOR: 379 and 1223).
// What a chained kernel reads may still be written while it is set up.  So no
// buffer that it reads is __restrict__: that would allow loads of the read-only
// path, which hold for data that stays as it is for the kernel's whole life, and
// loads moved above the wait.  (With the qualifiers conjugate gradient took 1802
// us for 1024^2 and 817 for 512^2, SOR the same.)
template <class... Params, class... Args>
inline void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared, cudaStream_t stream,
                           Args... args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = shared;
    cfg.stream = stream;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    AR_CUDA(cudaLaunchKernelEx(&cfg, kernel, Params(args)...));
}

__device__ __forceinline__ void after_previous() { cudaGridDependencySynchronize(); }

__global__ void k_rhs(uint32_t w, uint32_t h, const float* __restrict__ primal, const float* __restrict__ gx,
                      const float* __restrict__ gy, float alpha, bool neg_div, float* __restrict__ rhs,
                      float* __restrict__ img) {
    const uint32_t n = w * h;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t x = i % w, y = i / w;
        for (int c = 0; c < 3; ++c) {
            float div = gx[3 * i + c];
            if (x > 0) div -= gx[3 * (i - 1) + c];
            div += gy[3 * i + c];
            if (y > 0) div -= gy[3 * (i - w) + c];
            const float a = alpha * primal[3 * i + c];
            rhs[3 * i + c] = neg_div ? a - div : a + div;
            img[3 * i + c] = primal[3 * i + c];
        }
    }
}

// Red-black SOR, several half sweeps a launch.  A half sweep over a whole image
// in L2 takes 4 to 10 us however small the image is (launch, L2 latency), and a
// solve is hundreds of them.  Here a block of 16 warps holds a 64 x 64 region of
// the image in registers and runs up to `halo` half sweeps on it; each one makes
// the region's outermost ring of valid pixels stale, so the block keeps the
// inner (64 - 2 halo)^2 pixels and regions overlap by the rest.  Every pixel goes
// through the same operations in the same order as in whole-image sweeps, so
// the result is bit-identical.
//
// Warp w owns rows 4w..4w+3, lane k the pixel pair (2k, 2k + 1) of each: one
// red and one black pixel a row, with their right-hand sides.  Of a pixel's four
// neighbours (all of the other colour) one is the lane's own pair, one a
// neighbour lane's, and the vertical ones lie in the lane's own rows or, at the
// strip's edge, in shared memory.
//
// 200 iterations, whole-image sweeps against this: 64x64 1.69 -> 0.23 ms,
// 256x256 1.69 -> 0.26, 512x512 2.51 -> 0.37, 1024x1024 4.17 -> 1.22.
constexpr int kSorRegion = 64, kSorRows = 4, kSorWarps = kSorRegion / kSorRows;
// Half sweeps a launch (even, so that each starts with the same colour): as many
// as leave at most one region per SM, at least 10.  Measured with 8, 10, 12, 16, 20
// and 24: 1024x1024 1.37, 1.22, 1.33, 1.59, 2.64, 5.34 ms; 512x512, where 10 is the
// last with one region per SM, 0.43, 0.37, 0.57, 0.50, 0.84, 1.38; 256x256, where 20
// is, 0.41, 0.37, 0.32, 0.28, 0.26, 0.43; 64x64 0.38, 0.33, 0.30, 0.26, 0.26, 0.25.
int sor_halo(uint32_t w, uint32_t h, int num_sms) {
    for (int halo : {24, 20, 16, 12}) {
        const uint32_t inner = uint32_t(kSorRegion - 2 * halo);
        if (uint64_t((w + inner - 1) / inner) * ((h + inner - 1) / inner) <= uint64_t(num_sms)) return halo;
    }
    return 10;
}

__global__ void __launch_bounds__(kSorWarps * 32, 1) k_sor_sweeps(uint32_t w, uint32_t h, uint32_t tiles_x, int halo, int sweeps,
                                                                  const float* rhs, const float* in,
                                                                  float* __restrict__ out, float alpha, float omega,
                                                                  bool clamp) {
    // the first and last row of every strip: [strip][edge][colour][channel][lane]
    __shared__ float edge[kSorWarps + 2][2][2][3][32];
    after_previous();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int inner = kSorRegion - 2 * halo;
    const int gx0 = int(blockIdx.x % tiles_x) * inner - halo;  // even: region parity = image parity
    const int gy0 = int(blockIdx.x / tiles_x) * inner - halo;
    const int x0 = gx0 + 2 * lane, y0 = gy0 + kSorRows * warp;
    // colour c's pixel of row r is x0 + ((r + c) & 1)  (y0 is even)
    float v[kSorRows][2][3], b[kSorRows][2][3], inv[kSorRows][2];
    uint32_t in_image = 0;  // bit 2r + c: the pixel lies in the image (the others stay 0)
#pragma unroll
    for (int r = 0; r < kSorRows; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int x = x0 + ((r + c) & 1), y = y0 + r;
            const bool inside = x >= 0 && x < int(w) && y >= 0 && y < int(h);
            const size_t i = 3 * (size_t(inside ? y : 0) * w + (inside ? x : 0));
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                v[r][c][ch] = inside ? in[i + ch] : 0.f;
                b[r][c][ch] = inside ? rhs[i + ch] : 0.f;
            }
            const int nn = (x > 0) + (x + 1 < int(w)) + (y > 0) + (y + 1 < int(h));
            inv[r][c] = 1.0f / (alpha + float(nn));
            in_image |= uint32_t(inside) << (2 * r + c);
        }
    // strips above the first and below the last stay zero: their ring is stale from the first sweep on
    for (int k = threadIdx.x; k < 2 * 2 * 2 * 3 * 32; k += blockDim.x)
        (&edge[(k / (2 * 2 * 3 * 32)) ? kSorWarps + 1 : 0][0][0][0][0])[k % (2 * 2 * 3 * 32)] = 0.f;
    const auto publish = [&](int c) {
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            edge[warp + 1][0][c][ch][lane] = v[0][c][ch];
            edge[warp + 1][1][c][ch][lane] = v[kSorRows - 1][c][ch];
        }
    };
    publish(0);
    publish(1);
    __syncthreads();
    const float keep = 1.0f - omega;
    const auto half_sweep = [&](auto colour) {
        constexpr int c = decltype(colour)::value, d = 1 - c;
#pragma unroll
        for (int r = 0; r < kSorRows; ++r) {
            const bool odd = (r + c) & 1;  // the pixel is the pair's right one
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                const float mate = v[r][d][ch];
                const float side = odd ? __shfl_down_sync(0xffffffffu, mate, 1) : __shfl_up_sync(0xffffffffu, mate, 1);
                const float up = r > 0 ? v[r > 0 ? r - 1 : 0][d][ch] : edge[warp][1][d][ch][lane];
                const float down = r + 1 < kSorRows ? v[r + 1 < kSorRows ? r + 1 : 0][d][ch] : edge[warp + 2][0][d][ch][lane];
                // left, right, up, down; a neighbour outside the image adds 0
                float s = 0.f + (odd ? mate : side);
                s += odd ? side : mate;
                s += up;
                s += down;
                const float g = (b[r][c][ch] + s) * inv[r][c];
                const float n = keep * v[r][c][ch] + omega * g;
                v[r][c][ch] = (in_image >> (2 * r + c)) & 1u ? n : 0.f;
            }
        }
        publish(c);
        __syncthreads();
    };
    for (int k = 0; k < sweeps; k += 2) {
        half_sweep(std::integral_constant<int, 0>{});
        half_sweep(std::integral_constant<int, 1>{});
    }
#pragma unroll
    for (int r = 0; r < kSorRows; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int x = x0 + ((r + c) & 1), y = y0 + r;
            const int lx = x - gx0, ly = y - gy0;
            if (lx < halo || lx >= halo + inner || ly < halo || ly >= halo + inner || x >= int(w) || y >= int(h))
                continue;
            const size_t i = 3 * (size_t(y) * w + x);
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                const float n = v[r][c][ch];
                out[i + ch] = clamp ? (n > 0.f ? n : 0.f) : n;
            }
        }
}

// One half sweep over the whole image, in place: the pixels with (x + y) & 1 ==
// parity.  For images too thin to fill regions (see sor_thin).
__global__ void k_sor_half(uint32_t w, uint32_t h, uint32_t parity, const float* rhs, float* img, float alpha,
                           float omega) {
    after_previous();
    const uint32_t half_w = (w + 1) / 2;
    const uint32_t n = half_w * h;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t y = k / half_w;
        const uint32_t x = 2 * (k - y * half_w) + ((y + parity) & 1u);
        if (x >= w) continue;
        const uint32_t i = 3 * (y * w + x);
        const int nn = (x > 0) + (x + 1 < w) + (y > 0) + (y + 1 < h);
        const float inv = 1.0f / (alpha + float(nn));
        for (uint32_t c = i; c < i + 3; ++c) {
            float s = 0.f;
            if (x > 0) s += img[c - 3];
            if (x + 1 < w) s += img[c + 3];
            if (y > 0) s += img[c - 3 * w];
            if (y + 1 < h) s += img[c + 3 * w];
            img[c] = (1.0f - omega) * img[c] + omega * ((rhs[c] + s) * inv);
        }
    }
}

// Whether whole-image half sweeps are faster than regions: a region costs 4 to 5 ns
// a half sweep however few of its pixels lie in the image, a whole-image half sweep
// 2.2 us + 7.5 ns per 1000 pixels.  200 iterations, height x width, regions / whole
// image: 1x100000 3670 / 936 us, 1x1000000 35740 / 3452, 8x262144 9758 / 7323; on
// the other side of the line (whole image unchained) 1x10000 519 / 1686, 8x32768
// 1476 / 2509, 16x65536 2682 / 4249, 1024x1024 1219 / 4165.
bool sor_thin(uint64_t regions, uint64_t pixels) { return regions > 500 + pixels / 600; }

__global__ void k_clamp(size_t n, const float* __restrict__ in, float* __restrict__ out) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        out[i] = in[i] > 0.f ? in[i] : 0.f;
}

// ---- CG ----
// A sum over the image is spread over this many places (3 channels each).
constexpr uint32_t kCgSlots = 16, kCgSum = 3 * kCgSlots;

template <class T>
__device__ __forceinline__ void stencil(uint32_t w, uint32_t h, uint32_t i, const T* v, double alpha, double out[3]) {
    const uint32_t x = i % w, y = i / w;
    double s[3] = {0, 0, 0};
    int nn = 0;
    auto add = [&](uint32_t j) { for (int c = 0; c < 3; ++c) s[c] += double(v[3 * j + c]); nn++; };
    if (x > 0) add(i - 1);
    if (x + 1 < w) add(i + 1);
    if (y > 0) add(i - w);
    if (y + 1 < h) add(i + w);
    for (int c = 0; c < 3; ++c) out[c] = (alpha + nn) * double(v[3 * i + c]) - s[c];
}

__device__ __forceinline__ void block_add3(double a0, double a1, double a2, double* dst) {
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_down_sync(0xffffffffu, a0, o);
        a1 += __shfl_down_sync(0xffffffffu, a1, o);
        a2 += __shfl_down_sync(0xffffffffu, a2, o);
    }
    __shared__ double sm[3][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { sm[0][wid] = a0; sm[1][wid] = a1; sm[2][wid] = a2; }
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        a0 = lane < nw ? sm[0][lane] : 0.0;
        a1 = lane < nw ? sm[1][lane] : 0.0;
        a2 = lane < nw ? sm[2][lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            a0 += __shfl_down_sync(0xffffffffu, a0, o);
            a1 += __shfl_down_sync(0xffffffffu, a1, o);
            a2 += __shfl_down_sync(0xffffffffu, a2, o);
        }
        if (lane == 0) {
            dst += 3 * (blockIdx.x % kCgSlots);
            atomicAdd(dst, a0);
            atomicAdd(dst + 1, a1);
            atomicAdd(dst + 2, a2);
        }
    }
    __syncthreads();
}

// b (f64) = alpha*primal + div G; x (f64) = primal; bb += |b|^2.
__global__ void k_cg_setup(uint32_t w, uint32_t h, const float* primal, const float* gx, const float* gy, double alpha,
                           bool neg_div, double* b, double* x, double* bb) {
    const uint32_t n = w * h;
    double a[3] = {0, 0, 0};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t xx = i % w, yy = i / w;
        for (int c = 0; c < 3; ++c) {
            double div = gx[3 * i + c];
            if (xx > 0) div -= gx[3 * (i - 1) + c];
            div += gy[3 * i + c];
            if (yy > 0) div -= gy[3 * (i - w) + c];
            const double av = alpha * double(primal[3 * i + c]);
            const double bv = neg_div ? av - div : av + div;
            b[3 * i + c] = bv;
            x[3 * i + c] = primal[3 * i + c];
            a[c] += bv * bv;
        }
    }
    block_add3(a[0], a[1], a[2], bb);
}

// r (f32) = b - A x (f64 arithmetic); d = 0; rr += |r|^2 (f64).
__global__ void k_cg_residual(uint32_t w, uint32_t h, const double* b, const double* x, double alpha, float* r,
                              float* d, double* rr) {
    const uint32_t n = w * h;
    double a[3] = {0, 0, 0};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double ax[3];
        stencil(w, h, i, x, alpha, ax);
        for (int c = 0; c < 3; ++c) {
            const double rv = b[3 * i + c] - ax[c];
            r[3 * i + c] = float(rv);
            d[3 * i + c] = 0.f;
            a[c] += rv * rv;
        }
    }
    block_add3(a[0], a[1], a[2], rr);
}

// ---- the CG iteration ----
// Two kernels an iteration.  The arrays of an image do not fit the L1s, and half
// of an SM's L2 accesses go to the other die, so an iteration is bound by its
// passes over L2: 13 of them when direction, product and update were kernels of
// their own, 8 here (the first forms p = r + beta p for a float and its
// neighbours, stores p and sums p.Ap; the second forms A p again from p instead of
// storing it).  A thread owns one float column (a pixel column's channel) and
// walks down `rows` rows, so the vertical neighbours stay in registers, already
// widened; the horizontal ones come through L1.  The sums of a block go to one of
// kCgSlots places, so that hundreds of blocks do not queue on three addresses.
// Every float goes through the same operations as before: f64 stencil and
// sums, f32 vectors.  A solve to 1e-6 (64 iterations): 1024x1024 3.00 -> 2.08
// ms, 512x512 1.87 -> 1.13, 256x256 1.19 -> 0.92 (chained 1.81, 0.83 and 0.61).  Not
// faster, unchained: tiles with a rim in shared memory (2.7 ms at 1024x1024: their
// index arithmetic), loads batched four rows ahead (2.4), four floats a thread with
// neighbours by shuffle (2.6).
constexpr uint32_t kCgThreads = 192, kCgInner = 32;  // 64 pixels of a row

// How threads share the floats of an image.
struct CgShape {
    uint32_t w, h;   // of the walk
    uint32_t rows;   // that a thread walks down
    uint32_t log2p;  // a block is 2^log2p pixels wide and takes 64 >> log2p runs of rows
};

// Rows a thread walks: fewer halo rows and prologues the more there are, as
// long as five blocks an SM are left.  Measured with 1, 2, 4, 8 and 16: 1024x1024
// 3.90, 2.74, 2.19, 2.03, 1.80 ms; 512x512 1.29, 1.00, 0.82, 1.03, 1.45; 256x256 0.63,
// 0.56, 0.68, 0.86, 1.44.
// A block takes several runs of a narrow image (of 8 rows up to 16 pixels: 200000x5
// 2.98 ms, with 16 rows 3.32, with 4 3.30), a thread several columns, the grid's
// width apart, of a low one, and a column of pixels is walked as the row that it is
// in memory (the same operations).  Against 64 pixels of one run a block: 1000000x1
// 38.9 -> 2.55 ms, 500000x2 25.5 -> 2.9, 1x1000000 3.57 -> 2.55, 2000x3 616 -> 480 us.
CgShape cg_shape(uint32_t w, uint32_t h, int num_sms, dim3& grid) {
    CgShape s{w == 1 ? h : w, w == 1 ? 1u : h, 16, 6};
    while (s.log2p > 0 && (1u << (s.log2p - 1)) >= s.w) s.log2p--;
    if (s.log2p <= 4) s.rows = 8;
    const uint32_t cols = uint32_t((uint64_t(s.w) + (1u << s.log2p) - 1) >> s.log2p), runs = 64u >> s.log2p;
    const auto blocks_y = [&] { return ((s.h + s.rows - 1) / s.rows + runs - 1) / runs; };
    const uint64_t least = uint64_t(5 * num_sms);
    while (s.rows > 1 && uint64_t(cols) * blocks_y() < least) s.rows /= 2;
    while (blocks_y() > 65535u) s.rows *= 2;  // the grid's y extent
    uint32_t per = 1;                         // columns a thread
    while (per * std::min(s.rows, s.h) < 16 && uint64_t(cols) * blocks_y() / (2 * per) >= least) per *= 2;
    grid = dim3((cols + per - 1) / per, blocks_y());
    return s;
}

// coef[c] = num / den of channel c (0 where den is 0), from the slots of the two
// sums: warp c adds up channel c.  Visible to the block after its next barrier.
// (Plain loads: the sums are complete, and one copy in L1 serves all the blocks
// of an SM; read past L1 by every thread, these few lines cost 300 us.)
__device__ __forceinline__ void cg_ratio(const double* num, const double* den, float coef[3]) {
    const uint32_t warp = threadIdx.x / 32u, lane = threadIdx.x & 31u;
    if (warp >= 3) return;
    double a = lane < kCgSlots ? num[3 * lane + warp] : 0.0, b = lane < kCgSlots ? den[3 * lane + warp] : 0.0;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if (lane == 0) coef[warp] = b != 0.0 ? float(a / b) : 0.f;
}

// Adds each thread's `a`, of channel threadIdx.x % 3, to the block's slot of `sum`.
__device__ __forceinline__ void cg_add(double a, double* sum) {
    __shared__ double part[kCgThreads];
    part[threadIdx.x] = a;
    __syncthreads();
    const uint32_t warp = threadIdx.x / 32u, lane = threadIdx.x & 31u;
    if (warp < 3) {  // warp c adds up channel c
        double t = part[3 * lane + warp] + part[96 + 3 * lane + warp];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) atomicAdd(sum + 3 * ((blockIdx.x + blockIdx.y * gridDim.x) % kCgSlots) + warp, t);
    }
}

// Calls each(i, v, A v) for the floats of this thread's columns in its rows;
// at(i) gives v of float i (f32).
template <class At, class Each>
__device__ __forceinline__ void cg_walk(const CgShape& g, double alpha, At at, Each each) {
    const uint32_t run = (threadIdx.x / 3u) >> g.log2p, lanes = 3u << g.log2p, pitch = 3u * g.w;
    const uint32_t y0 = (blockIdx.y * (64u >> g.log2p) + run) * g.rows, y1 = min(g.h, y0 + g.rows);
    if (y0 >= g.h) return;
    for (uint32_t f = blockIdx.x * lanes + (threadIdx.x - run * lanes); f < pitch; f += gridDim.x * lanes) {
        const bool left = f >= 3u, right = f + 3u < pitch;
        const int nx = int(left) + int(right);
        uint32_t i = y0 * pitch + f;
        float m32 = at(i);
        double up = y0 > 0 ? double(at(i - pitch)) : 0.0, mid = double(m32);
#pragma unroll 4
        for (uint32_t y = y0; y < y1; ++y, i += pitch) {
            const float d32 = y + 1 < g.h ? at(i + pitch) : 0.f;
            const float l32 = left ? at(i - 3u) : 0.f, r32 = right ? at(i + 3u) : 0.f;
            const double down = double(d32);
            double s = double(l32);  // left, right, up, down; outside the image 0
            s += double(r32);
            s += up;
            s += down;
            const double diag = alpha + (nx + int(y > 0) + int(y + 1 < g.h));
            each(i, m32, diag * mid - s);
            up = mid;
            mid = down;
            m32 = d32;
        }
    }
}

// p = r + beta p (beta = rr / rr_prev; the first iteration takes p = r), pq += p.Ap
__global__ void __launch_bounds__(kCgThreads) k_cg_direction(CgShape g, const float* r, const float* p_in,
                                                             float* __restrict__ p_out, double alpha,
                                                             const double* rr, const double* rr_prev, double* pq) {
    __shared__ float coef[3];
    after_previous();
    double a = 0.0;
    const auto each = [&](uint32_t i, float p, double ap) {
        p_out[i] = p;
        a += double(p) * ap;
    };
    if (rr_prev) {
        cg_ratio(rr, rr_prev, coef);
        __syncthreads();
        const float be = coef[threadIdx.x % 3u];
        cg_walk(g, alpha, [&](uint32_t i) { return r[i] + be * p_in[i]; }, each);
    } else {
        cg_walk(g, alpha, [&](uint32_t i) { return r[i]; }, each);
    }
    cg_add(a, pq);
}

// d += al p, r -= al (A p), al = rr / pq; rr_new += r.r
__global__ void __launch_bounds__(kCgThreads) k_cg_update(CgShape g, const float* p, float* d, float* r, double alpha,
                                                          const double* rr, const double* pq, double* rr_new) {
    __shared__ float coef[3];
    after_previous();
    cg_ratio(rr, pq, coef);
    __syncthreads();
    const float al = coef[threadIdx.x % 3u];
    double a = 0.0;
    cg_walk(g, alpha, [&](uint32_t i) { return p[i]; },
            [&](uint32_t i, float pv, double ap) {
                d[i] += al * pv;
                const float rv = r[i] - al * float(ap);
                r[i] = rv;
                a += double(rv) * double(rv);
            });
    cg_add(a, rr_new);
}

__global__ void k_cg_accumulate(size_t n, double* x, const float* d) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        x[i] += double(d[i]);
}

__global__ void k_cg_output(size_t n, const double* x, float* out) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        out[i] = x[i] > 0.0 ? float(x[i]) : 0.f;
}

}  // namespace

// The red-black SOR solve with caller-provided scratch (rhs and img, 3*W*H
// floats each) on `stream`; launches only, no allocation, no synchronisation.
// `out` may be any of the inputs: they are read before it is first written.
// Returns the number of kernels.
uint64_t poisson_sor_with_scratch(cudaStream_t stream, int num_sms, const ar_integrator_cfg& cfg, uint32_t w,
                                  uint32_t h, const float* primal, const float* gx, const float* gy, float* rhs,
                                  float* img, float* out) {
    const size_t n = size_t(w) * h;
    const int grid = std::max(1, std::min(int((n + 255) / 256), num_sms * 8));
    const bool neg_div = (cfg.gdpt_flags & AR_GDPT_CONSISTENT_DIVERGENCE) != 0;
    // launches of `halo` half sweeps (two an iteration), ping-pong between img
    // and out so that the last one ends in out
    const int halo = sor_halo(w, h, num_sms);
    const uint64_t half = 2 * uint64_t(cfg.poisson_iterations), launches = (half + halo - 1) / halo;
    const uint32_t inner = uint32_t(kSorRegion - 2 * halo);
    const uint32_t tiles_x = (w + inner - 1) / inner, tiles_y = (h + inner - 1) / inner;
    k_rhs<<<grid, 256, 0, stream>>>(w, h, primal, gx, gy, cfg.alpha, neg_div, rhs, img);
    if (launches == 0 || sor_thin(uint64_t(tiles_x) * tiles_y, n)) {
        for (uint64_t k = 0; k < half; ++k)
            launch_chained(k_sor_half, grid, 256, 0, stream, w, h, uint32_t(k & 1), rhs, img, cfg.alpha, cfg.sor_omega);
        k_clamp<<<grid, 256, 0, stream>>>(3 * n, img, out);
        AR_CUDA(cudaGetLastError());
        return 2 + half;
    }
    float* src = launches & 1 ? img : out;
    float* dst = launches & 1 ? out : img;
    if (src != img)
        AR_CUDA(cudaMemcpyAsync(src, img, 3 * n * sizeof(float), cudaMemcpyDeviceToDevice, stream));
    for (uint64_t l = 0; l < launches; ++l) {
        const int sweeps = int(std::min<uint64_t>(halo, half - l * halo));
        launch_chained(k_sor_sweeps, tiles_x * tiles_y, kSorWarps * 32, 0, stream, w, h, tiles_x, halo, sweeps, rhs,
                       src, dst, cfg.alpha, cfg.sor_omega, l + 1 == launches);
        std::swap(src, dst);
    }
    AR_CUDA(cudaGetLastError());
    return 1 + launches;
}

uint64_t poisson_reconstruct(ar_context* ctx, const ar_integrator_cfg& cfg, uint32_t w, uint32_t h, const float* primal,
                         const float* gx, const float* gy, float* out, double* rel_residual) {
    const size_t n = size_t(w) * h;
    const int grid = std::max(1, std::min(int((n + 255) / 256), ctx->num_sms * 8));
    cudaStream_t st = ctx->stream;
    if (cfg.poisson_solver == AR_POISSON_SOR) {
        ctx->solver.ensure(2 * 3 * n * sizeof(float));
        float* rhs = ctx->solver.buf.as<float>();
        const uint64_t kernels =
            poisson_sor_with_scratch(st, ctx->num_sms, cfg, w, h, primal, gx, gy, rhs, rhs + 3 * n, out);
        if (rel_residual) *rel_residual = -1.0;
        return kernels;
    }
    // CG with FP64 refinement.
    const double alpha = double(cfg.alpha);
    const double tol = cfg.poisson_tolerance > 0 ? cfg.poisson_tolerance : 1e-6;
    const uint32_t max_total = cfg.poisson_iterations ? cfg.poisson_iterations : 1000;
    // sums: |b|^2, rr of iterations 0..kCgInner, pq of 0..kCgInner - 1
    const size_t sums = (2 * kCgInner + 2) * kCgSum * sizeof(double);
    ctx->solver.ensure(3 * n * (2 * sizeof(double) + 4 * sizeof(float)) + sums + 1024);
    double* b = ctx->solver.buf.as<double>();
    double* x = b + 3 * n;
    float* r = reinterpret_cast<float*>(x + 3 * n);
    float* p[2] = {r + 3 * n, r + 6 * n};
    float* d = r + 9 * n;
    double* bb = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(d + 3 * n) + 63) & ~uintptr_t(63));
    double* rr = bb + kCgSum;
    double* pq = rr + (kCgInner + 1) * kCgSum;
    AR_CUDA(cudaMemsetAsync(bb, 0, kCgSum * sizeof(double), st));
    k_cg_setup<<<grid, 256, 0, st>>>(w, h, primal, gx, gy, alpha,
                                     (cfg.gdpt_flags & AR_GDPT_CONSISTENT_DIVERGENCE) != 0, b, x, bb);
    dim3 blocks;
    const CgShape shape = cg_shape(w, h, ctx->num_sms, blocks);
    double hb[2 * kCgSum];
    double res = 0.0;
    uint32_t total = 0;
    uint64_t launches = 1;
    for (;;) {
        AR_CUDA(cudaMemsetAsync(rr, 0, sums - kCgSum * sizeof(double), st));
        k_cg_residual<<<grid, 256, 0, st>>>(w, h, b, x, alpha, r, d, rr);
        launches++;
        AR_CUDA(cudaMemcpyAsync(hb, bb, 2 * kCgSum * sizeof(double), cudaMemcpyDeviceToHost, st));
        AR_CUDA(cudaStreamSynchronize(st));
        res = 0.0;
        for (uint32_t c = 0; c < 3; ++c) {
            double sb = 0.0, sr = 0.0;
            for (uint32_t k = 0; k < kCgSlots; ++k) {
                sb += hb[3 * k + c];
                sr += hb[kCgSum + 3 * k + c];
            }
            res = std::max(res, std::sqrt(sr) / (sb > 0 ? std::sqrt(sb) : 1.0));
        }
        if (res <= tol || total >= max_total) break;
        for (uint32_t k = 0; k < kCgInner; ++k) {
            double *rr_k = rr + k * kCgSum, *pq_k = pq + k * kCgSum;
            launch_chained(k_cg_direction, blocks, kCgThreads, 0, st, shape, r, p[(k + 1) & 1], p[k & 1], alpha,
                           rr_k, k ? rr_k - kCgSum : nullptr, pq_k);
            launch_chained(k_cg_update, blocks, kCgThreads, 0, st, shape, p[k & 1], d, r, alpha, rr_k, pq_k,
                           rr_k + kCgSum);
        }
        total += kCgInner;
        k_cg_accumulate<<<grid, 256, 0, st>>>(3 * n, x, d);
        launches += 2 * kCgInner + 1;
    }
    k_cg_output<<<grid, 256, 0, st>>>(3 * n, x, out);
    AR_CUDA(cudaGetLastError());
    AR_CUDA(cudaStreamSynchronize(st));
    if (rel_residual) *rel_residual = res;
    return launches + 1;
}

}  // namespace ar
