// Learned denoiser (see rt_unet.cuh): kernels, forward, backward, Adam.
//
// Activations are NHWC BF16 with channel counts that are multiples of 16.
//   forward      out[p][co] = b[co] + sum_tap,ci x[p + off(tap)][ci] w[tap][ci][co]
//                on the fifth-generation tensor cores (convTc, rt_conv_tc.cu)
//                with K-major weights wT[tap][co][ci]
//   data grad    convTc on dY with B[ci][co] = w[8 - tap][ci][co]: the forward
//                weights read with the taps reversed
//   weight grad  dw[tap][ci][co] = sum_p x[p + off(tap)][ci] dY[p][co] on
//                the tensor cores (wgradTc, rt_wgrad_tc.cu; the 16x16x16
//                warp-level MMA kernel wgradKernel when the single-role
//                convolution path is selected)
#include <mma.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "rt_common.cuh"
#include "rt_conv_tc.cuh"
#include "rt_unet.cuh"

namespace rt {
namespace {

using bf16 = __nv_bfloat16;
using namespace nvcuda;

constexpr int kTileX = 16, kTileY = 4;
constexpr int kWidths[5] = {32, 48, 64, 96, 128};
constexpr int kInputChannels = 10, kInputPadded = 16, kOutChannels = 3;

inline int blocksFor(long long n, int b) { return (int)((n + b - 1) / b); }

// ---- weight gradient ----
// Block: one tap, 16 input channels, CT output channels, a chunk of 16-pixel
// row segments; per-warp shared staging; partial sums added to dw atomically.
template <int CT>
__global__ void __launch_bounds__(128) wgradKernel(const bf16* __restrict__ x, const bf16* __restrict__ dy, int N,
                                                   int H, int W, int Cin, int Cout, int segmentsPerBlock,
                                                   float* dw) {
    __shared__ __align__(32) bf16 sX[4][16][16];
    __shared__ __align__(32) bf16 sD[4][16][CT];
    __shared__ __align__(32) float sAcc[4][16][CT];
    const int tap = blockIdx.y % 9, ci0 = (blockIdx.y / 9) * 16, co0 = blockIdx.z * CT;
    const int ky = tap / 3 - 1, kx = tap % 3 - 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int segsPerRow = (W + 15) / 16;
    const long long segments = (long long)N * H * segsPerRow;
    wmma::fragment<wmma::accumulator, 16, 16, 16, float> acc[CT / 16];
#pragma unroll
    for (int f = 0; f < CT / 16; f++) wmma::fill_fragment(acc[f], 0.0f);
    const long long begin = (long long)blockIdx.x * segmentsPerBlock;
    for (long long s = begin + warp; s < begin + segmentsPerBlock && s < segments; s += 4) {
        int xs = (int)(s % segsPerRow) * 16;
        long long row = s / segsPerRow;
        int y = (int)(row % H), n = (int)(row / H);
        // x[n][y + ky][xs + px + kx][ci0 .. ci0 + 15], zero outside the image.
        for (int k = lane; k < 32; k += 32) {
            int px = k >> 1, half = k & 1;
            int yy = y + ky, xx = xs + px + kx;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (yy >= 0 && yy < H && xx >= 0 && xx < W && xs + px < W)
                v = *reinterpret_cast<const uint4*>(x + (((size_t)n * H + yy) * W + xx) * Cin + ci0 + half * 8);
            *reinterpret_cast<uint4*>(&sX[warp][px][half * 8]) = v;
        }
        constexpr int perPix = CT / 8;
        for (int k = lane; k < 16 * perPix; k += 32) {
            int px = k / perPix, part = k % perPix;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (xs + px < W)
                v = *reinterpret_cast<const uint4*>(dy + (((size_t)n * H + y) * W + xs + px) * Cout + co0 + part * 8);
            *reinterpret_cast<uint4*>(&sD[warp][px][part * 8]) = v;
        }
        __syncwarp();
        wmma::fragment<wmma::matrix_a, 16, 16, 16, bf16, wmma::col_major> a;  // (ci, pixel) = sX[pixel][ci]
        wmma::load_matrix_sync(a, &sX[warp][0][0], 16);
#pragma unroll
        for (int f = 0; f < CT / 16; f++) {
            wmma::fragment<wmma::matrix_b, 16, 16, 16, bf16, wmma::row_major> b;
            wmma::load_matrix_sync(b, &sD[warp][0][f * 16], CT);
            wmma::mma_sync(acc[f], a, b, acc[f]);
        }
        __syncwarp();
    }
#pragma unroll
    for (int f = 0; f < CT / 16; f++) wmma::store_matrix_sync(&sAcc[warp][0][f * 16], acc[f], CT, wmma::mem_row_major);
    __syncthreads();
    for (int k = threadIdx.x; k < 16 * CT; k += blockDim.x) {
        int ci = k / CT, c = k % CT;
        float v = sAcc[0][ci][c] + sAcc[1][ci][c] + sAcc[2][ci][c] + sAcc[3][ci][c];
        if (v != 0.0f) atomicAdd(&dw[((size_t)tap * Cin + ci0 + ci) * Cout + co0 + c], v);
    }
}

// ---- elementwise and reshaping kernels ----
// Position of pixel p of `total` = n * h * w; 32-bit divisions where the
// index fits (64-bit ones are a subroutine of ~70 instructions).
struct Pixel { int x, y, n; };
__device__ __forceinline__ Pixel pixelOf(long long p, long long total, int w, int h) {
    if (total <= 0xFFFFFFFFll) {
        const unsigned u = (unsigned)p, row = u / (unsigned)w;
        return Pixel{(int)(u % (unsigned)w), (int)(row % (unsigned)h), (int)(row / (unsigned)h)};
    }
    const long long row = p / w;
    return Pixel{(int)(p % w), (int)(row % h), (int)(row / h)};
}
__global__ void inputKernel(const float* aov, int n, int h, int w, int H, int W, bf16* x0, const int* batch,
                            const unsigned char* flips) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long total = (long long)n * H * W;
    if (i >= total) return;
    int X = (int)(i % W), Y = (int)((i / W) % H), b = (int)(i / ((long long)W * H));
    float v[kInputPadded] = {};
    {
        // The padded frame beyond w x h repeats the edge pixels.
        int src = batch ? batch[b] : b;
        int sx = min(X, w - 1), sy = min(Y, h - 1);
        if (flips) { if (flips[b] & 1) sx = w - 1 - sx; if (flips[b] & 2) sy = h - 1 - sy; }
        const float* a = aov + (((size_t)src * h + sy) * w + sx) * kInputChannels;
        v[0] = log1pf(fmaxf(a[0], 0.0f)); v[1] = log1pf(fmaxf(a[1], 0.0f)); v[2] = log1pf(fmaxf(a[2], 0.0f));
        v[3] = a[3]; v[4] = a[4]; v[5] = a[5];
        v[6] = a[6]; v[7] = a[7]; v[8] = a[8];
        v[9] = log1pf(fmaxf(a[9], 0.0f));
    }
    uint4 packed[2];
    uint32_t* words = reinterpret_cast<uint32_t*>(packed);
#pragma unroll
    for (int j = 0; j < kInputPadded / 2; j++) {
        __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        words[j] = *reinterpret_cast<uint32_t*>(&pair);
    }
    uint4* o = reinterpret_cast<uint4*>(x0 + (size_t)i * kInputPadded);
    o[0] = packed[0];
    o[1] = packed[1];
}
// 2x2 average pooling, 8 channels per thread (16-byte loads and stores).
__global__ void poolKernel(const bf16* in, int N, int H, int W, int C, bf16* out) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int Ho = H / 2, Wo = W / 2, C8 = C / 8;
    long long total = (long long)N * Ho * Wo * C8;
    if (i >= total) return;
    int c = (int)(i % C8) * 8;
    long long p = i / C8;
    int x = (int)(p % Wo), y = (int)((p / Wo) % Ho), n = (int)(p / ((long long)Wo * Ho));
    const bf16* b = in + (((size_t)n * H + 2 * y) * W + 2 * x) * C + c;
    uint4 q[4] = {*reinterpret_cast<const uint4*>(b), *reinterpret_cast<const uint4*>(b + C),
                  *reinterpret_cast<const uint4*>(b + (size_t)W * C), *reinterpret_cast<const uint4*>(b + (size_t)W * C + C)};
    const bf16* e[4] = {reinterpret_cast<const bf16*>(&q[0]), reinterpret_cast<const bf16*>(&q[1]),
                        reinterpret_cast<const bf16*>(&q[2]), reinterpret_cast<const bf16*>(&q[3])};
    uint4 r;
    bf16* o = reinterpret_cast<bf16*>(&r);
#pragma unroll
    for (int j = 0; j < 8; j++) {
        float s = __bfloat162float(e[0][j]) + __bfloat162float(e[1][j]) + __bfloat162float(e[2][j]) +
                  __bfloat162float(e[3][j]);
        o[j] = __float2bfloat16(0.25f * s);
    }
    *reinterpret_cast<uint4*>(out + (size_t)p * C + c) = r;
}
// out = concat(upsample2(low), skip) along channels, 8 channels per thread.
// Bound by the write of the concatenation; one element per thread (2-byte
// accesses, two 64-bit divisions each) took 264 us for 32 x 128 x 128 x 80.
__global__ void upConcatKernel(const bf16* low, int Cl, const bf16* skip, int Cs, int N, int H, int W, bf16* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int C = Cl + Cs, C8 = C / 8;
    const long long total = (long long)N * H * W * C8;
    if (i >= total) return;
    const int c = (int)(i % C8) * 8;
    const long long p = i / C8;
    const Pixel q = pixelOf(p, (long long)N * H * W, W, H);
    const uint4* src = c < Cl
        ? reinterpret_cast<const uint4*>(low + (((size_t)q.n * (H / 2) + q.y / 2) * (W / 2) + q.x / 2) * Cl + c)
        : reinterpret_cast<const uint4*>(skip + (size_t)p * Cs + (c - Cl));
    *reinterpret_cast<uint4*>(out + (size_t)p * C + c) = __ldg(src);
}

// Sums of N per-thread values over a block of up to 256 threads whose lanes hold
// the sums of GROUP interleaved owners (thread t belongs to owner t % GROUP,
// GROUP a power of two up to 32): add[owner * N + v] receives the totals,
// one atomic per value and block. scratch: 8 * GROUP * N floats.
template <int N, int GROUP>
__device__ __forceinline__ void blockSums(float (&v)[N], float* scratch, float* add) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < N; k++)
#pragma unroll
        for (int off = 16; off >= GROUP; off >>= 1) v[k] += __shfl_xor_sync(0xFFFFFFFFu, v[k], off);
    if (lane < GROUP)
#pragma unroll
        for (int k = 0; k < N; k++) scratch[(warp * GROUP + lane) * N + k] = v[k];
    __syncthreads();
    for (int i = threadIdx.x; i < GROUP * N; i += blockDim.x) {
        float s = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += scratch[w * GROUP * N + i];
        if (s != 0.0f) atomicAdd(add + i, s);
    }
    __syncthreads();
}

// The training head in one pass over the last activations d (32 channels):
// the 1x1 output layer (pred[k] = b[k] + sum_c d[c] w[c][k], channels in
// order as in outForwardKernel), the L1 loss against log1p of the target, the
// output layer's gradients, and the gradient at the last 3x3 layer's
// pre-activation (BF16, masked by d > 0) with that layer's bias gradient.
// Two lanes per pixel, 16 channels each (32-byte loads); the sums stay in
// registers over the pixels of a thread. It replaces five passes with one
// global atomic per warp and sum (loss 83, output layer backward 705, mask 69,
// bias 29, target 7 us at 32 x 128 x 128 pixels). Bound by its 73 MB of
// traffic (11 us at copy bandwidth) and its ~460 instructions per 16 pixels.
constexpr int kHeadHalf = 16;  // channels per lane
__global__ void __launch_bounds__(128, 3) headKernel(const bf16* d, const float* target, int n, int h, int w,
                                                     const int* batch, const unsigned char* flips, const float* wt,
                                                     const float* b, bf16* dPre, float* loss, float* dW, float* dB,
                                                     float* dBias) {
    constexpr int C = 2 * kHeadHalf;
    __shared__ float sW[C * kOutChannels];
    __shared__ float scratch[8 * 2 * kHeadHalf * kOutChannels];
    for (int i = threadIdx.x; i < C * kOutChannels; i += blockDim.x) sW[i] = wt[i];
    __syncthreads();
    const int half = threadIdx.x & 1;
    const float* myW = sW + half * kHeadHalf * kOutChannels;
    const long long total = (long long)n * h * w;
    const float count = (float)(total * kOutChannels);
    const float step = 1.0f / count;
    float accW[kHeadHalf * kOutChannels] = {}, accBias[kHeadHalf] = {}, accB[kOutChannels + 1] = {};
    const float bias[kOutChannels] = {b[0], b[1], b[2]};
    // Whole warps walk the pixels (the channel sum passes between lanes).
    for (long long base = (long long)blockIdx.x * (blockDim.x / 2); base < total;
         base += (long long)gridDim.x * (blockDim.x / 2)) {
        const long long p = base + (threadIdx.x >> 1);
        const bool valid = p < total;
        uint4 q[2] = {};
        float t[kOutChannels] = {0.0f, 0.0f, 0.0f};
        if (valid) {
            const uint4* src = reinterpret_cast<const uint4*>(d + (size_t)p * C + half * kHeadHalf);
            q[0] = __ldg(src);
            q[1] = __ldg(src + 1);
            const Pixel at = pixelOf(p, total, w, h);
            int sx = at.x, sy = at.y;
            if (flips) {
                const unsigned char f = flips[at.n];
                if (f & 1) sx = w - 1 - sx;
                if (f & 2) sy = h - 1 - sy;
            }
            const float* tp = target + (((size_t)(batch ? batch[at.n] : at.n) * h + sy) * w + sx) * kOutChannels;
            for (int k = 0; k < kOutChannels; k++) t[k] = log1pf(fmaxf(tp[k], 0.0f));
        }
        float x[kHeadHalf];
        const bf16* e = reinterpret_cast<const bf16*>(q);
#pragma unroll
        for (int j = 0; j < kHeadHalf; j++) x[j] = __bfloat162float(e[j]);
        // Channels 0-15 on the even lane, then 16-31 on the odd one.
        float s[kOutChannels] = {bias[0], bias[1], bias[2]};
#pragma unroll
        for (int part = 0; part < 2; part++) {
            if (part == 1)
                for (int k = 0; k < kOutChannels; k++) s[k] = __shfl_xor_sync(0xFFFFFFFFu, s[k], 1);
#pragma unroll
            for (int j = 0; j < kHeadHalf; j++)
#pragma unroll
                for (int k = 0; k < kOutChannels; k++) s[k] += x[j] * myW[j * kOutChannels + k];
        }
        float g[kOutChannels];
#pragma unroll
        for (int k = 0; k < kOutChannels; k++) {
            const float pred = __shfl_sync(0xFFFFFFFFu, s[k], (threadIdx.x & 31) | 1);
            const float diff = pred - t[k];
            g[k] = !valid ? 0.0f : diff > 0.0f ? step : (diff < 0.0f ? -step : 0.0f);
            if (valid && half == 0) {
                accB[k] += g[k];
                accB[kOutChannels] += fabsf(diff);
            }
        }
        uint4 o[2];
        bf16* oe = reinterpret_cast<bf16*>(o);
#pragma unroll
        for (int j = 0; j < kHeadHalf; j++) {
            float dd = 0.0f;
#pragma unroll
            for (int k = 0; k < kOutChannels; k++) {
                accW[j * kOutChannels + k] += x[j] * g[k];
                dd += g[k] * myW[j * kOutChannels + k];
            }
            oe[j] = __float2bfloat16(x[j] > 0.0f ? dd : 0.0f);
            accBias[j] += __bfloat162float(oe[j]);
        }
        if (valid) {
            uint4* dst = reinterpret_cast<uint4*>(dPre + (size_t)p * C + half * kHeadHalf);
            dst[0] = o[0];
            dst[1] = o[1];
        }
    }
    accB[kOutChannels] /= count;
    blockSums<kHeadHalf * kOutChannels, 2>(accW, scratch, dW);
    blockSums<kHeadHalf, 2>(accBias, scratch, dBias);
    float onlyB[kOutChannels] = {accB[0], accB[1], accB[2]}, onlyLoss[1] = {accB[kOutChannels]};
    blockSums<kOutChannels, 1>(onlyB, scratch, dB);
    blockSums<1, 1>(onlyLoss, scratch, loss);
}

// Gradient at a layer's pre-activation (BF16, masked by its output y > 0) and
// its bias gradient, from the FP32 gradient of its output, which is
//   KIND 0  dOut itself (C channels per pixel);
//   KIND 1  the upsampled half of a decoder's input gradient: the sum of the
//           2x2 pixels of dOut's first C channels (dOut: Cd channels, 2H x 2W);
//   KIND 2  the skip half (channels Cd - C ... of dOut) plus a quarter of the
//           pooled level's gradient dPool (H/2 x W/2 x C).
// Eight channels per thread (32-byte FP32 loads, 16-byte BF16 ones); a
// thread keeps its channels over its pixels, so the bias sums stay in
// registers until the block's end. Bound by memory traffic: one pass over
// dOut, y and dPre in place of one pass per operation with an element per
// thread (32 x 128 x 128 x 32 channels: mask 69 + bias 29 us, pool backward
// 102 and skip copy 57).
template <int KIND>
__global__ void __launch_bounds__(256) preGradKernel(const float* dOut, int Cd, const float* dPool, const bf16* y,
                                                     int N, int H, int W, int C, bf16* dPre, float* db) {
    extern __shared__ float sums[];  // [slots][C]
    const int C8 = C / 8, slots = blockDim.x / C8;
    const int cg = threadIdx.x % C8, slot = threadIdx.x / C8;
    const long long total = (long long)N * H * W;
    float acc[8] = {};
    if (slot < slots) {
        for (long long p = (long long)blockIdx.x * slots + slot; p < total; p += (long long)gridDim.x * slots) {
            const uint4 yq = __ldg(reinterpret_cast<const uint4*>(y + (size_t)p * C) + cg);
            float v[8];
            auto load = [&](const float* src, float (&to)[8]) {
                const float4 a = __ldg(reinterpret_cast<const float4*>(src)), b = __ldg(reinterpret_cast<const float4*>(src) + 1);
                to[0] = a.x; to[1] = a.y; to[2] = a.z; to[3] = a.w;
                to[4] = b.x; to[5] = b.y; to[6] = b.z; to[7] = b.w;
            };
            if (KIND == 0) {
                load(dOut + (size_t)p * C + cg * 8, v);
            } else {
                const Pixel q = pixelOf(p, total, W, H);
                if (KIND == 1) {
                    const size_t row = (size_t)(2 * W) * Cd;
                    const float* src = dOut + ((size_t)q.n * 2 * H + 2 * q.y) * row + (size_t)(2 * q.x) * Cd + cg * 8;
                    float b[8], c[8], d[8];
                    load(src, v); load(src + Cd, b); load(src + row, c); load(src + row + Cd, d);
#pragma unroll
                    for (int j = 0; j < 8; j++) v[j] = v[j] + b[j] + c[j] + d[j];
                } else {
                    float b[8];
                    load(dOut + (size_t)p * Cd + (Cd - C) + cg * 8, v);
                    load(dPool + (((size_t)q.n * (H / 2) + q.y / 2) * (W / 2) + q.x / 2) * C + cg * 8, b);
#pragma unroll
                    for (int j = 0; j < 8; j++) v[j] = v[j] + 0.25f * b[j];
                }
            }
            const bf16* ye = reinterpret_cast<const bf16*>(&yq);
            uint4 out;
            bf16* oe = reinterpret_cast<bf16*>(&out);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                oe[j] = __float2bfloat16(__bfloat162float(ye[j]) > 0.0f ? v[j] : 0.0f);
                acc[j] += __bfloat162float(oe[j]);
            }
            *(reinterpret_cast<uint4*>(dPre + (size_t)p * C) + cg) = out;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) sums[slot * C + cg * 8 + j] = acc[j];
    }
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        float s = 0.0f;
        for (int k = 0; k < slots; k++) s += sums[k * C + c];
        if (s != 0.0f) atomicAdd(&db[c], s);
    }
}
template <int KIND>
cudaError_t launchPreGrad(const float* dOut, int Cd, const float* dPool, const bf16* y, int N, int H, int W, int C,
                          bf16* dPre, float* db, cudaStream_t s) {
    const int slots = 256 / (C / 8);
    const long long blocks = ((long long)N * H * W + slots - 1) / slots;
    preGradKernel<KIND><<<(int)std::min<long long>(blocks, 148 * 8), 256, sizeof(float) * slots * C, s>>>(
        dOut, Cd, dPool, y, N, H, W, C, dPre, db);
    return cudaGetLastError();
}
// 1x1 output layer, forward: pred[p][k] = b[k] + sum_c d[p][c] w[c][k].
__global__ void outForwardKernel(const bf16* d, long long pixels, int C, const float* w, const float* b, float* pred) {
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= pixels) return;
    float s[kOutChannels] = {b[0], b[1], b[2]};
    for (int c8 = 0; c8 < C; c8 += 8) {
        uint4 q = *reinterpret_cast<const uint4*>(d + p * C + c8);
        const bf16* e = reinterpret_cast<const bf16*>(&q);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            float v = __bfloat162float(e[j]);
            for (int k = 0; k < kOutChannels; k++) s[k] += v * w[(c8 + j) * kOutChannels + k];
        }
    }
    for (int k = 0; k < kOutChannels; k++) pred[p * kOutChannels + k] = s[k];
}
// The parameters' BF16 copies, after an Adam step when ADAM: wbf in the flat
// layout, wT K-major per 3x3 layer (wT[tap][co][ci] = w[tap][ci][co]). A block
// owns 16 input channels of one tap of one layer (16 * cout consecutive
// parameters, transposed through shared memory into 32-byte runs of wT), or a
// layer's bias, or the output layer. One launch of ~830 blocks replaces Adam,
// the conversion and 18 transposes (73 us, launch-bound). Bound by the latency
// of a thread's parameters one after another: 24 us in blocks of 128 threads,
// 12 in blocks of 512 (32 MB of traffic: 5 us).
constexpr int kWeightThreads = 512;
struct WeightTable {
    int blocks[19];               // first block of each layer's entries (taps x cin / 16, then its bias)
    int cin[19], cout[19];
    unsigned wOffset[19], bOffset[19];
    int total;                    // blocks in all
};
template <bool ADAM>
__global__ void __launch_bounds__(kWeightThreads) weightsKernel(const WeightTable T, float* p, const float* g, float* m, float* v,
                                                     float lr, float b1, float b2, float eps, float c1, float c2,
                                                     bf16* wbf, bf16* wT) {
    __shared__ bf16 tile[16 * 129];  // [ci][co], padded against bank conflicts
    int l = 0;
    while (l < 18 && (int)blockIdx.x >= T.blocks[l + 1]) l++;
    const int cin = T.cin[l], cout = T.cout[l], part = (int)blockIdx.x - T.blocks[l];
    const int groups = l < 18 ? 9 * (cin / 16) : 0;
    const bool transposed = part < groups;
    const size_t first = transposed ? T.wOffset[l] + (size_t)part * 16 * cout : l < 18 ? T.bOffset[l] : T.wOffset[l];
    const int count = transposed ? 16 * cout : l < 18 ? cout : cin * cout + cout;
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
        const size_t k = first + i;
        float x = p[k];
        if (ADAM) {
            const float gi = g[k];
            const float mi = b1 * m[k] + (1.0f - b1) * gi, vi = b2 * v[k] + (1.0f - b2) * gi * gi;
            m[k] = mi;
            v[k] = vi;
            x -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
            p[k] = x;
        }
        const bf16 h = __float2bfloat16(x);
        wbf[k] = h;
        if (transposed) tile[i / cout * 129 + i % cout] = h;
    }
    if (!transposed) return;
    __syncthreads();
    const int tap = part / (cin / 16), ci0 = part % (cin / 16) * 16;
    bf16* out = wT + T.wOffset[l] + (size_t)tap * cin * cout + ci0;
    for (int i = threadIdx.x; i < 16 * cout; i += blockDim.x)
        out[(size_t)(i / 16) * cin + i % 16] = tile[i % 16 * 129 + i / 16];
}
// Network input straight from the running sums: the AOVs of RtxReadAovs
// (sum / samples, normalised normal, distance / samples), then the input
// transform of inputKernel, for every pixel of the padded frame (beyond w x h
// the edge pixels repeat).
__global__ void sumsInputKernel(const float* sums, const float* depthSums, unsigned samples, int h, int w, int H,
                                int W, bf16* x0, unsigned char* coverage) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)H * W) return;
    const int X = (int)(i % W), Y = (int)(i / W);
    const size_t src = (size_t)min(Y, h - 1) * w + min(X, w - 1);
    const float* a = sums + src * 10;
    const float inv = 1.0f / (float)samples;
    const float3 c = scale(v3(a[0], a[1], a[2]), inv), al = scale(v3(a[3], a[4], a[5]), inv);
    const float3 nr = normalize(v3(a[6], a[7], a[8]));
    const float depth = depthSums[src] * inv;
    if (X < w && Y < h) coverage[src] = __float_as_uint(a[9]) != 0u;
    float v[kInputPadded] = {};
    v[0] = log1pf(fmaxf(c.x, 0.0f)); v[1] = log1pf(fmaxf(c.y, 0.0f)); v[2] = log1pf(fmaxf(c.z, 0.0f));
    v[3] = al.x; v[4] = al.y; v[5] = al.z;
    v[6] = nr.x; v[7] = nr.y; v[8] = nr.z;
    v[9] = log1pf(fmaxf(depth, 0.0f));
    uint4 packed[2];
    uint32_t* words = reinterpret_cast<uint32_t*>(packed);
#pragma unroll
    for (int j = 0; j < kInputPadded / 2; j++) {
        __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        words[j] = *reinterpret_cast<uint32_t*>(&pair);
    }
    uint4* o = reinterpret_cast<uint4*>(x0 + (size_t)i * kInputPadded);
    o[0] = packed[0];
    o[1] = packed[1];
}
// Output layer and crop in one pass: the 1x1 convolution of outForwardKernel
// (same summation order) for the pixels inside w x h, then expm1 and the
// clamp of outputKernel.
__global__ void outputFusedKernel(const bf16* d, int H, int W, int h, int w, int C, const float* wt, const float* b,
                                  float* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * h) return;
    const int x = i % w, y = i / w;
    const long long p = (long long)y * W + x;
    float s[kOutChannels] = {b[0], b[1], b[2]};
    for (int c8 = 0; c8 < C; c8 += 8) {
        uint4 q = *reinterpret_cast<const uint4*>(d + p * C + c8);
        const bf16* e = reinterpret_cast<const bf16*>(&q);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            float v = __bfloat162float(e[j]);
            for (int k = 0; k < kOutChannels; k++) s[k] += v * wt[(c8 + j) * kOutChannels + k];
        }
    }
    for (int k = 0; k < kOutChannels; k++) out[(size_t)i * 3 + k] = fmaxf(expm1f(s[k]), 0.0f);
}

// Network output (log space, padded frame) to linear radiance (w x h x 3).
__global__ void outputKernel(const float* pred, int H, int W, int h, int w, float* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * h) return;
    int x = i % w, y = i / w;
    const float* p = pred + ((size_t)y * W + x) * kOutChannels;
    for (int k = 0; k < kOutChannels; k++) out[(size_t)i * 3 + k] = fmaxf(expm1f(p[k]), 0.0f);
}

template <int CT>
cudaError_t launchWgrad(const bf16* x, const bf16* dy, int N, int H, int W, int Cin, int Cout, float* dw, cudaStream_t s) {
    long long segments = (long long)N * H * ((W + 15) / 16);
    int chunks = (int)std::min<long long>(64, std::max<long long>(1, segments / 64));
    int per = (int)((segments + chunks - 1) / chunks);
    dim3 grid(chunks, 9 * (Cin / 16), Cout / CT);
    wgradKernel<CT><<<grid, 128, 0, s>>>(x, dy, N, H, W, Cin, Cout, per, dw);
    return cudaGetLastError();
}
// Weight gradient: the tcgen05 kernel (rt_wgrad_tc.cu) unless the
// single-role convolution path is selected (RtxSetConvPath(1)), then the
// warp-level MMA kernel above.
cudaError_t wgrad(const bf16* x, const bf16* dy, int N, int H, int W, int Cin, int Cout, float* dw, int* errorFlag,
                  cudaStream_t s) {
    if (convPath() == 0 && wgradTcSupported(Cin, Cout)) {
        cudaError_t e = wgradTc(x, dy, N, H, W, Cin, Cout, dw, errorFlag, s);
        if (e != cudaErrorNotSupported) return e;
    }
    if (Cout % 64 == 0) return launchWgrad<64>(x, dy, N, H, W, Cin, Cout, dw, s);
    if (Cout % 48 == 0) return launchWgrad<48>(x, dy, N, H, W, Cin, Cout, dw, s);
    if (Cout % 32 == 0) return launchWgrad<32>(x, dy, N, H, W, Cin, Cout, dw, s);
    return launchWgrad<16>(x, dy, N, H, W, Cin, Cout, dw, s);
}

}  // namespace

// Activations and gradients for one (n, H, W) configuration.
struct Unet::Activations {
    int n = 0, H = 0, W = 0;
    bool training = false;
    bf16* x0 = nullptr;
    bf16* a[18] = {};        // outputs of the 18 3x3 layers
    bf16* pool[4] = {};      // pooled encoder outputs (levels 1..4 inputs)
    bf16* cat[4] = {};       // decoder inputs: concat(upsample(lower), skip) at levels 3..0
    // Two-pass form of the decoders' first convolutions (inference): the
    // upsampled half at half resolution (4 parity blocks of cout channels)
    // and each layer's combined weights (low half, skip half).
    bf16* upHalf = nullptr;
    bf16* upWeights[4] = {};
    bf16* skipWeights[4] = {};
    float* pred = nullptr;   // network output, log space
    float* dAct[18] = {};    // fp32 gradients of the outputs of each level's first layers (even k)
    float* dCat[4] = {};     // of the decoders' inputs
    float* dPool[4] = {};    // of the pooled inputs
    bf16* dPre[18] = {};     // gradients at the layers' pre-activations, bf16
    float* loss = nullptr;
    int* batch = nullptr;
    unsigned char* flips = nullptr;
    std::vector<void*> owned;
    template <class T>
    cudaError_t make(T*& p, size_t count) {
        cudaError_t e = rt::deviceAlloc(&p, sizeof(T) * std::max<size_t>(count, 1));
        if (e == cudaSuccess) owned.push_back(p);
        return e;
    }
    ~Activations() {
        for (void* p : owned) rt::deviceFree(p);
    }
};

namespace {
// Layer table: 10 encoder/bottleneck layers then 8 decoder layers.
void layerTable(std::vector<UnetLayer>& layers, size_t& params) {
    int cin[18], cout[18];
    int prev = kInputPadded, k = 0;
    for (int l = 0; l < 5; l++) {
        cin[k] = prev; cout[k] = kWidths[l]; k++;
        cin[k] = kWidths[l]; cout[k] = kWidths[l]; k++;
        prev = kWidths[l];
    }
    for (int l = 3; l >= 0; l--) {
        cin[k] = prev + kWidths[l]; cout[k] = kWidths[l]; k++;
        cin[k] = kWidths[l]; cout[k] = kWidths[l]; k++;
        prev = kWidths[l];
    }
    params = 0;
    for (int i = 0; i < 18; i++) {
        UnetLayer L{cin[i], cout[i], params, params + (size_t)9 * cin[i] * cout[i]};
        params = L.bOffset + cout[i];
        layers.push_back(L);
    }
    UnetLayer out{kWidths[0], kOutChannels, params, params + (size_t)kWidths[0] * kOutChannels};
    params = out.bOffset + kOutChannels;
    layers.push_back(out);
}
}  // namespace

Unet::Unet(unsigned seed) {
    layerTable(layers_, params_);
    std::vector<float> host(params_, 0.0f);
    std::mt19937 rng(seed);
    for (size_t l = 0; l < layers_.size(); l++) {
        const UnetLayer& L = layers_[l];
        bool out = l + 1 == layers_.size();
        int fanIn = (out ? 1 : 9) * (l == 0 ? kInputChannels : L.cin);
        std::normal_distribution<float> dist(0.0f, std::sqrt((out ? 1.0f : 2.0f) / (float)fanIn));
        size_t nw = L.bOffset - L.wOffset;
        for (size_t i = 0; i < nw; i++) {
            float v = dist(rng);
            if (l == 0) {  // padding input channels carry zeros: their weights stay zero
                size_t ci = (i / L.cout) % L.cin;
                if ((int)ci >= kInputChannels) v = 0.0f;
            }
            host[L.wOffset + i] = v;
        }
    }
    // Every copy and fill goes through stream_: it is non-blocking, so it is
    // not ordered after work on the legacy default stream. Nothing is launched
    // once a step has failed.
    auto attempt = [&](auto step) { if (status_ == cudaSuccess) status_ = step(); };
    attempt([&] { return rt::deviceAlloc(&master_, sizeof(float) * params_); });
    attempt([&] { return rt::deviceAlloc(&grad_, sizeof(float) * params_); });
    attempt([&] { return rt::deviceAlloc(&adamM_, sizeof(float) * params_); });
    attempt([&] { return rt::deviceAlloc(&adamV_, sizeof(float) * params_); });
    attempt([&] { return rt::deviceAlloc(&wbf_, sizeof(bf16) * params_); });
    attempt([&] { return rt::deviceAlloc(&wT_, sizeof(bf16) * params_); });
    attempt([&] { return rt::deviceAlloc(&convError_, sizeof(int)); });
    attempt([&] { return cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking); });
    attempt([&] { return cudaStreamCreateWithFlags(&side_, cudaStreamNonBlocking); });
    attempt([&] { return cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming); });
    attempt([&] { return cudaEventCreateWithFlags(&join_, cudaEventDisableTiming); });
    attempt([&] { return cudaMemsetAsync(convError_, 0, sizeof(int), stream_); });
    attempt([&] { return cudaMemcpyAsync(master_, host.data(), sizeof(float) * params_, cudaMemcpyHostToDevice, stream_); });
    attempt([&] { return cudaMemsetAsync(adamM_, 0, sizeof(float) * params_, stream_); });
    attempt([&] { return cudaMemsetAsync(adamV_, 0, sizeof(float) * params_, stream_); });
    attempt([&] { return syncWeights(stream_); });
    attempt([&] { return cudaStreamSynchronize(stream_); });
}

Unet::~Unet() {
    settleStreams();
    delete act_;
    rt::deviceFree(master_); rt::deviceFree(grad_); rt::deviceFree(adamM_); rt::deviceFree(adamV_); rt::deviceFree(wbf_); rt::deviceFree(wT_); rt::deviceFree(convError_);
    if (fork_) cudaEventDestroy(fork_);
    if (join_) cudaEventDestroy(join_);
    if (side_) cudaStreamDestroy(side_);
    if (stream_) cudaStreamDestroy(stream_);
}

namespace {
WeightTable weightTable(const std::vector<UnetLayer>& layers) {
    WeightTable T{};
    int blocks = 0;
    for (size_t l = 0; l < layers.size(); l++) {
        const UnetLayer& L = layers[l];
        T.blocks[l] = blocks;
        T.cin[l] = L.cin; T.cout[l] = L.cout;
        T.wOffset[l] = (unsigned)L.wOffset; T.bOffset[l] = (unsigned)L.bOffset;
        blocks += l + 1 < layers.size() ? 9 * (L.cin / 16) + 1 : 1;
    }
    T.total = blocks;
    return T;
}
}  // namespace

cudaError_t Unet::syncWeights(cudaStream_t s) {
    const WeightTable T = weightTable(layers_);
    weightsKernel<false><<<T.total, kWeightThreads, 0, s>>>(T, master_, nullptr, nullptr, nullptr, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f,
                                                 1.0f, wbf_, wT_);
    return cudaGetLastError();
}

cudaError_t Unet::checkConvolutions(std::string& error) {
    int flag = 0;
    cudaError_t e = cudaMemcpy(&flag, convError_, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return e;
    if (!flag) return cudaSuccess;
    e = cudaMemsetAsync(convError_, 0, sizeof(int), stream_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
    if (e != cudaSuccess) return e;
    error = "tensor-core convolution stopped: a wait on the tensor cores ran past its limit";
    return cudaErrorLaunchTimeout;
}

cudaError_t Unet::getParams(float* host) const {
    cudaError_t e = cudaMemcpyAsync(host, master_, sizeof(float) * params_, cudaMemcpyDeviceToHost, stream_);
    return e == cudaSuccess ? cudaStreamSynchronize(stream_) : e;
}
cudaError_t Unet::setParams(const float* host) {
    cudaError_t e = cudaMemcpyAsync(master_, host, sizeof(float) * params_, cudaMemcpyHostToDevice, stream_);
    if (e != cudaSuccess) return e;
    e = syncWeights(stream_);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(stream_);
}

void Unet::settleStreams() {
    if (stream_) settle(stream_);
    if (side_) settle(side_);
}

cudaError_t Unet::ensure(int n, int h, int w, bool training) {
    int H = (h + 15) / 16 * 16, W = (w + 15) / 16 * 16;
    if (act_ && act_->n == n && act_->H == H && act_->W == W && (act_->training || !training)) return cudaSuccess;
    settleStreams();
    delete act_;
    act_ = new Activations();
    act_->n = n; act_->H = H; act_->W = W; act_->training = training;
    const cudaError_t e = allocate(*act_);
    if (e != cudaSuccess) {  // nothing half made is found by the next call of this size
        delete act_;
        act_ = nullptr;
    }
    return e;
}

cudaError_t Unet::allocate(Activations& A) const {
    const int n = A.n, H = A.H, W = A.W;
    const bool training = A.training;
    cudaError_t e = cudaSuccess;
    auto px = [&](int level) { return (size_t)n * (H >> level) * (W >> level); };
    if ((e = A.make(A.x0, px(0) * kInputPadded)) != cudaSuccess) return e;
    for (int k = 0; k < 18; k++) {
        int level = k < 10 ? k / 2 : 3 - (k - 10) / 2;
        if ((e = A.make(A.a[k], px(level) * layers_[k].cout)) != cudaSuccess) return e;
        if (training && (e = A.make(A.dPre[k], px(level) * layers_[k].cout)) != cudaSuccess) return e;
        if (training && k % 2 == 0 && (e = A.make(A.dAct[k], px(level) * layers_[k].cout)) != cudaSuccess) return e;
    }
    for (int l = 1; l <= 4; l++) {
        if ((e = A.make(A.pool[l - 1], px(l) * kWidths[l - 1])) != cudaSuccess) return e;
        if (training && (e = A.make(A.dPool[l - 1], px(l) * kWidths[l - 1])) != cudaSuccess) return e;
    }
    size_t upHalf = 0;
    for (int j = 0; j < 4; j++) {  // decoder level 3 - j
        int level = 3 - j;
        const UnetLayer& L = layers_[10 + 2 * j];
        const int Cl = layers_[9 + 2 * j].cout;
        if (upsampledSplitSupported(L.cin, L.cout, Cl)) {
            upHalf = std::max(upHalf, px(level) * L.cout);  // (H / 2) x (W / 2) x 4 cout
            if ((e = A.make(A.upWeights[j], (size_t)9 * 4 * L.cout * Cl)) != cudaSuccess) return e;
            if ((e = A.make(A.skipWeights[j], (size_t)9 * L.cout * (L.cin - Cl))) != cudaSuccess) return e;
        }
        if ((training || !A.upWeights[j]) && (e = A.make(A.cat[j], px(level) * layers_[10 + 2 * j].cin)) != cudaSuccess) return e;
        if (training && (e = A.make(A.dCat[j], px(level) * layers_[10 + 2 * j].cin)) != cudaSuccess) return e;
    }
    if (upHalf && (e = A.make(A.upHalf, upHalf)) != cudaSuccess) return e;
    // Inference writes it, of one image (also over the buffers of a training
    // call of that size); training's output layer is headKernel's.
    if (n == 1 && (e = A.make(A.pred, px(0) * kOutChannels)) != cudaSuccess) return e;
    if (training) {
        if ((e = A.make(A.loss, 1)) != cudaSuccess) return e;
        if ((e = A.make(A.batch, n)) != cudaSuccess) return e;
        if ((e = A.make(A.flips, n)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t Unet::forward(cudaStream_t s, bool training, bool outputLayer, const ConvHead* head, bool* headDone) {
    if (headDone) *headDone = false;
    Activations& A = *act_;
    const int n = A.n;
    cudaError_t e;
    const bf16* x = A.x0;
    int k = 0;
    // The decoders' combined weights, 14 us of small kernels at 1080p that
    // only the decoders need, beside the encoder.
    const bool combine = !training && convPath() == 0;
    struct Join {  // the side stream's work never outlives the call's order on s
        cudaStream_t s;
        cudaEvent_t pending;
        ~Join() {
            if (pending) cudaStreamWaitEvent(s, pending, 0);
        }
    } join{s, nullptr};
    if (combine) {
        if ((e = cudaEventRecord(fork_, s)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(side_, fork_, 0)) != cudaSuccess) return e;
        cudaError_t made = cudaSuccess;
        for (int j = 0; j < 4; j++) {
            const UnetLayer& L = layers_[10 + 2 * j];
            if (A.upWeights[j] && made == cudaSuccess)
                made = combineUpsampledWeights(wT_ + L.wOffset, L.cout, L.cin, layers_[9 + 2 * j].cout, A.upWeights[j],
                                               A.skipWeights[j], side_);
        }
        e = cudaEventRecord(join_, side_);
        join.pending = join_;
        if (made != cudaSuccess) e = made;
        if (e != cudaSuccess) return e;
    }
    for (int l = 0; l < 5; l++) {
        int H = A.H >> l, W = A.W >> l;
        if (l > 0) {
            int C = kWidths[l - 1];
            poolKernel<<<blocksFor((long long)n * H * W * (C / 8), 256), 256, 0, s>>>(A.a[k - 1], n, H * 2, W * 2, C, A.pool[l - 1]);
            x = A.pool[l - 1];
        }
        for (int r = 0; r < 2; r++, k++) {
            const UnetLayer& L = layers_[k];
            if ((e = convTc(x, nullptr, 0, n, H, W, L.cin, wT_ + L.wOffset, false, master_ + L.bOffset, L.cout, A.a[k], nullptr, true, false, convError_, s)) != cudaSuccess) return e;
            x = A.a[k];
        }
    }
    if (combine && (e = cudaStreamWaitEvent(s, join_, 0)) != cudaSuccess) return e;
    join.pending = nullptr;
    for (int j = 0; j < 4; j++) {
        int level = 3 - j, H = A.H >> level, W = A.W >> level;
        int Cl = layers_[k - 1].cout, Cs = kWidths[level];
        const bf16* low = A.a[k - 1];
        const bf16* skip = A.a[2 * level + 1];
        for (int r = 0; r < 2; r++, k++) {
            const UnetLayer& L = layers_[k];
            if (r == 0 && (training || (!A.upWeights[j] && A.cat[j] && convPath() == 0))) {
                // The weight gradient reads the concatenated input; at inference
                // the streamed convolution does (8 + 22 us against 73 for the
                // single-role kernel reading its halves in place, 240 x 136),
                // and no other: buffers left by a training call of this size
                // hold a concatenation for every level.
                upConcatKernel<<<blocksFor((long long)n * H * W * ((Cl + Cs) / 8), 256), 256, 0, s>>>(low, Cl, skip, Cs, n, H, W, A.cat[j]);
                e = convTc(A.cat[j], nullptr, 0, n, H, W, L.cin, wT_ + L.wOffset, false, master_ + L.bOffset, L.cout, A.a[k], nullptr, true, false, convError_, s);
            } else if (r == 0 && A.upWeights[j] && combine) {
                // Inference, two passes: the upsampled half at half
                // resolution (4 parity blocks), then the skip half adding it.
                e = convTc(low, nullptr, 0, n, H / 2, W / 2, Cl, A.upWeights[j], false, nullptr, 4 * L.cout, A.upHalf,
                           nullptr, false, false, convError_, s, nullptr, nullptr, true);
                if (e == cudaSuccess)
                    e = convTc(skip, nullptr, 0, n, H, W, Cs, A.skipWeights[j], false, master_ + L.bOffset, L.cout, A.a[k],
                               nullptr, true, false, convError_, s, A.upHalf);
            } else if (r == 0) {
                // Inference: the convolution reads [upsample(low), skip] in place.
                e = convTc(skip, low, Cl, n, H, W, L.cin, wT_ + L.wOffset, false, master_ + L.bOffset, L.cout, A.a[k], nullptr, true, false, convError_, s);
            } else if (k == 17 && head && !training && convPath() == 0 && convPipePreferred(L.cin, L.cout, 0)) {
                // The last convolution with the output head in its epilogue.
                e = convTc(A.a[k - 1], nullptr, 0, n, H, W, L.cin, wT_ + L.wOffset, false, master_ + L.bOffset, L.cout,
                           nullptr, nullptr, true, false, convError_, s, nullptr, head);
                if (e == cudaSuccess && headDone) *headDone = true;
                if (e == cudaErrorNotSupported)
                    e = convTc(A.a[k - 1], nullptr, 0, n, H, W, L.cin, wT_ + L.wOffset, false, master_ + L.bOffset,
                               L.cout, A.a[k], nullptr, true, false, convError_, s);
            } else {
                e = convTc(A.a[k - 1], nullptr, 0, n, H, W, L.cin, wT_ + L.wOffset, false, master_ + L.bOffset, L.cout, A.a[k], nullptr, true, false, convError_, s);
            }
            if (e != cudaSuccess) return e;
        }
    }
    if (!outputLayer) return cudaGetLastError();
    const UnetLayer& O = layers_[18];
    long long pixels = (long long)n * A.H * A.W;
    outForwardKernel<<<blocksFor(pixels, 128), 128, 0, s>>>(A.a[17], pixels, O.cin, master_ + O.wOffset, master_ + O.bOffset, A.pred);
    return cudaGetLastError();
}

cudaError_t Unet::lossAndBackward(const float* targets, const int* batch, const unsigned char* flips, float* loss,
                                  cudaStream_t s) {
    Activations& A = *act_;
    const int n = A.n;
    cudaError_t e;
    if ((e = cudaMemsetAsync(grad_, 0, sizeof(float) * params_, s)) != cudaSuccess) return e;
    const UnetLayer& O = layers_[18];
    const long long pixels0 = (long long)n * A.H * A.W;
    headKernel<<<(int)std::min<long long>(blocksFor(pixels0, 64), 148 * 3), 128, 0, s>>>(
        A.a[17], targets, n, A.H, A.W, batch, flips, master_ + O.wOffset, master_ + O.bOffset, A.dPre[17], loss,
        grad_ + O.wOffset, grad_ + O.bOffset, grad_ + layers_[17].bOffset);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // Layer k from the gradient at its pre-activation (A.dPre[k]): its weight
    // gradient, and its input's gradient into dIn (fp32) unless dIn is null.
    // Nothing on the way down to the first layer needs the weight gradients, so
    // they run on a stream of their own beside it: the deep levels' kernels
    // leave most SMs free. Eight steps of 32 x 128 x 128 pixels, copies
    // included: 18.6 ms in one stream, 16.7 ms so.
    if ((e = cudaEventRecord(fork_, s)) != cudaSuccess) return e;  // the cleared gradients
    if ((e = cudaStreamWaitEvent(side_, fork_, 0)) != cudaSuccess) return e;
    auto layerBack = [&](int k, const bf16* input, int H, int W, float* dIn) -> cudaError_t {
        const UnetLayer& L = layers_[k];
        cudaError_t err = cudaEventRecord(fork_, s);
        if (err == cudaSuccess) err = cudaStreamWaitEvent(side_, fork_, 0);
        if (err == cudaSuccess)
            err = wgrad(input, A.dPre[k], n, H, W, L.cin, L.cout, grad_ + L.wOffset, convError_, side_);
        if (err != cudaSuccess || !dIn) return err;
        return convTc(A.dPre[k], nullptr, 0, n, H, W, L.cout, wbf_ + L.wOffset, true, nullptr, L.cin, nullptr, dIn, false, false, convError_, s);
    };
    // Ends the fork whatever happened, so that nothing on the side stream
    // outlives the call's order on s.
    auto join = [&](cudaError_t result) {
        cudaError_t err = cudaEventRecord(join_, side_);
        if (err == cudaSuccess) err = cudaStreamWaitEvent(s, join_, 0);
        return result != cudaSuccess ? result : err;
    };
    // The second, then the first 3x3 layer of a level (k and k - 1).
    auto levelBack = [&](int k, const bf16* input, int H, int W, float* dIn) -> cudaError_t {
        cudaError_t err = layerBack(k, A.a[k - 1], H, W, A.dAct[k - 1]);
        if (err == cudaSuccess)
            err = launchPreGrad<0>(A.dAct[k - 1], 0, nullptr, A.a[k - 1], n, H, W, layers_[k - 1].cout, A.dPre[k - 1],
                                   grad_ + layers_[k - 1].bOffset, s);
        return err == cudaSuccess ? layerBack(k - 1, input, H, W, dIn) : err;
    };
    int k = 17;
    for (int j = 3; j >= 0; j--) {  // decoder level 3 - j, from the top (level 0) down
        int level = 3 - j, H = A.H >> level, W = A.W >> level;
        if ((e = levelBack(k, A.cat[j], H, W, A.dCat[j])) != cudaSuccess) return join(e);
        k -= 2;  // the layer below, whose output was upsampled; the skip half waits in dCat for the encoder
        if ((e = launchPreGrad<1>(A.dCat[j], layers_[k + 1].cin, nullptr, A.a[k], n, H / 2, W / 2, layers_[k].cout, A.dPre[k],
                                  grad_ + layers_[k].bOffset, s)) != cudaSuccess) return join(e);
    }
    // Bottleneck and encoder: k = 9 down to 0.
    for (int l = 4; l >= 0; l--, k -= 2) {
        int H = A.H >> l, W = A.W >> l;
        if ((e = levelBack(k, l == 0 ? A.x0 : A.pool[l - 1], H, W, l == 0 ? nullptr : A.dPool[l - 1])) != cudaSuccess) return join(e);
        // The encoder output of level l - 1 receives the pooled gradient and its skip gradient.
        if (l > 0 && (e = launchPreGrad<2>(A.dCat[4 - l], layers_[10 + 2 * (4 - l)].cin, A.dPool[l - 1], A.a[k - 2], n, H * 2,
                                           W * 2, kWidths[l - 1], A.dPre[k - 2], grad_ + layers_[k - 2].bOffset, s)) != cudaSuccess)
            return join(e);
    }
    return join(cudaGetLastError());
}

cudaError_t Unet::lossAndGradient(const float* aovs, const float* targets, int n, int h, int w, float* loss, float* grads,
                                  std::string& error) {
    if (h % 16 || w % 16) { error = "training crops must be multiples of 16 pixels"; return cudaErrorInvalidValue; }
    cudaError_t e = ensure(n, h, w, true);
    if (e != cudaSuccess) return e;
    Activations& A = *act_;
    float *dA = nullptr, *dT = nullptr;
    size_t px = (size_t)n * h * w;
    if ((e = rt::deviceAlloc(&dA, sizeof(float) * px * kInputChannels)) != cudaSuccess) return e;
    if ((e = rt::deviceAlloc(&dT, sizeof(float) * px * 3)) != cudaSuccess) { rt::deviceFree(dA); return e; }
    cudaMemcpyAsync(dA, aovs, sizeof(float) * px * kInputChannels, cudaMemcpyHostToDevice, stream_);
    cudaMemcpyAsync(dT, targets, sizeof(float) * px * 3, cudaMemcpyHostToDevice, stream_);
    inputKernel<<<blocksFor((long long)px, 256), 256, 0, stream_>>>(dA, n, h, w, A.H, A.W, A.x0, nullptr, nullptr);
    cudaMemsetAsync(A.loss, 0, sizeof(float), stream_);
    if ((e = forward(stream_, true, false)) == cudaSuccess) e = lossAndBackward(dT, nullptr, nullptr, A.loss, stream_);
    if (e == cudaSuccess) e = cudaMemcpyAsync(loss, A.loss, sizeof(float), cudaMemcpyDeviceToHost, stream_);
    if (e == cudaSuccess && grads) e = cudaMemcpyAsync(grads, grad_, sizeof(float) * params_, cudaMemcpyDeviceToHost, stream_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
    if (e == cudaSuccess) e = checkConvolutions(error);
    if (e != cudaSuccess) settleStreams();
    rt::deviceFree(dA); rt::deviceFree(dT);
    return e;
}

cudaError_t Unet::train(const float* aovs, const float* targets, int count, int h, int w, int steps, int batch,
                        float lr, unsigned seed, float* losses, std::string& error) {
    if (h % 16 || w % 16) { error = "training crops must be multiples of 16 pixels"; return cudaErrorInvalidValue; }
    if (batch < 1 || count < 1) { error = "empty training set"; return cudaErrorInvalidValue; }
    cudaError_t e = ensure(batch, h, w, true);
    if (e != cudaSuccess) return e;
    Activations& A = *act_;
    float *dA = nullptr, *dT = nullptr;
    size_t px = (size_t)count * h * w;
    if ((e = rt::deviceAlloc(&dA, sizeof(float) * px * kInputChannels)) != cudaSuccess) return e;
    if ((e = rt::deviceAlloc(&dT, sizeof(float) * px * 3)) != cudaSuccess) { rt::deviceFree(dA); return e; }
    cudaMemcpyAsync(dA, aovs, sizeof(float) * px * kInputChannels, cudaMemcpyHostToDevice, stream_);
    cudaMemcpyAsync(dT, targets, sizeof(float) * px * 3, cudaMemcpyHostToDevice, stream_);
    std::mt19937 rng(seed);
    std::vector<int> idx(batch);
    std::vector<unsigned char> flips(batch);
    std::vector<float> lossHost(steps, 0.0f);
    float* dLosses = nullptr;
    if ((e = rt::deviceAlloc(&dLosses, sizeof(float) * std::max(steps, 1))) != cudaSuccess) {
        settleStreams();
        rt::deviceFree(dA); rt::deviceFree(dT);
        return e;
    }
    cudaMemsetAsync(dLosses, 0, sizeof(float) * std::max(steps, 1), stream_);
    const size_t bpx = (size_t)batch * h * w;
    const WeightTable table = weightTable(layers_);
    for (int step = 0; step < steps && e == cudaSuccess; step++) {
        for (int b = 0; b < batch; b++) { idx[b] = (int)(rng() % (unsigned)count); flips[b] = (unsigned char)(rng() & 3u); }
        cudaMemcpyAsync(A.batch, idx.data(), sizeof(int) * batch, cudaMemcpyHostToDevice, stream_);
        cudaMemcpyAsync(A.flips, flips.data(), batch, cudaMemcpyHostToDevice, stream_);
        inputKernel<<<blocksFor((long long)bpx, 256), 256, 0, stream_>>>(dA, batch, h, w, A.H, A.W, A.x0, A.batch, A.flips);
        if ((e = forward(stream_, true, false)) != cudaSuccess) break;
        if ((e = lossAndBackward(dT, A.batch, A.flips, dLosses + step, stream_)) != cudaSuccess) break;
        adamStep_++;
        const float b1 = 0.9f, b2 = 0.999f;
        float c1 = 1.0f - std::pow(b1, (float)adamStep_), c2 = 1.0f - std::pow(b2, (float)adamStep_);
        weightsKernel<true><<<table.total, kWeightThreads, 0, stream_>>>(table, master_, grad_, adamM_, adamV_, lr, b1, b2, 1e-8f, c1,
                                                              c2, wbf_, wT_);
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        // The tiny host copies above wait for the stream; keep them ordered.
        if ((step & 63) == 63) e = cudaStreamSynchronize(stream_);
    }
    if (e == cudaSuccess && losses) e = cudaMemcpyAsync(losses, dLosses, sizeof(float) * steps, cudaMemcpyDeviceToHost, stream_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
    if (e == cudaSuccess) e = checkConvolutions(error);
    if (e != cudaSuccess) settleStreams();
    rt::deviceFree(dA); rt::deviceFree(dT); rt::deviceFree(dLosses);
    return e;
}

cudaError_t Unet::inferFromSums(const float* sums, const float* depthSums, unsigned samples, int h, int w,
                                float* radiance, unsigned char* coverage, cudaStream_t s) {
    cudaError_t e = ensure(1, h, w, false);
    if (e != cudaSuccess) return e;
    Activations& A = *act_;
    sumsInputKernel<<<blocksFor((long long)A.H * A.W, 256), 256, 0, s>>>(sums, depthSums, samples, h, w, A.H, A.W, A.x0,
                                                                        coverage);
    const UnetLayer& O = layers_[18];
    const ConvHead head{master_ + O.wOffset, master_ + O.bOffset, radiance, h, w};
    bool fused = false;
    if ((e = forward(s, false, false, &head, &fused)) != cudaSuccess) return e;
    if (!fused)
        outputFusedKernel<<<blocksFor((long long)w * h, 256), 256, 0, s>>>(A.a[17], A.H, A.W, h, w, O.cin,
                                                                          master_ + O.wOffset, master_ + O.bOffset,
                                                                          radiance);
    return cudaGetLastError();
}

cudaError_t Unet::inferDevice(const float* aovs, int h, int w, float* radiance, cudaStream_t s, std::string&) {
    cudaError_t e = ensure(1, h, w, false);
    if (e != cudaSuccess) return e;
    Activations& A = *act_;
    inputKernel<<<blocksFor((long long)A.H * A.W, 256), 256, 0, s>>>(aovs, 1, h, w, A.H, A.W, A.x0, nullptr, nullptr);
    if ((e = forward(s, false)) != cudaSuccess) return e;
    outputKernel<<<blocksFor((long long)w * h, 256), 256, 0, s>>>(A.pred, A.H, A.W, h, w, radiance);
    return cudaGetLastError();
}

// Checkpoint: "RTUNET01", parameter count (u64), Adam step (i64), optimiser
// state flag (u64), FP32 parameters, then Adam m and v when the flag is set.
cudaError_t Unet::save(const char* path, bool optimizerState, std::string& error) const {
    std::vector<float> host(params_ * (optimizerState ? 3 : 1));
    cudaError_t e = cudaMemcpyAsync(host.data(), master_, sizeof(float) * params_, cudaMemcpyDeviceToHost, stream_);
    if (optimizerState) {
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(host.data() + params_, adamM_, sizeof(float) * params_, cudaMemcpyDeviceToHost, stream_);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(host.data() + 2 * params_, adamV_, sizeof(float) * params_, cudaMemcpyDeviceToHost, stream_);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
    if (e != cudaSuccess) return e;
    FILE* f = std::fopen(path, "wb");
    if (!f) { error = std::string("cannot write ") + path; return cudaErrorInvalidValue; }
    const char magic[8] = {'R', 'T', 'U', 'N', 'E', 'T', '0', '1'};
    unsigned long long count = params_, state = optimizerState ? 1 : 0;
    long long step = optimizerState ? adamStep_ : 0;
    bool ok = std::fwrite(magic, 1, 8, f) == 8 && std::fwrite(&count, 8, 1, f) == 1 && std::fwrite(&step, 8, 1, f) == 1 &&
              std::fwrite(&state, 8, 1, f) == 1 && std::fwrite(host.data(), sizeof(float), host.size(), f) == host.size();
    ok = std::fclose(f) == 0 && ok;
    if (!ok) { error = std::string("short write to ") + path; return cudaErrorInvalidValue; }
    return cudaSuccess;
}

cudaError_t Unet::load(const char* path, std::string& error) {
    FILE* f = std::fopen(path, "rb");
    if (!f) { error = std::string("cannot read ") + path; return cudaErrorInvalidValue; }
    char magic[8];
    unsigned long long count = 0, state = 0;
    long long step = 0;
    std::vector<float> host;
    bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "RTUNET01", 8) == 0 && std::fread(&count, 8, 1, f) == 1 &&
              count == params_ && std::fread(&step, 8, 1, f) == 1 && std::fread(&state, 8, 1, f) == 1 && state <= 1;
    if (ok) {
        host.assign(params_ * (state ? 3 : 1), 0.0f);
        ok = std::fread(host.data(), sizeof(float), host.size(), f) == host.size() && std::fgetc(f) == EOF;
    }
    std::fclose(f);
    if (!ok) { error = std::string("not a denoiser checkpoint of this network: ") + path; return cudaErrorInvalidValue; }
    adamStep_ = state ? step : 0;
    cudaError_t e = cudaMemcpyAsync(master_, host.data(), sizeof(float) * params_, cudaMemcpyHostToDevice, stream_);
    if (state) {
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(adamM_, host.data() + params_, sizeof(float) * params_, cudaMemcpyHostToDevice, stream_);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(adamV_, host.data() + 2 * params_, sizeof(float) * params_, cudaMemcpyHostToDevice, stream_);
    } else {
        if (e == cudaSuccess) e = cudaMemsetAsync(adamM_, 0, sizeof(float) * params_, stream_);
        if (e == cudaSuccess) e = cudaMemsetAsync(adamV_, 0, sizeof(float) * params_, stream_);
    }
    if (e == cudaSuccess) e = syncWeights(stream_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream_);
    return e;
}

}  // namespace rt
