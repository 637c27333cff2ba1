// loss.cu - (1 - lambda) L1 + lambda (1 - SSIM) and its gradient (photometricLoss, Loss.cpp:47-184).
//
// The reference runs four separable passes over (channel, row) pairs with full-image scratch maps.
// Here two tiled kernels do the same arithmetic with the blurs staged in shared memory, one CTA per
// 32x16 tile and colour channel (the three channels in parallel CTAs: a CTA per tile walking the channels
// in turn was 11 % slower):
//   lossForwardKernel : L1 term + horizontal blur of x, y, x^2, y^2, xy + vertical blur + SSIM and
//                       its three per-pixel partials (passes 1 and 2), block partial sums in double;
//   lossBackwardKernel: horizontal + vertical blur of the partials and the chain rule into
//                       dL/drender (passes 3 and 4; the Gaussian blur is self-adjoint). One more block
//                       adds up the forward's partial sums: the loss, the PSNR and the statistics.
// Both are bound by instructions (0.64 issued per cycle and scheduler; the traffic stays in L2): a thread
// slides its window over registers (4 columns, or 2 rows: 1.3 shared loads per tap instead of 2 to 5) and
// two maps share an instruction. Loss per step, 640x480: 55.7 -> 42.0 us, 320x240: 25.1 -> 19.5,
// 96x72: 15.6 -> 13.3, where a kernel of its own for the sums cost 2 us.
// Zero padding is reproduced by loading zeros outside the image: the reference skips out-of-image
// taps, and adding w * 0 to the running sums leaves every intermediate value unchanged, so each
// per-pixel value keeps the reference's rounding (the file is compiled with -fmad=false). The
// block sums are reduced in a fixed order, so the loss is deterministic.

#include "common.cuh"
#include "kernels.h"
#include "paired.cuh"

#include <cmath>

namespace u3dg {

namespace {

constexpr int kR = 5;                    // 11x11 window (Loss.cpp:11)
constexpr int kTW = 32, kTH = 16;        // output tile
constexpr int kIW = kTW + 2 * kR, kIH = kTH + 2 * kR;
constexpr int kThreads = 256;

// The 11 blur weights, passed to the loss kernels by value: kernel parameters sit in the constant
// bank like a __constant__ array, but need no upload into each device context (no synchronous copy
// before the first launch, nothing to redo after a context is recreated, nothing shared between host
// threads), and a captured graph keeps them with the launch.
struct SsimWindow {
    float w[2 * kR + 1];
    float one = 1.0f; // addProduct
};

// The window exactly as Loss.cpp:15-27 builds it (host float arithmetic with glibc expf).
struct HostWindow : SsimWindow {
    HostWindow()
    {
        float sum = 0;
        for (int k = -kR; k <= kR; ++k) {
            w[k + kR] = std::exp(-float(k * k) / (2.0f * 1.5f * 1.5f));
            sum += w[k + kR];
        }
        for (float &v : w)
            v /= sum;
    }
};

__device__ __forceinline__ double blockSumDouble(double v)
{
    __shared__ double warpSums[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0)
        warpSums[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kThreads / 32; ++w)
            t += warpSums[w];
    __syncthreads();
    return t;
}

// A tile's halo rows hold pixels side by side; H outputs of the horizontal blurs lie in groups of kQuad columns,
// V outputs of the vertical ones in pairs of rows, so that a thread slides its window over registers.
constexpr int kQuad = 4, kQuads = kTW / kQuad, kRowPairs = kTH / 2;
static_assert(kIH * kQuads <= kThreads && kRowPairs * kTW == kThreads, "one group per thread");

// s + p, each lane rounded, p a paired product: a paired add would be fused with the product, a multiplication
// by a 1 that the compiler does not know is not.
__device__ __forceinline__ float2 addProduct(const SsimWindow &win, float2 s, float2 p) { return fma2rn(p, both(win.one), s); }

// The image position and channel of a block's tile.
struct LossTile {
    int x0, y0, c;
};

__device__ __forceinline__ LossTile lossTile(int block, int W, int H)
{
    const int tx = (W + kTW - 1) / kTW, ty = (H + kTH - 1) / kTH, row = block / tx;
    return {block % tx * kTW, row % ty * kTH, row / ty};
}

// f(row, column, inside the image, pixel index) for every place of a tile with its halo: a thread takes one
// column in every kHaloStep-th row.
constexpr int kHaloStep = kThreads / kIW;

template <class F>
__device__ __forceinline__ void forHalo(int x0, int y0, int W, int H, F f)
{
    const int ix = threadIdx.x % kIW, first = threadIdx.x / kIW, gx = x0 + ix - kR, gy0 = y0 + first - kR;
    const bool column = gx >= 0 && gx < W;
    const long long at = (long long)gy0 * W + gx;
#pragma unroll
    for (int r = 0; r < (kIH + kHaloStep - 1) / kHaloStep; ++r) {
        const int iy = first + r * kHaloStep, gy = gy0 + r * kHaloStep;
        if (first < kHaloStep && iy < kIH)
            f(iy, ix, column && gy >= 0 && gy < H, size_t(at + (long long)r * kHaloStep * W));
    }
}

__global__ void __launch_bounds__(kThreads) lossForwardKernel(const float *render, const float *targetF,
                                                              const uint8_t *targetU8, int W, int H, float lambda,
                                                              float *grad, float *abc, double *blockSums,
                                                              const StepDesc *desc, const SsimWindow cWin)
{
    pdlEntry();
    if (desc)
        targetU8 = desc->target;
    __shared__ __align__(16) float2 sIn[kIH][kIW];                        // x, y
    __shared__ __align__(16) float2 hMean[kIH][kTW], hSquare[kIH][kTW];   // blurred x, y; x^2, y^2
    __shared__ __align__(16) float hCross[kIH][kTW];                      // xy
    const LossTile tile = lossTile(blockIdx.x, W, H);
    const int x0 = tile.x0, y0 = tile.y0, c = tile.c, tid = threadIdx.x;
    const size_t P = size_t(W) * H;
    const float invCount = 1.0f / float(P * 3);
    const float l1Scale = (1.0f - lambda) * invCount;
    const float dLds = -lambda * invCount;
    const float kC1 = 0.01f * 0.01f, kC2 = 0.03f * 0.03f;
    const float inv255 = 1.0f / 255.0f;
    double l1 = 0.0, ssim = 0.0, sq = 0.0;
    forHalo(x0, y0, W, H, [&](int iy, int ix, bool in, size_t pixel) {
        float a = 0.0f, b = 0.0f;
        if (in) {
            a = render[pixel * 3 + c];
            b = targetU8 ? float(targetU8[pixel * 3 + c]) * inv255 : targetF[pixel * 3 + c];
        }
        sIn[iy][ix] = make_float2(a, b);
    });
    __syncthreads();
    const int ox = tid % kTW, oy = tid / kTW * 2, gx = x0 + ox;
    // L1 term for this thread's two pixels (Loss.cpp:68-74).
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int gy = y0 + oy + r;
        if (gx < W && gy < H) {
            const float2 v = sIn[oy + r + kR][ox + kR];
            const float d = v.x - v.y;
            l1 += fabs(double(d));
            const double dd = double(v.x) - double(v.y);
            sq += dd * dd;
            if (!(lambda > 0.0f)) // else the backward kernel's
                grad[(size_t(gy) * W + gx) * 3 + c] = l1Scale * (d > 0 ? 1.0f : (d < 0 ? -1.0f : 0.0f));
        }
    }
    if (lambda > 0.0f) {
        // Horizontal blur of x, y, x^2, y^2, xy (Loss.cpp:77-94).
        if (tid < kIH * kQuads) {
            const int iy = tid / kQuads, q = tid % kQuads * kQuad;
            float2 in[kQuad + 2 * kR];
#pragma unroll
            for (int k = 0; k < kQuad + 2 * kR; k += 2) {
                const float4 two = *reinterpret_cast<const float4 *>(&sIn[iy][q + k]);
                in[k] = make_float2(two.x, two.y);
                in[k + 1] = make_float2(two.z, two.w);
            }
            float2 mean[kQuad], square[kQuad];
            float cross[kQuad];
#pragma unroll
            for (int k = 0; k < kQuad; ++k) {
                mean[k] = square[k] = both(0.0f);
                cross[k] = 0.0f;
#pragma unroll
                for (int t = 0; t <= 2 * kR; ++t) {
                    const float2 v = in[k + t], wv = mul2rn(both(cWin.w[t]), v);
                    mean[k] = addProduct(cWin, mean[k], wv);
                    square[k] = addProduct(cWin, square[k], mul2rn(wv, v));
                    cross[k] += wv.x * v.y;
                }
            }
#pragma unroll
            for (int k = 0; k < kQuad; k += 2) {
                *reinterpret_cast<float4 *>(&hMean[iy][q + k]) = make_float4(mean[k].x, mean[k].y, mean[k + 1].x, mean[k + 1].y);
                *reinterpret_cast<float4 *>(&hSquare[iy][q + k]) =
                    make_float4(square[k].x, square[k].y, square[k + 1].x, square[k + 1].y);
            }
            *reinterpret_cast<float4 *>(&hCross[iy][q]) = make_float4(cross[0], cross[1], cross[2], cross[3]);
        }
        __syncthreads();
        // Vertical blur, SSIM and its partials (Loss.cpp:113-137).
        float2 mean[2] = {}, square[2] = {};
        float cross[2] = {};
#pragma unroll
        for (int k = 0; k < 2 + 2 * kR; ++k) {
            const float2 m = hMean[oy + k][ox], s = hSquare[oy + k][ox];
            const float x = hCross[oy + k][ox];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = k - r;
                if (t < 0 || t > 2 * kR)
                    continue;
                const float w = cWin.w[t];
                mean[r] = addProduct(cWin, mean[r], mul2rn(both(w), m));
                square[r] = addProduct(cWin, square[r], mul2rn(both(w), s));
                cross[r] += w * x;
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int gy = y0 + oy + r;
            if (gx >= W || gy >= H)
                continue;
            const float mx = mean[r].x, my = mean[r].y;
            const float vx = square[r].x - mx * mx, vy = square[r].y - my * my, vxy = cross[r] - mx * my;
            const float a1 = 2 * mx * my + kC1, a2 = 2 * vxy + kC2;
            const float b1 = mx * mx + my * my + kC1, b2 = vx + vy + kC2;
            // SSIM and its partials, dLds apart.
            float v, dmu, dsq, dxy;
            auto partials = [&](auto by1, auto by2, auto by12, Operands &ops) {
                v = by12.under(a1 * a2, ops);
                dmu = by12.under(2 * my * a2 - 2 * my * a1, ops) - v * (by1.under(2 * mx, ops) - by2.under(2 * mx, ops));
                dsq = by2.under(-v, ops);
                dxy = by12.under(2 * a1, ops);
            };
            Operands ops;
            partials(Divisor(b1, ops), Divisor(b2, ops), Divisor(b1 * b2, ops), ops);
            if (!ops.usual())
                partials(Division(b1, ops), Division(b2, ops), Division(b1 * b2, ops), ops);
            ssim += double(v);
            const size_t o = size_t(c) * P + size_t(gy) * W + gx;
            abc[o] = dLds * dmu;
            abc[3 * P + o] = dLds * dsq;
            abc[6 * P + o] = dLds * dxy;
        }
    }
    __shared__ double warpSums[3][kThreads / 32];
    double part[3] = {l1, ssim, sq};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            part[k] += __shfl_down_sync(0xffffffffu, part[k], o);
    if ((tid & 31) == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            warpSums[k][tid >> 5] = part[k];
    __syncthreads();
    if (tid < 3) {
        double t = 0.0;
        for (int w = 0; w < kThreads / 32; ++w)
            t += warpSums[tid][w];
        blockSums[3 * blockIdx.x + tid] = t;
    }
}

// Where a step's loss values go.
struct LossOut {
    DevStats *stats;
    int iteration;
    const BinCounts *counts;
    float *out3, *psnrOut;
};

// Fixed-order sum of the block partials, LossValue, PSNR and the EMA stats, by one block of NT threads: the
// order is that of kFinalThreads threads, of which each thread here is several.
constexpr int kFinalThreads = 1024;

template <int NT>
__device__ __forceinline__ void lossFinalize(const double *blockSums, int blocks, int W, int H, float lambda, LossOut out,
                                             const StepDesc *desc)
{
    if (desc)
        out.iteration = desc->iteration + 1;
    if (out.counts != nullptr && out.counts->abortIter >= 0)
        out.stats = nullptr; // an aborted step leaves the statistics alone (it is replayed)
    __shared__ double warpSums[kFinalThreads / 32][3];
    for (int first = threadIdx.x; first < kFinalThreads; first += NT) {
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        for (int b = first; b < blocks; b += kFinalThreads) {
            s0 += blockSums[3 * b];
            s1 += blockSums[3 * b + 1];
            s2 += blockSums[3 * b + 2];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s0 += __shfl_down_sync(0xffffffffu, s0, o);
            s1 += __shfl_down_sync(0xffffffffu, s1, o);
            s2 += __shfl_down_sync(0xffffffffu, s2, o);
        }
        if ((first & 31) == 0) {
            warpSums[first >> 5][0] = s0;
            warpSums[first >> 5][1] = s1;
            warpSums[first >> 5][2] = s2;
        }
    }
    __syncthreads();
    if (threadIdx.x != 0)
        return;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int w = 0; w < kFinalThreads / 32; ++w) {
        s0 += warpSums[w][0];
        s1 += warpSums[w][1];
        s2 += warpSums[w][2];
    }
    const size_t P = size_t(W) * H;
    const float invCount = 1.0f / float(P * 3);
    const float l1 = float(s0 * invCount);
    float ssim = 0.0f, total = l1;
    if (lambda > 0.0f) {
        ssim = float(s1 * invCount);
        total = (1.0f - lambda) * l1 + lambda * (1.0f - ssim);
    }
    double mse = s2 / double(P * 3 > 0 ? P * 3 : 1);
    const float psnr = mse <= 1e-12 ? 99.0f : float(-10.0 * log10(mse));
    if (out.out3) {
        out.out3[0] = total;
        out.out3[1] = l1;
        out.out3[2] = ssim;
    }
    if (out.psnrOut)
        *out.psnrOut = psnr;
    if (DevStats *stats = out.stats) {
        const float k = stats->iteration == 0 ? 1.0f : 0.05f;
        stats->loss += k * (total - stats->loss);
        stats->psnr += k * (psnr - stats->psnr);
        stats->iteration = out.iteration;
        stats->lastLoss = total;
        stats->lastL1 = l1;
        stats->lastSsim = ssim;
        stats->lastPsnr = psnr;
    }
}

__global__ void __launch_bounds__(kFinalThreads) lossFinalizeKernel(const double *blockSums, int blocks, int W, int H,
                                                                    float lambda, LossOut out, const StepDesc *desc)
{
    pdlEntry();
    lossFinalize<kFinalThreads>(blockSums, blocks, W, H, lambda, out, desc);
}

// Block 0 finalizes the loss, which needs the forward kernel only; the others are the tiles.
__global__ void __launch_bounds__(kThreads) lossBackwardKernel(const float *render, const float *targetF,
                                                               const uint8_t *targetU8, int W, int H, float lambda,
                                                               const float *abc, float *grad, const double *blockSums,
                                                               LossOut out, const StepDesc *desc, const SsimWindow cWin)
{
    pdlEntry();
    if (blockIdx.x == 0) {
        lossFinalize<kThreads>(blockSums, gridDim.x - 1, W, H, lambda, out, desc);
        return;
    }
    if (desc)
        targetU8 = desc->target;
    constexpr int kStride = kIW + 2; // floats: rows of whole float4
    __shared__ __align__(16) float2 sAB[kIH][kIW], hAB[kIH][kTW];
    __shared__ __align__(16) float sC[kIH][kStride], hC[kIH][kTW];
    const LossTile tile = lossTile(blockIdx.x - 1, W, H);
    const int x0 = tile.x0, y0 = tile.y0, c = tile.c, tid = threadIdx.x;
    const size_t P = size_t(W) * H;
    const float l1Scale = (1.0f - lambda) * (1.0f / float(P * 3));
    const float inv255 = 1.0f / 255.0f;
    const float *mapA = abc + size_t(c) * P, *mapB = mapA + 3 * P, *mapC = mapB + 3 * P;
    forHalo(x0, y0, W, H, [&](int iy, int ix, bool in, size_t pixel) {
        sAB[iy][ix] = in ? make_float2(mapA[pixel], mapB[pixel]) : both(0.0f);
        sC[iy][ix] = in ? mapC[pixel] : 0.0f;
    });
    const int ox = tid % kTW, oy = tid / kTW * 2, gx = x0 + ox;
    // This thread's two pixels, for the chain rule.
    float x[2] = {}, y[2] = {};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int gy = y0 + oy + r;
        if (gx < W && gy < H) {
            const size_t idx = (size_t(gy) * W + gx) * 3 + c;
            x[r] = render[idx];
            y[r] = targetU8 ? float(targetU8[idx]) * inv255 : targetF[idx];
        }
    }
    __syncthreads();
    // Pass 3: horizontal blur of the partials (Loss.cpp:142-157).
    if (tid < kIH * kQuads) {
        const int iy = tid / kQuads, q = tid % kQuads * kQuad;
        float2 ab[kQuad + 2 * kR], sumAB[kQuad];
        float in[kQuad + 2 * kR + 2], sumC[kQuad];
#pragma unroll
        for (int k = 0; k < kQuad + 2 * kR; k += 2) {
            const float4 two = *reinterpret_cast<const float4 *>(&sAB[iy][q + k]);
            ab[k] = make_float2(two.x, two.y);
            ab[k + 1] = make_float2(two.z, two.w);
        }
#pragma unroll
        for (int k = 0; k < kQuad + 2 * kR + 2; k += 4)
            *reinterpret_cast<float4 *>(in + k) = *reinterpret_cast<const float4 *>(&sC[iy][q + k]);
#pragma unroll
        for (int k = 0; k < kQuad; ++k) {
            sumAB[k] = both(0.0f);
            sumC[k] = 0.0f;
#pragma unroll
            for (int t = 0; t <= 2 * kR; ++t) {
                sumAB[k] = addProduct(cWin, sumAB[k], mul2rn(both(cWin.w[t]), ab[k + t]));
                sumC[k] += cWin.w[t] * in[k + t];
            }
        }
#pragma unroll
        for (int k = 0; k < kQuad; k += 2)
            *reinterpret_cast<float4 *>(&hAB[iy][q + k]) = make_float4(sumAB[k].x, sumAB[k].y, sumAB[k + 1].x, sumAB[k + 1].y);
        *reinterpret_cast<float4 *>(&hC[iy][q]) = make_float4(sumC[0], sumC[1], sumC[2], sumC[3]);
    }
    __syncthreads();
    // Pass 4: vertical blur + chain rule (Loss.cpp:160-177), on top of the L1 term's gradient.
    float2 g[2] = {};
    float g2[2] = {};
#pragma unroll
    for (int k = 0; k < 2 + 2 * kR; ++k) {
        const float2 ab = hAB[oy + k][ox];
        const float v = hC[oy + k][ox];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = k - r;
            if (t < 0 || t > 2 * kR)
                continue;
            g[r] = addProduct(cWin, g[r], mul2rn(both(cWin.w[t]), ab));
            g2[r] += cWin.w[t] * v;
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int gy = y0 + oy + r;
        if (gx >= W || gy >= H)
            continue;
        const float d = x[r] - y[r];
        const float l1 = l1Scale * (d > 0 ? 1.0f : (d < 0 ? -1.0f : 0.0f));
        grad[(size_t(gy) * W + gx) * 3 + c] = l1 + (g[r].x + 2.0f * x[r] * g[r].y + y[r] * g2[r]);
    }
}

// Sum of squared differences in double, one partial per block, then a fixed-order final sum.
__global__ void __launch_bounds__(kThreads) sqDiffKernel(const float *a, const float *bF, const uint8_t *bU8,
                                                         size_t count, double *partial)
{
    const float inv255 = 1.0f / 255.0f;
    double s = 0.0;
    for (size_t k = size_t(blockIdx.x) * kThreads + threadIdx.x; k < count; k += size_t(gridDim.x) * kThreads) {
        const float b = bU8 ? float(bU8[k]) * inv255 : bF[k];
        const double d = double(a[k]) - double(b);
        s += d * d;
    }
    s = blockSumDouble(s);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = s;
}

__global__ void __launch_bounds__(kThreads) sumPartialsKernel(const double *partial, int n, double *out)
{
    double s = 0.0;
    for (int k = threadIdx.x; k < n; k += kThreads)
        s += partial[k];
    s = blockSumDouble(s);
    if (threadIdx.x == 0)
        *out = s;
}

__global__ void quantizeKernel(const float *rgb, size_t count, uint8_t *out)
{
    const size_t k = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= count)
        return;
    const float v = rgb[k];
    const float c = (v < 0.0f) ? 0.0f : v;            // std::max(0.0f, v)
    const float y = ((1.0f < c) ? 1.0f : c) * 255.0f; // std::min(1.0f, c) * 255.0f
    int r = int(y);                                   // y >= 0: truncation, then round half up = lround
    if (y - float(r) >= 0.5f)
        ++r;
    out[k] = uint8_t(r);
}

const SsimWindow &window()
{
    static const HostWindow w; // thread-safe one-time initialisation
    return w;
}

constexpr int kSqBlocks = 296; // 2 x 148 SMs

} // namespace

int lossBlocks(int width, int height) { return 3 * ((width + kTW - 1) / kTW) * ((height + kTH - 1) / kTH); }

void launchLoss(const float *render, const float *targetF, const uint8_t *targetU8, int width, int height, float lambda,
                float *grad, const LossScratch &ls, DevStats *stats, int iteration, const BinCounts *counts, float *out3,
                float *psnrOut, cudaStream_t s, const StepDesc *desc)
{
    const SsimWindow &win = window();
    const LossOut out{stats, iteration, counts, out3, psnrOut};
    const int blocks = lossBlocks(width, height);
    { launchPdl(lossForwardKernel, blocks, kThreads, 0, s, render, targetF, targetU8, width, height, lambda, grad, ls.abc,
                                             ls.blockSums, desc, win); countLaunch(); }
    if (lambda > 0.0f)
        { launchPdl(lossBackwardKernel, blocks + 1, kThreads, 0, s, render, targetF, targetU8, width, height, lambda, ls.abc, grad,
                                             ls.blockSums, out, desc, win); countLaunch(); }
    else
        { launchPdl(lossFinalizeKernel, 1, kFinalThreads, 0, s, ls.blockSums, blocks, width, height, lambda, out, desc); countLaunch(); }
}

void launchPsnrU8(const float *render, const uint8_t *target, size_t count, double *sumOut, cudaStream_t s)
{
    // sumOut must hold kSqBlocks + 1 doubles; the total lands in sumOut[kSqBlocks].
    { sqDiffKernel<<<kSqBlocks, kThreads, 0, s>>>(render, nullptr, target, count, sumOut); countLaunch(); }
    { sumPartialsKernel<<<1, kThreads, 0, s>>>(sumOut, kSqBlocks, sumOut + kSqBlocks); countLaunch(); }
}

void launchQuantize(const float *rgb, size_t count, uint8_t *out, cudaStream_t s)
{
    if (count)
        { quantizeKernel<<<unsigned((count + 255) / 256), 256, 0, s>>>(rgb, count, out); countLaunch(); }
}

void launchPsnrF(const float *a, const float *b, size_t count, double *sumOut, cudaStream_t s)
{
    { sqDiffKernel<<<kSqBlocks, kThreads, 0, s>>>(a, b, nullptr, count, sumOut); countLaunch(); }
    { sumPartialsKernel<<<1, kThreads, 0, s>>>(sumOut, kSqBlocks, sumOut + kSqBlocks); countLaunch(); }
}

} // namespace u3dg
