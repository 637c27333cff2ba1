// warmstart.cu - learned warm-start: neighbourhood features, a small FP32 MLP (forward, backward, Adam)
// and its inference into an initial GaussianModel. No reference counterpart: the reference initialises
// with initGaussiansFromPoints (GaussianModel.cpp:68-144), which stays the fallback and the reference
// point of every comparison.
//
// Features (134 floats per SfM point):
//   [0, 48)    relative positions of the 16 nearest points, divided by the point's plain-init scale
//   [48, 64)   natural log of the 16 neighbour distances
//   [64, 112)  colours of the 16 nearest points
//   [112, 133) colour samples (minus 0.5) from the 7 nearest views that see the point in their image
//   133        number of those views / 7
// Network: 134 -> 128 -> 128 -> 128 -> 11, ReLU between layers, FP32. Parameters in one flat vector,
// per layer W (out x in, row-major) then b. All reductions run in a fixed order (deterministic).
//
// The work is tiny next to training (51.7k parameters); the kernels are plain SIMT FP32: register-tiled
// GEMMs with shared-memory staging (split over the rows for the weight gradients), brute-force k-nearest-neighbour search by warps.

#include "kernels.h"
#include "warmstart.h"

#include <algorithm>
#include <cfloat>

namespace u3dg {

namespace {

inline int cdiv(long long a, int b) { return int((a + b - 1) / b); }

// Squared distance and dot products with every product and sum rounded on its own (no FMA
// contraction), in a fixed order, so a host restatement reproduces neighbour order and view choice.
__device__ __forceinline__ float dist2(float dx, float dy, float dz)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}
__device__ __forceinline__ float dot3(const float *r, float x, float y, float z)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(r[0], x), __fmul_rn(r[1], y)), __fmul_rn(r[2], z));
}

// ------------------------------------------------------------------ k nearest neighbours

// For every query, the K nearest points (squared distance, ties by lower index). excludeSelf skips the
// point with the query's own index.
//
// A warp searches for kKnnQueries queries at once: each lane holds one candidate of the 32 at hand (read
// from shared memory once for all of the warp's queries) and computes its distance to each query, and a
// query's sorted list of the K best lies across the warp's lanes, entry k in lane k. A candidate enters
// only if it is below the list's last entry, about K ln(n / K) times per query, by one vote and one
// shuffle of the list, in index order (an equal distance stays behind the entries found before it). A
// thread per query with its list in registers, one pass of 118 CTAs over 30,000 points, spent half its
// instructions shifting lists for one lane in 32: 2.32 ms for 30,000 points and K = 16, now 1.10 ms.
constexpr int kKnnQueries = 4;
constexpr int kKnnWarps = 8;
constexpr int kKnnStage = 1024;

template <int K>
__global__ void __launch_bounds__(32 * kKnnWarps) knnKernel(const float *queries, int nq, const float *points, int np,
                                                            int excludeSelf, int *outIdx, float *outD2)
{
    static_assert(K <= 32, "a list lies across one warp");
    __shared__ float sx[kKnnStage], sy[kKnnStage], sz[kKnnStage];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q0 = (blockIdx.x * kKnnWarps + warp) * kKnnQueries;
    float qx[kKnnQueries], qy[kKnnQueries], qz[kKnnQueries];
    float bd[kKnnQueries], worst[kKnnQueries];
    int bi[kKnnQueries];
#pragma unroll
    for (int j = 0; j < kKnnQueries; ++j) {
        const bool in = q0 + j < nq;
        qx[j] = in ? queries[3 * (q0 + j)] : 0.0f;
        qy[j] = in ? queries[3 * (q0 + j) + 1] : 0.0f;
        qz[j] = in ? queries[3 * (q0 + j) + 2] : 0.0f;
        bd[j] = FLT_MAX;
        worst[j] = in ? FLT_MAX : 0.0f; // nothing enters a list without a query
        bi[j] = -1;
    }
    for (int c0 = 0; c0 < np; c0 += kKnnStage) {
        const int cnt = min(kKnnStage, np - c0);
        __syncthreads();
        for (int e = threadIdx.x; e < 3 * cnt; e += 32 * kKnnWarps) {
            const int c = e / 3, axis = e - 3 * c;
            (axis == 0 ? sx : axis == 1 ? sy : sz)[c] = points[size_t(3) * c0 + e];
        }
        __syncthreads();
        for (int g = 0; g < cnt; g += 32) {
            const int c = g + lane;
            const bool have = c < cnt;
            const float x = have ? sx[c] : 0.0f, y = have ? sy[c] : 0.0f, z = have ? sz[c] : 0.0f;
#pragma unroll
            for (int j = 0; j < kKnnQueries; ++j) {
                const float d = dist2(x - qx[j], y - qy[j], z - qz[j]);
                const bool hit = have && d < worst[j] && !(excludeSelf && c0 + c == q0 + j);
                uint32_t hits = __ballot_sync(0xffffffffu, hit);
                while (hits) {
                    const int src = __ffs(hits) - 1;
                    hits &= hits - 1;
                    const float nd = __shfl_sync(0xffffffffu, d, src);
                    if (!(nd < worst[j]))
                        continue;
                    const int at = __ffs(__ballot_sync(0xffffffffu, nd < bd[j])) - 1;
                    const float upD = __shfl_up_sync(0xffffffffu, bd[j], 1);
                    const int upI = __shfl_up_sync(0xffffffffu, bi[j], 1);
                    if (lane >= at) {
                        bd[j] = lane == at ? nd : upD;
                        bi[j] = lane == at ? c0 + g + src : upI;
                    }
                    worst[j] = __shfl_sync(0xffffffffu, bd[j], K - 1);
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kKnnQueries; ++j)
        if (q0 + j < nq && lane < K) {
            outIdx[size_t(q0 + j) * K + lane] = bi[j];
            outD2[size_t(q0 + j) * K + lane] = bd[j];
        }
}

// ------------------------------------------------------------------ features

struct ViewRef {
    u3dg_camera cam;
    const uint8_t *rgb;
    float cx, cy, cz; // camera centre
};

__global__ void __launch_bounds__(128) featuresKernel(const float *xyz, const float *rgb, int n, const int *nbr,
                                                      const float *nd2, const float *baseScale,
                                                      const ViewRef *views, int nViews, float *feat)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float *f = feat + size_t(i) * kWarmInputs;
    const float px = xyz[3 * i], py = xyz[3 * i + 1], pz = xyz[3 * i + 2];
    const float s = baseScale[i];
    const float inv = s > 0.0f ? __fdiv_rn(1.0f, s) : 0.0f;
    for (int k = 0; k < kWarmNeighbours; ++k) {
        const int j = nbr[size_t(i) * kWarmNeighbours + k];
        if (j < 0) {
            f[3 * k] = f[3 * k + 1] = f[3 * k + 2] = 0.0f;
            f[48 + k] = 0.0f;
            f[64 + 3 * k] = f[64 + 3 * k + 1] = f[64 + 3 * k + 2] = 0.0f;
            continue;
        }
        f[3 * k] = __fmul_rn(xyz[3 * j] - px, inv);
        f[3 * k + 1] = __fmul_rn(xyz[3 * j + 1] - py, inv);
        f[3 * k + 2] = __fmul_rn(xyz[3 * j + 2] - pz, inv);
        f[48 + k] = 0.5f * logf(fmaxf(nd2[size_t(i) * kWarmNeighbours + k], 1e-20f));
        for (int c = 0; c < 3; ++c)
            f[64 + 3 * k + c] = rgb ? rgb[3 * j + c] : 0.5f;
    }
    // The 7 nearest views (camera centre distance) in which the point lies in front and inside.
    float bd[kWarmViews];
    int bv[kWarmViews];
    int bu[kWarmViews], bw[kWarmViews];
    for (int k = 0; k < kWarmViews; ++k) {
        bd[k] = FLT_MAX;
        bv[k] = -1;
        bu[k] = bw[k] = 0;
    }
    for (int v = 0; v < nViews; ++v) {
        const ViewRef &vr = views[v];
        const float *R = vr.cam.R;
        const float x = __fadd_rn(dot3(R, px, py, pz), vr.cam.t[0]);
        const float y = __fadd_rn(dot3(R + 3, px, py, pz), vr.cam.t[1]);
        const float z = __fadd_rn(dot3(R + 6, px, py, pz), vr.cam.t[2]);
        if (!(z > 1e-3f))
            continue;
        const float uf = __fadd_rn(__fdiv_rn(__fmul_rn(vr.cam.fx, x), z), vr.cam.cx);
        const float wf = __fadd_rn(__fdiv_rn(__fmul_rn(vr.cam.fy, y), z), vr.cam.cy);
        // Inside the image (also rejects non-finite coordinates before the integer conversion).
        if (!(uf > -0.5f && wf > -0.5f && uf < float(vr.cam.width) - 0.5f && wf < float(vr.cam.height) - 0.5f))
            continue;
        const int u = __float2int_rn(uf);
        const int w = __float2int_rn(wf);
        if (u < 0 || w < 0 || u >= vr.cam.width || w >= vr.cam.height)
            continue;
        float d = dist2(px - vr.cx, py - vr.cy, pz - vr.cz);
        int vv = v, uu = u, ww = w;
        bool shifting = false; // insertion as in knnKernel: ties keep the lower view index first
        for (int k = 0; k < kWarmViews; ++k) {
            if (shifting || d < bd[k]) {
                shifting = true;
                const float td = bd[k];
                const int tv = bv[k], tu = bu[k], tw = bw[k];
                bd[k] = d;
                bv[k] = vv;
                bu[k] = uu;
                bw[k] = ww;
                d = td;
                vv = tv;
                uu = tu;
                ww = tw;
            }
        }
    }
    int seen = 0;
    for (int k = 0; k < kWarmViews; ++k) {
        float c3[3] = {0.0f, 0.0f, 0.0f};
        if (bv[k] >= 0) {
            const ViewRef &vr = views[bv[k]];
            const uint8_t *px8 = vr.rgb + (size_t(bw[k]) * vr.cam.width + bu[k]) * 3;
            for (int c = 0; c < 3; ++c)
                c3[c] = __fadd_rn(__fmul_rn(float(px8[c]), 1.0f / 255.0f), -0.5f);
            ++seen;
        }
        for (int c = 0; c < 3; ++c)
            f[112 + 3 * k + c] = c3[c];
    }
    f[133] = float(seen) / float(kWarmViews);
}

// ------------------------------------------------------------------ GEMM for the MLP

// Register-tiled FP32 product of one BM x BN output tile over k in [kBegin, kEnd), k ascending for every
// output: acc[r][c] = sum_k A(m, k) B(k, n). kA / kB: the operand is contiguous along k (A(m, k) =
// A[m * lda + k], B(k, n) = B[n * ldb + k]), else along its tile dimension (A[k * lda + m],
// B[k * ldb + n]); either way consecutive threads read consecutive addresses. k is staged 16 at a time
// in shared memory, the next 16 held in registers while the current ones are multiplied; each thread
// owns TM x TN outputs, in groups of four so its shared-memory reads are float4 (conflict-free: the
// threads of a warp read at most 8 distinct float4 of A and 32 consecutive ones of B).
// The layers are far too narrow (128 columns) for the tensor cores to matter next to a host upload of
// their inputs, and FP32 keeps the network's arithmetic as it was.
constexpr int kGemmK = 16;
constexpr int kGemmThreads = 256;

template <int BM, int BN, int TM, int TN, bool kA, bool kB>
__device__ __forceinline__ void gemmTile(const float *A, int lda, const float *B, int ldb, int M, int N, int kBegin,
                                         int kEnd, int m0, int n0, float (&acc)[TM][TN],
                                         float (*As)[BM + 4], float (*Bs)[BN + 4], float *colSum)
{
    static_assert((BM / TM) * (BN / TN) == kGemmThreads && TM % 4 == 0 && TN % 4 == 0, "tile shape");
    constexpr int LA = BM * kGemmK / kGemmThreads, LB = BN * kGemmK / kGemmThreads;
    const int tid = threadIdx.x, tx = tid % (BN / TN), ty = tid / (BN / TN);
    float ra[LA], rb[LB];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int e = i * kGemmThreads + tid;
            const int kk = kA ? e % kGemmK : e / BM, mm = kA ? e / kGemmK : e % BM;
            const int m = m0 + mm, k = k0 + kk;
            ra[i] = (m < M && k < kEnd) ? A[kA ? size_t(m) * lda + k : size_t(k) * lda + m] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int e = i * kGemmThreads + tid;
            const int kk = kB ? e % kGemmK : e / BN, nn = kB ? e / kGemmK : e % BN;
            const int n = n0 + nn, k = k0 + kk;
            rb[i] = (n < N && k < kEnd) ? B[kB ? size_t(n) * ldb + k : size_t(k) * ldb + n] : 0.0f;
        }
    };
#pragma unroll
    for (int r = 0; r < TM; ++r)
#pragma unroll
        for (int c = 0; c < TN; ++c)
            acc[r][c] = 0.0f;
    float column = 0.0f;
    fetch(kBegin);
    for (int k0 = kBegin; k0 < kEnd; k0 += kGemmK) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int e = i * kGemmThreads + tid;
            As[kA ? e % kGemmK : e / BM][kA ? e / kGemmK : e % BM] = ra[i];
        }
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int e = i * kGemmThreads + tid;
            Bs[kB ? e % kGemmK : e / BN][kB ? e / kGemmK : e % BN] = rb[i];
        }
        __syncthreads();
        if (k0 + kGemmK < kEnd)
            fetch(k0 + kGemmK);
        if (colSum != nullptr && tid < BM) {
#pragma unroll
            for (int kk = 0; kk < kGemmK; ++kk)
                column += As[kk][tid];
        }
#pragma unroll
        for (int kk = 0; kk < kGemmK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int r = 0; r < TM; r += 4)
                *reinterpret_cast<float4 *>(a + r) = *reinterpret_cast<const float4 *>(&As[kk][ty * TM + r]);
#pragma unroll
            for (int c = 0; c < TN; c += 4)
                *reinterpret_cast<float4 *>(b + c) = *reinterpret_cast<const float4 *>(&Bs[kk][tx * TN + c]);
#pragma unroll
            for (int r = 0; r < TM; ++r)
#pragma unroll
                for (int c = 0; c < TN; ++c)
                    acc[r][c] += a[r] * b[c];
        }
        __syncthreads();
    }
    if (colSum != nullptr && tid < BM)
        *colSum = column;
}

// C (M x N, row-major) = A B (+ bias[n]), then ReLU (relu), or zero where gate (C's shape) is not
// positive (the backward of a ReLU whose output gate is). A is contiguous along k.
template <int BM, int BN, int TM, int TN, bool kB>
__global__ void __launch_bounds__(kGemmThreads) gemmKernel(const float *A, int lda, const float *B, int ldb, float *C,
                                                           int M, int N, int K, const float *bias, int relu,
                                                           const float *gate)
{
    __shared__ __align__(16) float As[kGemmK][BM + 4];
    __shared__ __align__(16) float Bs[kGemmK][BN + 4];
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
    gemmTile<BM, BN, TM, TN, true, kB>(A, lda, B, ldb, M, N, 0, K, m0, n0, acc, As, Bs, nullptr);
    const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
#pragma unroll
    for (int r = 0; r < TM; ++r) {
        const int m = m0 + ty * TM + r;
        if (m >= M)
            continue;
#pragma unroll
        for (int c = 0; c < TN; ++c) {
            const int n = n0 + tx * TN + c;
            if (n >= N)
                continue;
            float v = acc[r][c];
            if (bias)
                v += bias[n];
            if (relu)
                v = v > 0.0f ? v : 0.0f;
            if (gate && !(gate[size_t(m) * N + n] > 0.0f))
                v = 0.0f;
            C[size_t(m) * N + n] = v;
        }
    }
}

// Weight and bias gradients of one layer, dW (out x in) = dOut^T In and db = column sums of dOut, over
// the row chunk blockIdx.z: one partial per chunk at w / b of a parameter-sized array, added up in chunk
// order by reduceGradKernel. The sum runs over every row of the batch and its result is one or a few
// tiles, so without the chunks one to six CTAs walk all rows: on 16,384 rows 3.0 ms per layer and 0.9 ms
// per column sum, against 0.02 ms per layer split.
constexpr int kGradTile = 64;

__global__ void __launch_bounds__(kGemmThreads) gradKernel(const float *dOut, const float *in, int n, int out, int inW,
                                                           int chunk, float *partial, size_t w, size_t b)
{
    __shared__ __align__(16) float As[kGemmK][kGradTile + 4];
    __shared__ __align__(16) float Bs[kGemmK][kGradTile + 4];
    const int m0 = blockIdx.y * kGradTile, n0 = blockIdx.x * kGradTile;
    const int k0 = blockIdx.z * chunk, k1 = min(n, k0 + chunk);
    float *dst = partial + size_t(blockIdx.z) * kWarmParams;
    float acc[4][4], column = 0.0f;
    gemmTile<kGradTile, kGradTile, 4, 4, false, false>(dOut, out, in, inW, out, inW, k0, k1, m0, n0, acc, As, Bs,
                                                       blockIdx.x == 0 ? &column : nullptr);
    const int tx = threadIdx.x % (kGradTile / 4), ty = threadIdx.x / (kGradTile / 4);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int m = m0 + ty * 4 + r, j = n0 + tx * 4 + c;
            if (m < out && j < inW)
                dst[w + size_t(m) * inW + j] = acc[r][c];
        }
    if (blockIdx.x == 0 && threadIdx.x < kGradTile && m0 + int(threadIdx.x) < out)
        dst[b + m0 + threadIdx.x] = column;
}

// grad[k] = sum over the chunks of partial[chunk][k], in chunk order.
__global__ void __launch_bounds__(256) reduceGradKernel(const float *partial, int chunks, float *grad)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kWarmParams)
        return;
    float s = partial[k];
#pragma unroll 8
    for (int c = 1; c < chunks; ++c)
        s += partial[size_t(c) * kWarmParams + k];
    grad[k] = s;
}

// Weighted MSE: per block partial loss, and dY = 2 w (y - t) / (n * outputs).
__global__ void __launch_bounds__(256) mseKernel(const float *y, const float *t, const float *w, int n, float *dy,
                                                 double *partial)
{
    __shared__ double sh[256];
    const size_t total = size_t(n) * kWarmOutputs;
    const float scale = 2.0f / float(total);
    double s = 0.0;
    for (size_t k = size_t(blockIdx.x) * blockDim.x + threadIdx.x; k < total; k += size_t(gridDim.x) * blockDim.x) {
        const int o = int(k % kWarmOutputs);
        const float e = y[k] - t[k];
        s += double(w[o]) * double(e) * double(e);
        dy[k] = scale * w[o] * e;
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        partial[blockIdx.x] = sh[0];
}

// One warp: strided sums per lane, then a butterfly (a fixed order).
__global__ void sumDoublesKernel(const double *p, int n, size_t count, float *out)
{
    double s = 0.0;
    for (int k = threadIdx.x; k < n; k += 32)
        s += p[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0)
        *out = float(s / double(count));
}

__global__ void adamFlatKernel(float *p, const float *g, float *m, float *v, int n, float stepSize, float invSqrtBc2,
                               float eps)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n)
        return;
    const float gk = g[k];
    const float mk = 0.9f * m[k] + 0.1f * gk;
    const float vk = 0.999f * v[k] + 0.001f * gk * gk;
    m[k] = mk;
    v[k] = vk;
    p[k] -= stepSize * mk / (sqrtf(vk) * invSqrtBc2 + eps);
}

__global__ void gatherRowsKernel(const float *src, int width, const int *rows, int n, float *dst)
{
    const size_t k = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < size_t(n) * width) {
        const size_t r = k / width, c = k % width;
        dst[k] = src[size_t(rows[r]) * width + c];
    }
}

// logit(0.05).
constexpr float kWarmOpacityFloor = -2.9444389f;

// Initial model from the plain initialisation and the network's 11 outputs: log-scales and DC colour
// as residuals over the plain values, quaternion and logit opacity directly. Non-finite outputs fall
// back to the plain values for that Gaussian.
__global__ void combineKernel(const float *pred, int n, float *scales, float *quats, float *opac, float *colors)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float *y = pred + size_t(i) * kWarmOutputs;
    bool ok = true;
    for (int k = 0; k < kWarmOutputs; ++k)
        ok = ok && isfinite(y[k]);
    if (!ok)
        return;
    for (int k = 0; k < 3; ++k) {
        scales[3 * i + k] += y[k];
        colors[3 * i + k] += y[8 + k];
    }
    for (int k = 0; k < 4; ++k)
        quats[4 * i + k] = y[3 + k];
    // Opacity floored at 0.05: the labels include Gaussians that the fixed-set runs drove transparent,
    // and an initial opacity below the pruning threshold (0.005) would remove them at the first
    // densification, leaving holes for the later steps to fill (held-out seeds reach the target sooner
    // with the floor).
    opac[i] = fmaxf(y[7], kWarmOpacityFloor);
}

} // namespace

void launchKnn(const float *queries, int nq, const float *points, int np, int k, int excludeSelf, int *idx,
               float *d2, cudaStream_t s)
{
    if (nq <= 0)
        return;
    const int grid = cdiv(nq, kKnnWarps * kKnnQueries);
    if (k == 16)
        knnKernel<16><<<grid, 32 * kKnnWarps, 0, s>>>(queries, nq, points, np, excludeSelf, idx, d2);
    else if (k == 3)
        knnKernel<3><<<grid, 32 * kKnnWarps, 0, s>>>(queries, nq, points, np, excludeSelf, idx, d2);
    else
        knnKernel<1><<<grid, 32 * kKnnWarps, 0, s>>>(queries, nq, points, np, excludeSelf, idx, d2);
    countLaunch();
}

void launchWarmFeatures(const float *xyz, const float *rgb, int n, const int *nbr, const float *nd2,
                        const float *baseScale, const void *views, int nViews, float *feat, cudaStream_t s)
{
    if (n > 0)
        { featuresKernel<<<cdiv(n, 128), 128, 0, s>>>(xyz, rgb, n, nbr, nd2, baseScale, static_cast<const ViewRef *>(views), nViews, feat); countLaunch(); }
}

size_t warmViewRefBytes() { return sizeof(ViewRef); }

void fillWarmViewRef(void *dst, const u3dg_camera &cam, const uint8_t *rgbDev)
{
    ViewRef v;
    v.cam = cam;
    v.rgb = rgbDev;
    v.cx = -(cam.R[0] * cam.t[0] + cam.R[3] * cam.t[1] + cam.R[6] * cam.t[2]);
    v.cy = -(cam.R[1] * cam.t[0] + cam.R[4] * cam.t[1] + cam.R[7] * cam.t[2]);
    v.cz = -(cam.R[2] * cam.t[0] + cam.R[5] * cam.t[1] + cam.R[8] * cam.t[2]);
    *static_cast<ViewRef *>(dst) = v;
}

namespace {

// 128 x 64 tiles with 8 x 4 outputs per thread where they fill the 148 SMs (16,384 rows by 128 columns:
// 256 tiles), 64 x 64 tiles for shorter batches; every output's sum has the same order either way.
template <bool kB>
void runGemm(const float *A, int lda, const float *B, int ldb, float *C, int M, int N, int K, const float *bias,
             bool relu, const float *gate, cudaStream_t s)
{
    if ((long long)cdiv(N, 64) * cdiv(M, 128) >= 148)
        gemmKernel<128, 64, 8, 4, kB><<<dim3(cdiv(N, 64), cdiv(M, 128)), kGemmThreads, 0, s>>>(A, lda, B, ldb, C, M, N, K, bias, relu ? 1 : 0, gate);
    else
        gemmKernel<64, 64, 4, 4, kB><<<dim3(cdiv(N, 64), cdiv(M, 64)), kGemmThreads, 0, s>>>(A, lda, B, ldb, C, M, N, K, bias, relu ? 1 : 0, gate);
    countLaunch();
}

// Rows per chunk of the weight gradients: at least 64 (four staged k tiles), and at most kGradChunks
// chunks.
int gradChunkRows(int n) { return std::max(64, cdiv(cdiv(n, kGradChunks), kGemmK) * kGemmK); }

} // namespace

void launchLayer(const float *x, int in, const float *W, const float *b, float *y, int out, int n, bool relu,
                 cudaStream_t s)
{
    if (n > 0)
        runGemm<true>(x, in, W, in, y, n, out, in, b, relu, nullptr, s);
}

void launchLayerInputGrad(const float *dOut, int out, const float *W, int in, const float *act, float *dIn, int n,
                          cudaStream_t s)
{
    if (n > 0)
        runGemm<false>(dOut, out, W, in, dIn, n, in, out, nullptr, false, act, s);
}

void launchLayerParamGrad(const float *dOut, int out, const float *act, int in, int n, float *partial, size_t w,
                          size_t b, cudaStream_t s)
{
    const int rows = gradChunkRows(n);
    { gradKernel<<<dim3(cdiv(in, kGradTile), cdiv(out, kGradTile), cdiv(n, rows)), kGemmThreads, 0, s>>>(dOut, act, n, out, in, rows, partial, w, b); countLaunch(); }
}

void launchReduceGrad(const float *partial, int n, float *grad, cudaStream_t s)
{
    { reduceGradKernel<<<cdiv(kWarmParams, 256), 256, 0, s>>>(partial, cdiv(n, gradChunkRows(n)), grad); countLaunch(); }
}

size_t gradPartialEntries(int n) { return size_t(cdiv(n, gradChunkRows(n))) * kWarmParams; }

int mseBlocks() { return 148; }

void launchMse(const float *y, const float *t, const float *w, int n, float *dy, double *partial, float *lossOut,
               cudaStream_t s)
{
    { mseKernel<<<mseBlocks(), 256, 0, s>>>(y, t, w, n, dy, partial); countLaunch(); }
    { sumDoublesKernel<<<1, 32, 0, s>>>(partial, mseBlocks(), size_t(n) * kWarmOutputs, lossOut); countLaunch(); }
}

void launchAdamFlat(float *p, const float *g, float *m, float *v, int n, float stepSize, float invSqrtBc2, float eps,
                    cudaStream_t s)
{
    if (n > 0)
        { adamFlatKernel<<<cdiv(n, 256), 256, 0, s>>>(p, g, m, v, n, stepSize, invSqrtBc2, eps); countLaunch(); }
}

void launchGatherRows(const float *src, int width, const int *rows, int n, float *dst, cudaStream_t s)
{
    if (n > 0)
        { gatherRowsKernel<<<cdiv((long long)n * width, 256), 256, 0, s>>>(src, width, rows, n, dst); countLaunch(); }
}

void launchWarmCombine(const float *pred, int n, float *scales, float *quats, float *opac, float *colors, cudaStream_t s)
{
    if (n > 0)
        { combineKernel<<<cdiv(n, 256), 256, 0, s>>>(pred, n, scales, quats, opac, colors); countLaunch(); }
}

} // namespace u3dg
