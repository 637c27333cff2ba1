// The library's rounded quotients and roots (csrc/rounded.cuh) and CUDA's correctly rounded ones on the same
// operands, for tests/test_rounding.py. Host arrays in and out; every function returns a cudaError_t.
#include "rounded.cuh"

#include <cstddef>

namespace {

using namespace u3dg;

enum Kind { kDivisor, kQuotient, kQuotient2, kRoot, kAdam1, kAdam32 };

__global__ void compareKernel(int kind, const float *a, const float *b, size_t n, float *fused, float *exact, unsigned char *usual)
{
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        Operands ops;
        if (kind == kDivisor) {
            fused[i] = Divisor(b[i], ops).under(a[i], ops);
            exact[i] = Division(b[i], ops).under(a[i], ops);
        } else if (kind == kQuotient) {
            fused[i] = roundedQuotient(a[i], b[i]);
            exact[i] = __fdiv_rn(a[i], b[i]);
        } else if (kind == kQuotient2) {
            float2 y;
            // Both lanes, the second with the next operands.
            const size_t j = i + 1 < n ? i + 1 : i;
            const float2 q = roundedQuotient2(make_float2(a[j], a[i]), make_float2(-b[j], -b[i]), y);
            fused[i] = i & 1 ? q.y : roundedQuotient2(make_float2(a[i], a[j]), make_float2(-b[i], -b[j]), y).x;
            exact[i] = __fdiv_rn(a[i], b[i]);
        } else if (kind == kRoot) {
            fused[i] = roundedRoot(a[i]);
            exact[i] = __fsqrt_rn(a[i]);
        } else {
            const float inv = kind == kAdam1 ? 1.0f : 31.9f;
            fused[i] = roundedQuotient(a[i], __fadd_rn(__fmul_rn(roundedRoot(b[i]), inv), 1e-15f));
            exact[i] = __fdiv_rn(a[i], __fadd_rn(__fmul_rn(__fsqrt_rn(b[i]), inv), 1e-15f));
        }
        usual[i] = kind >= kAdam1 ? adamUsual(a[i], b[i]) : ops.usual();
    }
}

// Roots of all floats with bits in [first, last) that are not __fsqrt_rn's.
__global__ void rootsKernel(uint32_t first, uint32_t last, unsigned long long *wrong)
{
    unsigned long long mine = 0;
    for (uint64_t i = first + uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < last; i += uint64_t(gridDim.x) * blockDim.x) {
        const float v = __uint_as_float(uint32_t(i));
        mine += roundedRoot(v) != __fsqrt_rn(v);
    }
    if (mine)
        atomicAdd(wrong, mine);
}

template <class T>
struct Device {
    T *p = nullptr;
    explicit Device(size_t n) { error = cudaMalloc(&p, n * sizeof(T)); }
    ~Device() { cudaFree(p); }
    cudaError_t error;
};

} // namespace

extern "C" int rounding_compare(int kind, const float *a, const float *b, size_t n, float *fused, float *exact, unsigned char *usual)
{
    Device<float> da(n), db(n), df(n), de(n);
    Device<unsigned char> du(n);
    for (cudaError_t e : {da.error, db.error, df.error, de.error, du.error})
        if (e != cudaSuccess)
            return e;
    cudaMemcpy(da.p, a, n * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(db.p, b, n * sizeof(float), cudaMemcpyHostToDevice);
    compareKernel<<<1184, 256>>>(kind, da.p, db.p, n, df.p, de.p, du.p);
    cudaMemcpy(fused, df.p, n * sizeof(float), cudaMemcpyDeviceToHost);
    cudaMemcpy(exact, de.p, n * sizeof(float), cudaMemcpyDeviceToHost);
    cudaMemcpy(usual, du.p, n, cudaMemcpyDeviceToHost);
    return cudaDeviceSynchronize();
}

extern "C" int rounding_roots(unsigned first, unsigned last, unsigned long long *wrong)
{
    Device<unsigned long long> dw(1);
    if (dw.error != cudaSuccess)
        return dw.error;
    cudaMemset(dw.p, 0, sizeof(*wrong));
    rootsKernel<<<1184, 256>>>(first, last, dw.p);
    cudaMemcpy(wrong, dw.p, sizeof(*wrong), cudaMemcpyDeviceToHost);
    return cudaDeviceSynchronize();
}
