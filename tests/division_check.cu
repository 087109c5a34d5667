// Compares the quotients that the 3-D kernels form from shared or hardware reciprocals with IEEE
// division, on the device.  Built by tests/test_gpu_division.py.
#include "../cmakepro_cuda_seissim_v2_b200/csrc/seis3d_kernels.cuh"
#include "../cmakepro_cuda_seissim_v2_b200/csrc/seis3d_shade.cuh"

#include <cuda_runtime.h>

namespace {

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

__global__ void checkMeans(const float* a, const float* b, long long n, unsigned long long* wrong) {
    for (long long i = 2 * (blockIdx.x * (long long)blockDim.x + threadIdx.x); i + 1 < n; i += 2LL * gridDim.x * blockDim.x) {
        const float2 p = make_float2(a[i], a[i + 1]), q = make_float2(b[i], b[i + 1]);
        const float2 m = seis3d::harmonic2(p, q);
        const bool ok = same(m.x, __fdiv_rn(2 * p.x * q.x, p.x + q.x)) && same(m.y, __fdiv_rn(2 * p.y * q.y, p.y + q.y));
        if (!ok) atomicAdd(wrong, 1ULL);
    }
}

__global__ void checkQuotients(const float* x, const float* d, long long n, unsigned long long* wrong) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const seis3d::shade::Divisor by(d[i]);
        const float exact = __fdiv_rn(x[i], d[i]);
        // A quotient that overflows is not the plain form's case.
        if (!same(by.underWide(x[i]), exact) || (isfinite(exact) && !same(by.under(x[i]), exact)) ||
            !same(by.fraction(x[i]), fminf(fmaxf(exact, 0.0f), 1.0f)))
            atomicAdd(wrong, 1ULL);
    }
}

}  // namespace

// Device pointers; the number of operand pairs (an even one for the means) whose result differs, or -1.
extern "C" long long division_check(int means, const float* a, const float* b, long long n) {
    unsigned long long* wrong = nullptr;
    unsigned long long host = 0;
    if (cudaMallocManaged(&wrong, sizeof(*wrong)) != cudaSuccess) return -1;
    *wrong = 0;
    if (means) checkMeans<<<1184, 256>>>(a, b, n, wrong);
    else checkQuotients<<<1184, 256>>>(a, b, n, wrong);
    const cudaError_t e = cudaDeviceSynchronize();
    host = *wrong;
    cudaFree(wrong);
    return e == cudaSuccess ? (long long)host : -1;
}
