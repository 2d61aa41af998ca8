// The exact arithmetic's special functions of pyvr_gb300/csrc/pvr_device.cuh,
// for every float: pvr_expf against its definition with rintf and an integer
// exponent (any NaN for a NaN), rsqrt_rn against __frsqrt_rn for every
// positive float.  Prints the mismatches of both.
#include <cstdio>

#include "pvr_device.cuh"

__device__ float exp_definition(float x) {
    if (x != x) return x;
    if (x > 88.72283f) return __int_as_float(0x7f800000);
    if (x < -87.33654f) return 0.0f;
    const float kf = rintf(x * 1.44269504f);
    float r = fmaf(kf, -0.693359375f, x);
    r = fmaf(kf, 2.12194440e-4f, r);
    float p = 1.98412698e-4f;
    p = fmaf(p, r, 1.38888889e-3f);
    p = fmaf(p, r, 8.33333333e-3f);
    p = fmaf(p, r, 4.16666667e-2f);
    p = fmaf(p, r, 1.66666667e-1f);
    p = fmaf(p, r, 0.5f);
    p = fmaf(p, r, 1.0f);
    p = fmaf(p, r, 1.0f);
    const int k = (int)kf;
    if (k <= 127) return p * __int_as_float((k + 127) << 23);
    return (p * __int_as_float((64 + 127) << 23)) * __int_as_float((k - 64 + 127) << 23);
}

__global__ void check(unsigned long long *c) {
    unsigned long long e = 0, r = 0;
    for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < (1ull << 32); i += gridDim.x * 256ull) {
        const float x = __uint_as_float((unsigned)i);
        if (x == x) e += __float_as_uint(pvr::pvr_expf(x)) != __float_as_uint(exp_definition(x));
        else e += pvr::pvr_expf(x) == pvr::pvr_expf(x);
        if (x > 0.0f) r += __float_as_uint(pvr::rsqrt_rn(x)) != __float_as_uint(__frsqrt_rn(x));
    }
    if (e) atomicAdd(c, e);
    if (r) atomicAdd(c + 1, r);
}

int main() {
    unsigned long long *dc = nullptr, c[2] = {0, 0};
    if (cudaMalloc(&dc, sizeof(c)) != cudaSuccess) return 1;
    cudaMemset(dc, 0, sizeof(c));
    check<<<152 * 8, 256>>>(dc);
    const cudaError_t e = cudaMemcpy(c, dc, sizeof(c), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        std::printf("error: %s\n", cudaGetErrorString(e));
        return 1;
    }
    std::printf("%llu %llu\n", c[0], c[1]);
    cudaFree(dc);
    return 0;
}
