// rcp_newton of pyvr_gb300/csrc/pvr_device.cuh for every float in
// [2^-24, 2^126]: prints the largest error, in millionths of a unit in the last
// place of the exact reciprocal, and the number of arguments.
#include <cstdio>

#include "pvr_device.cuh"

__global__ void check(unsigned lo, unsigned hi, unsigned long long *c) {
    unsigned long long worst = 0, n = 0;
    for (unsigned long long i = lo + blockIdx.x * 256ull + threadIdx.x; i <= hi; i += gridDim.x * 256ull) {
        const float x = __uint_as_float((unsigned)i);
        const double y = (double)pvr::rcp_newton(x), inv = 1.0 / (double)x;
        // y x - 1 is exact: the product of two floats has 48 bits
        const double err = fabs(fma(y, (double)x, -1.0)) * inv / ldexp(1.0, ilogb(inv) - 23);
        // an error that is no number, or of an ulp and more, counts as an ulp
        const unsigned long long e = err < 1.0 ? (unsigned long long)ceil(err * 1e6) : 1000000ull;
        worst = e > worst ? e : worst;
        ++n;
    }
    atomicMax(c, worst);
    atomicAdd(c + 1, n);
}

int main() {
    unsigned long long *dc = nullptr, c[2] = {0, 0};
    if (cudaMalloc(&dc, sizeof(c)) != cudaSuccess) return 1;
    cudaMemset(dc, 0, sizeof(c));
    check<<<152 * 8, 256>>>((127u - 24u) << 23, (127u + 126u) << 23, dc);
    const cudaError_t e = cudaMemcpy(c, dc, sizeof(c), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        std::printf("error: %s\n", cudaGetErrorString(e));
        return 1;
    }
    std::printf("%llu %llu\n", c[0], c[1]);
    cudaFree(dc);
    return 0;
}
