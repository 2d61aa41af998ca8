// Exhaustive checks of the half-precision normals of pyvr_gb300/csrc/normals.cuh.
//  u8: for every gradient triple a uint8 volume can produce (767^3), component
//      0 of u8_halves, where it decides the rounding, against the component of
//      GradientArith<uint8_t> rounded to half.  Prints triples, mismatches and
//      undecided triples.
//  f16: half_root against the IEEE root for every positive finite half, and
//      half_quotient against the IEEE division for every pair of a half g and
//      a positive finite half n, all rounded to half.  Prints pairs and
//      mismatches.
#include <cstdio>
#include <vector>

#include "normals.cuh"

__global__ void check_u8(const float *g, int n, unsigned long long *c) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)n * n) return;
    const float g0 = g[t / n], g1 = g[t % n];
    unsigned long long bad = 0, open = 0;
    for (int k = 0; k < n; ++k) {
        __half2 h[3];
        if (!pvr::u8_halves(pvr::both(g0), pvr::both(g1), pvr::both(g[k]), h)) {
            ++open;
            continue;
        }
        const unsigned short want =
            __half_as_ushort(__float2half_rn(pvr::u8_component(g0, pvr::u8_norm(g0, g1, g[k]))));
        bad += __half_as_ushort(__low2half(h[0])) != want || __half_as_ushort(__high2half(h[0])) != want;
    }
    if (bad) atomicAdd(c, bad);
    if (open) atomicAdd(c + 1, open);
}

__global__ void check_f16(unsigned long long *c) {
    const unsigned n_bits = blockIdx.x + 1;  // 1 .. 0x7bff: positive, finite
    const float n = __half2float(__ushort_as_half((unsigned short)n_bits)), r = pvr::rcp_approx(n);
    unsigned long long bad = 0;
    const float root = pvr::half_root(pvr::both(n)).x;
    bad += threadIdx.x == 0 &&
           __half_as_ushort(__float2half_rn(root)) != __half_as_ushort(__float2half_rn(__fsqrt_rn(n)));
    for (unsigned b = threadIdx.x; b < 0x10000u; b += blockDim.x) {
        if ((b & 0x7c00u) == 0x7c00u) continue;  // infinities and NaN
        const float g = __half2float(__ushort_as_half((unsigned short)b));
        const unsigned short got = __half_as_ushort(__float2half_rn(pvr::half_quotient(pvr::both(g), pvr::both(n), pvr::both(r)).y));
        const unsigned short want = __half_as_ushort(__float2half_rn(__fdiv_rn(g, n)));
        bad += got != want && !((got | want) == 0x8000u);  // a zero of either sign
    }
    if (bad) atomicAdd(c + 2, bad);
}

int main() {
    std::vector<float> g;
    for (int i = -255; i <= 255; ++i) g.push_back((float)i);
    for (int i = -255; i <= 255; i += 2) g.push_back(0.5f * (float)i);  // the odd halves
    const int n = (int)g.size();
    float *dg = nullptr;
    unsigned long long *dc = nullptr, c[3] = {0, 0, 0};
    if (cudaMalloc(&dg, n * sizeof(float)) != cudaSuccess || cudaMalloc(&dc, sizeof(c)) != cudaSuccess) return 1;
    cudaMemcpy(dg, g.data(), n * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemset(dc, 0, sizeof(c));
    const long long threads = (long long)n * n;
    check_u8<<<(unsigned)((threads + 255) / 256), 256>>>(dg, n, dc);
    check_f16<<<0x7bff, 256>>>(dc);
    const cudaError_t e = cudaMemcpy(c, dc, sizeof(c), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        std::printf("error: %s\n", cudaGetErrorString(e));
        return 1;
    }
    std::printf("%lld %llu %llu %lld %llu\n", threads * n, c[0], c[1], 0x7bffLL * (0x10000 - 0x800), c[2]);
    cudaFree(dg);
    cudaFree(dc);
    return 0;
}
