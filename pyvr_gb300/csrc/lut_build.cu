// The RGBA LUT of set_transfer_functions, built on the device from the
// transfer functions' control points (pyvr/transferfunctions/color.py:185-197,
// opacity.py:185-193, pyvr/moderngl_renderer/manager.py:162-175): entry i is
// each channel's piecewise-linear interpolation at x_i = linspace(0, 1, size)[i],
// evaluated in double and rounded once to float32, with the "clear entry"
// prefix counts of the empty-space skip computed in the same launch.
//
// The interpolation restates numpy.interp: below the first control point the
// first value, above the last (or at it) the last value, otherwise the
// segment j = the last point with xp[j] <= x; at x == xp[j] the value fp[j];
// else slope = (fp[j+1] - fp[j]) / (xp[j+1] - xp[j]) and
// slope * (x - xp[j]) + fp[j] (if that is NaN, from the right end; if still
// NaN and both ends are equal, the end value).  linspace(0, 1, n) is
// i * (1 / (n - 1)) with the last entry exactly 1.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "pvr_internal.h"

namespace pvr {
namespace {

constexpr int kMaxPoints = 256;
constexpr int kFewPoints = 32;  // most transfer functions: a 1.6 KB parameter block instead of 12 KB
constexpr int kBuildThreads = 1024;
constexpr int kMaxBuildSize = 1 << 16;

template <int POINTS> struct LutBuildParams {
    float4 *lut;
    int *prefix;
    int size;
    int n_ctf, n_otf;
    double step;  // 1 / (size - 1)
    double cx[POINTS];
    double crgb[POINTS][3];
    double ox[POINTS];
    double oa[POINTS];
};

// One transfer function in shared memory: n points, C channels and their
// segments' slopes.
template <int POINTS, int C> struct Curve {
    double x[POINTS], y[POINTS * C], slope[POINTS * C];

    __device__ __forceinline__ void load(const double *px, const double *py, int n, int first) {
        for (int k = (int)threadIdx.x - first; k < n * C; k += blockDim.x) {
            if (k < 0) continue;
            if (k < n) x[k] = px[k];
            y[k] = py[k];
            if (k < (n - 1) * C) slope[k] = (py[k + C] - py[k]) / (px[k / C + 1] - px[k / C]);
        }
    }
    // values at v, all channels
    __device__ __forceinline__ void at(double v, int n, double out[C]) const {
        int seg = -1, j = 0;  // seg: interpolate in segment j; else the value of point j
        if (n > 1 && !(v < x[0])) {
            if (v >= x[n - 1]) {
                j = n - 1;
            } else {
                int lo = 1, hi = n - 1;  // the last j with x[j] <= v
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (v >= x[mid]) lo = mid + 1;
                    else hi = mid;
                }
                j = lo - 1;
                if (x[j] != v) seg = j;
            }
        }
        const double dx = v - x[j];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const double y0 = y[j * C + c];
            out[c] = y0;
            if (seg < 0) continue;
            double r = slope[j * C + c] * dx + y0;
            if (r != r) {
                const double y1 = y[(j + 1) * C + c];
                r = slope[j * C + c] * (v - x[j + 1]) + y1;
                if (r != r && y0 == y1) r = y0;
            }
            out[c] = r;
        }
    }
};

// One block.  What bounds it: latency, and double precision (2 lanes per
// cycle and SM): a division per channel and entry took most of the 12 us of
// a 256-entry table.  The slopes are computed once per segment, from the
// points in shared memory, and an entry is one multiplication and one
// addition per channel (the same roundings); the prefix counts are ballots.
// 256 entries, 6 + 8 points: 12.1 -> 6.3 us.
template <int POINTS>
__global__ void __launch_bounds__(kBuildThreads) lut_build_kernel(const __grid_constant__ LutBuildParams<POINTS> p) {
    __shared__ Curve<POINTS, 3> s_ctf;
    __shared__ Curve<POINTS, 1> s_otf;
    __shared__ int s_count[kBuildThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    s_ctf.load(p.cx, &p.crgb[0][0], p.n_ctf, 0);
    s_otf.load(p.ox, p.oa, p.n_otf, 128);  // another warp than the first points of the colours
    __syncthreads();
    int before = 0;  // entries of earlier rounds that are not clear
    for (int i0 = 0; i0 < p.size; i0 += blockDim.x) {
        const int i = i0 + threadIdx.x;
        bool opaque = false;
        if (i < p.size) {
            const double x = (p.size > 1 && i == p.size - 1) ? 1.0 : (double)i * p.step;
            double rgb[3], a[1];
            s_ctf.at(x, p.n_ctf, rgb);
            s_otf.at(x, p.n_otf, a);
            const float4 e = make_float4(__double2float_rn(rgb[0]), __double2float_rn(rgb[1]),
                                         __double2float_rn(rgb[2]), __double2float_rn(a[0]));
            p.lut[i] = e;
            opaque = !(e.w == 0.0f && isfinite(e.x) && isfinite(e.y) && isfinite(e.z));
        }
        const unsigned set = __ballot_sync(0xffffffffu, opaque);
        if (lane == 0) s_count[warp] = __popc(set);
        __syncthreads();
        int run = before, total = 0;
        for (int w = 0; w < warps; ++w) {
            if (w < warp) run += s_count[w];
            total += s_count[w];
        }
        if (i < p.size) p.prefix[i] = run + __popc(set & ((1u << lane) - 1u));
        before += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) p.prefix[p.size] = before;
}

template <int POINTS>
cudaError_t launch_build(pvr_lut *l, const double *ctf_x, const double *ctf_rgb, int n_ctf, const double *otf_x,
                         const double *otf_a, int n_otf, int size, cudaStream_t st) {
    LutBuildParams<POINTS> p;
    p.lut = l->d_lut;
    p.prefix = l->d_prefix;
    p.size = size;
    p.n_ctf = n_ctf;
    p.n_otf = n_otf;
    p.step = size > 1 ? 1.0 / (double)(size - 1) : 0.0;
    std::memcpy(p.cx, ctf_x, sizeof(double) * n_ctf);
    std::memcpy(p.crgb, ctf_rgb, sizeof(double) * 3 * n_ctf);
    std::memcpy(p.ox, otf_x, sizeof(double) * n_otf);
    std::memcpy(p.oa, otf_a, sizeof(double) * n_otf);
    void *args[] = {&p};
    const int threads = std::min(kBuildThreads, std::max(160, (size + 31) & ~31));
    return cudaLaunchKernel((const void *)lut_build_kernel<POINTS>, dim3(1), dim3(threads), args, 0, st);
}

bool sorted_finite(const double *x, int n) {
    for (int i = 0; i < n; ++i) {
        if (!std::isfinite(x[i])) return false;
        if (i && x[i] < x[i - 1]) return false;
    }
    return true;
}

}  // namespace
}  // namespace pvr

using pvr::fail;

extern "C" int pvr_lut_build(pvr_lut *l, const double *ctf_x, const double *ctf_rgb, int n_ctf,
                             const double *otf_x, const double *otf_a, int n_otf, int size, void *stream) {
    if (!l) return fail(PVR_ERR_VALUE, "null LUT handle");
    if (!ctf_x || !ctf_rgb || !otf_x || !otf_a) return fail(PVR_ERR_VALUE, "control points are NULL");
    if (n_ctf < 1 || n_ctf > pvr::kMaxPoints || n_otf < 1 || n_otf > pvr::kMaxPoints)
        return fail(PVR_ERR_VALUE, "1..%d control points per function", pvr::kMaxPoints);
    if (size < 1 || size > pvr::kMaxBuildSize)
        return fail(PVR_ERR_VALUE, "LUT size must be in 1..%d, got %d", pvr::kMaxBuildSize, size);
    if (!pvr::sorted_finite(ctf_x, n_ctf) || !pvr::sorted_finite(otf_x, n_otf))
        return fail(PVR_ERR_VALUE, "control point positions must be finite and sorted");
    if (size > l->cap) {
        if (l->d_lut || l->d_prefix) {
            cudaDeviceSynchronize();  // a queued batch may still read the old table
            cudaFree(l->d_lut);
            cudaFree(l->d_prefix);
            l->d_lut = nullptr;
            l->d_prefix = nullptr;
            l->cap = 0;
        }  // a new table waits for nothing
        PVR_CUDA(cudaMalloc(&l->d_lut, (size_t)size * sizeof(float4)));
        PVR_CUDA(cudaMalloc(&l->d_prefix, (size_t)(size + 1) * sizeof(int)));
        l->cap = size;
    }
    PVR_CUDA(std::max(n_ctf, n_otf) <= pvr::kFewPoints
                 ? pvr::launch_build<pvr::kFewPoints>(l, ctf_x, ctf_rgb, n_ctf, otf_x, otf_a, n_otf, size,
                                                      (cudaStream_t)stream)
                 : pvr::launch_build<pvr::kMaxPoints>(l, ctf_x, ctf_rgb, n_ctf, otf_x, otf_a, n_otf, size,
                                                      (cudaStream_t)stream));
    l->size = size;
    // the table is not on the host: the march keeps the exact per-brick skip
    // test, which finds no clear range when the table has no clear entry
    l->has_clear = true;
    return PVR_OK;
}

extern "C" int pvr_lut_read(const pvr_lut *l, float *rgba_out) {
    if (!l || !rgba_out) return fail(PVR_ERR_VALUE, "NULL argument");
    PVR_CUDA(cudaDeviceSynchronize());
    PVR_CUDA(cudaMemcpy(rgba_out, l->d_lut, (size_t)l->size * sizeof(float4), cudaMemcpyDeviceToHost));
    return PVR_OK;
}
