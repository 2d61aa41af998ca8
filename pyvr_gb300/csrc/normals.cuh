// Normals of the volume texels with the semantics of the reference's
// compute_normal_volume (pyvr/datasets/synthetic.py:109-122):
// g_axis = numpy.gradient along each array axis (central difference / 2
// inside, one-sided on the two faces, unit spacing), n = |g| + 1e-8 with the
// squares summed left to right, normal = g / n, cast to float32.  numpy
// evaluates this in float64 for integer input, in float16 (each operation
// rounded to half, sums accumulated in float) for float16 input, and in
// float32 for float32 input; GradientArith<T> gives the same float32 results
// for each storage type T.  axis() takes the values at i-1, i, i+1 along one
// axis (as floats, exact for every storage type; the ones outside [0, n) are
// not used), n >= 2; finish() turns the three gradients into the normal.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>
#include <string.h>

namespace pvr {

__device__ __forceinline__ float round_half(float x) { return __half2float(__float2half_rn(x)); }

template <typename T> struct GradientArith;

template <> struct GradientArith<float> {
    static __device__ __forceinline__ float axis(float vm, float v0, float vp, int i, int n) {
        if (i == 0) return __fsub_rn(vp, v0);
        if (i == n - 1) return __fsub_rn(v0, vm);
        return __fmul_rn(__fsub_rn(vp, vm), 0.5f);
    }
    static __device__ __forceinline__ float3 finish(float g0, float g1, float g2) {
        const float ss = __fadd_rn(__fadd_rn(__fmul_rn(g0, g0), __fmul_rn(g1, g1)), __fmul_rn(g2, g2));
        const float nrm = __fadd_rn(__fsqrt_rn(ss), 1e-8f);
        return make_float3(__fdiv_rn(g0, nrm), __fdiv_rn(g1, nrm), __fdiv_rn(g2, nrm));
    }
};

template <> struct GradientArith<__half> {
    static __device__ __forceinline__ float axis(float vm, float v0, float vp, int i, int n) {
        if (i == 0) return round_half(__fsub_rn(vp, v0));
        if (i == n - 1) return round_half(__fsub_rn(v0, vm));
        return round_half(__fdiv_rn(round_half(__fsub_rn(vp, vm)), 2.0f));
    }
    static __device__ __forceinline__ float3 finish(float g0, float g1, float g2) {
        // squares rounded to half; the sum accumulates in float, rounds once
        const float q0 = round_half(__fmul_rn(g0, g0));
        const float q1 = round_half(__fmul_rn(g1, g1));
        const float q2 = round_half(__fmul_rn(g2, g2));
        const float ss = round_half(__fadd_rn(__fadd_rn(q0, q1), q2));
        const float nrm = round_half(__fsqrt_rn(ss));  // + 1e-8 rounds to + 0 in half
        return make_float3(round_half(__fdiv_rn(g0, nrm)), round_half(__fdiv_rn(g1, nrm)),
                           round_half(__fdiv_rn(g2, nrm)));
    }
};

// uint8 input: numpy's float64 result, RN32(RN64(g / N)) with
// N = RN64(RN64(sqrt(S)) + 1e-8), S = g0^2 + g1^2 + g2^2, computed in float32
// arithmetic.  The gradients are exact in float32 (integers in [-255, 255]
// one-sided, multiples of 0.5 in [-127.5, 127.5] central) and so is S (a
// multiple of 0.25 below 2^18).  sqrt(S) + 1e-8 is carried as an unevaluated
// float pair Nh + Nl (Nh = RN(sqrt S), the exact remainder S - Nh^2 by FMA
// gives the low part), the quotient as qh ~ g / Nh, a product with one
// reciprocal per normal, plus a correction from the remainder g - qh*N by
// two FMAs.  The pair approximates g / N to about 2^-43 relative; when that
// interval around it does not decide the float32 rounding (the quotient lies
// within 2^-38 relative of a rounding boundary), the component is computed in
// float64 as numpy does.  Every (g0, g1, g2) a uint8 volume can produce -- the
// gradient set above cubed -- is checked against the float64 formula on the
// GPU by the tests.
struct U8Norm {
    float nh, nl;  // N ~ nh + nl
    float s;       // S
    float r;       // ~ 1 / nh (0 for S = 0)
};

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ U8Norm u8_norm(float g0, float g1, float g2) {
    U8Norm r;
    r.s = fmaf(g0, g0, fmaf(g1, g1, __fmul_rn(g2, g2)));  // exact
    const float sh = __fsqrt_rn(r.s);
    const float rem = fmaf(-sh, sh, r.s);  // exact
    r.r = sh > 0.0f ? rcp_approx(sh) : 0.0f;
    r.nh = sh;
    r.nl = fmaf(rem, 0.5f * r.r, 1e-8f);
    return r;
}

__device__ __noinline__ float u8_component_f64(float g, float s) {
    const double n = __dadd_rn(__dsqrt_rn((double)s), 1e-8);
    return __double2float_rn(__ddiv_rn((double)g, n));
}

__device__ __forceinline__ float u8_component(float g, const U8Norm &n) {
    if (g == 0.0f) return 0.0f;  // +0 / N (numpy's differences of equal values are +0)
    const float qh = __fmul_rn(g, n.r);
    const float e = fmaf(-qh, n.nh, g);   // g - qh*nh, to 2^-46 of g (qh may be an ulp off)
    const float e2 = fmaf(-qh, n.nl, e);  // g - qh*(nh + nl)
    const float corr = __fmul_rn(e2, n.r);
    const float eb = fabsf(qh) * 3.637978807091713e-12f;  // 2^-38 |q|
    const float lo = __fadd_rn(qh, __fsub_rn(corr, eb));
    const float hi = __fadd_rn(qh, __fadd_rn(corr, eb));
    if (lo == hi) return lo;
    return u8_component_f64(g, n.s);
}

__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t half_bits(__half2 h) {
    uint32_t u;
    memcpy(&u, &h, sizeof(u));
    return u;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// Pairs of normals in half precision: the lanes x and y of each argument
// belong to two texels, and the packed float instructions do both at once.

// The u8 components rounded once more to half (half records).  One
// approximate reciprocal square root decides almost every rounding:
// rsqrt.approx is within 2^-22.9 of 1 / sqrt(S), the 1e-8 in N is one FMA,
// the product adds 2^-24, so g / N lies within 2^-22 relative of q.  Where
// both ends of that interval round to the same half, the double rounding
// (RN16 of RN32 of numpy's quotient, both monotone) gives that half.  False
// where some component of the pair is not decided (about 0.3 % of the
// pairs), which then takes u8_component.
__device__ __forceinline__ bool u8_halves(float2 g0, float2 g1, float2 g2, __half2 h[3]) {
    const float2 s = __ffma2_rn(g0, g0, __ffma2_rn(g1, g1, __fmul2_rn(g2, g2)));  // exact
    // S = 0: all components are 0 whatever r is
    float2 r = make_float2(rsqrt_ftz(fmaxf(s.x, 0.25f)), rsqrt_ftz(fmaxf(s.y, 0.25f)));
    r = __ffma2_rn(__fmul2_rn(r, both(-1e-8f)), r, r);
    const float2 g[3] = {g0, g1, g2};
    bool same = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float2 q = __fmul2_rn(g[a], r);
        const float2 lo = __ffma2_rn(q, both(-2.3841858e-7f), q), hi = __ffma2_rn(q, both(2.3841858e-7f), q);
        h[a] = __floats2half2_rn(lo.x, lo.y);
        const __half2 up = __floats2half2_rn(hi.x, hi.y);
        same = same && half_bits(h[a]) == half_bits(up);
    }
    return same;
}

// float16 input: numpy's steps through one reciprocal (square root) per
// normal.  The differences, halvings and squares are rounded to half from
// exact results by the half instructions (a sum, product, quotient or root
// of halves rounded to 24 bits and then to 11 is the one rounded to 11 at
// once); the sum of squares accumulates in float32 and rounds once.  Its
// root and the quotients come from approximations and one remainder step
// each, the remainders by FMA (Markstein 1990): RN16 of them equals RN16 of
// the IEEE results for every half, and for every pair of halves (tests; zeros
// keep their sign).  False where a sum of squares is 0, infinite or NaN.
__device__ __forceinline__ float2 half_root(float2 x) {
    const float2 r = make_float2(rsqrt_ftz(x.x), rsqrt_ftz(x.y));
    const float2 s = __fmul2_rn(x, r);
    return __ffma2_rn(__ffma2_rn(__fmul2_rn(s, both(-1.0f)), s, x), __fmul2_rn(r, both(0.5f)), s);
}
// The remainder enters negated, q n - g times -r: as g - q n times r (one
// product fewer) a g of -0 gave +0, where the division gives -0.
__device__ __forceinline__ float2 half_quotient(float2 g, float2 n, float2 r) {
    const float2 q = __fmul2_rn(g, r);
    return __ffma2_rn(__ffma2_rn(q, n, __fmul2_rn(g, both(-1.0f))), __fmul2_rn(r, both(-1.0f)), q);
}
__device__ __forceinline__ float2 f16_square_sum(__half2 g0, __half2 g1, __half2 g2) {
    const float2 s = __fadd2_rn(__fadd2_rn(__half22float2(__hmul2(g0, g0)), __half22float2(__hmul2(g1, g1))),
                                __half22float2(__hmul2(g2, g2)));
    return __half22float2(__floats2half2_rn(s.x, s.y));
}
__device__ __forceinline__ bool f16_halves(__half2 g0, __half2 g1, __half2 g2, __half2 h[3]) {
    const float2 ss = f16_square_sum(g0, g1, g2);
    const float p = __fmul_rn(ss.x, ss.y);  // 2^-48 .. 2^32 for two positive finite halves
    if (!(p > 0.0f && p < 1e10f)) return false;
    const float2 root = half_root(ss);
    const float2 n = __half22float2(__floats2half2_rn(root.x, root.y));  // + 1e-8 rounds to + 0 in half
    const float2 r = make_float2(rcp_approx(n.x), rcp_approx(n.y));
    const __half2 g[3] = {g0, g1, g2};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float2 q = half_quotient(__half22float2(g[a]), n, r);
        h[a] = __floats2half2_rn(q.x, q.y);
    }
    return true;
}

template <> struct GradientArith<uint8_t> {
    static __device__ __forceinline__ float axis(float vm, float v0, float vp, int i, int n) {
        if (i == 0) return __fsub_rn(vp, v0);
        if (i == n - 1) return __fsub_rn(v0, vm);
        return __fmul_rn(__fsub_rn(vp, vm), 0.5f);  // exact
    }
    static __device__ __forceinline__ float3 finish(float g0, float g1, float g2) {
        const U8Norm n = u8_norm(g0, g1, g2);
        return make_float3(u8_component(g0, n), u8_component(g1, n), u8_component(g2, n));
    }
};

}  // namespace pvr
