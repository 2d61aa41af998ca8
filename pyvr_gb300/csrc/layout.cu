// Device layout of a loaded volume for the march kernel.
//
// The reference keeps the voxels and the normals as two 3D textures
// (pyvr/moderngl_renderer/manager.py:77-135).  Here both are re-laid out
// once per volume into texel records {stored value, nx, ny, nz}: 16-byte
// floats, or 8-byte halves for uint8 and float16 volumes (whose values are
// halves exactly; the normals are then rounded to half) -- the stored value
// keeps its value, the scale to density is applied after interpolation --
// grouped in bricks of (B+1)^3 records for bricks of B^3 texels.  The
// brick grid is shifted by one texel: brick b holds, at local index l, the
// texel clamp(b*B - 1 + l, 0, extent - 1) on each axis.  A sample with
// lower texel k = floor(u) in [-1, extent-1] uses brick (k+1)/B and local
// indices j = (k+1) % B and j+1, which hold exactly the clamp-to-edge texels
// clamp(k) and clamp(k+1) of the GL filter: the clamping is baked into the
// records, and the 8 texels of a sample sit at fixed offsets from one
// record address.  A volume without normals has quads of values in its records
// instead: {(y, z), (y + 1, z), (y, z + 1), (y + 1, z + 1)} of the texel.  Bricks are stored in Morton order of their brick
// coordinates (a warp's rays walk neighbouring bricks, which then sit in
// neighbouring memory), located through the brick array.  A per-brick
// min/max of the stored values lets the march skip bricks that the current
// LUT makes exactly transparent.
#include <algorithm>
#include <cstring>

#include "normals.cuh"
#include "pvr_device.cuh"
#include "pvr_internal.h"

namespace pvr {

namespace {

template <typename T> __device__ __forceinline__ float raw_value(const T *p, long long i);
template <> __device__ __forceinline__ float raw_value<float>(const float *p, long long i) { return p[i]; }
template <> __device__ __forceinline__ float raw_value<uint8_t>(const uint8_t *p, long long i) {
    return (float)p[i];
}
template <> __device__ __forceinline__ float raw_value<__half>(const __half *p, long long i) {
    return __half2float(p[i]);
}


template <typename Rec> __device__ __forceinline__ Rec make_record(float v, float3 n);
template <> __device__ __forceinline__ float4 make_record<float4>(float v, float3 n) {
    return make_float4(v, n.x, n.y, n.z);
}
// {value, nx, ny, nz} as halves, each rounded to nearest
template <> __device__ __forceinline__ uint2 make_record<uint2>(float v, float3 n) {
    const uint32_t h0 = __half_as_ushort(__float2half_rn(v)), h1 = __half_as_ushort(__float2half_rn(n.x));
    const uint32_t h2 = __half_as_ushort(__float2half_rn(n.y)), h3 = __half_as_ushort(__float2half_rn(n.z));
    return make_uint2(h0 | (h1 << 16), h2 | (h3 << 16));
}

// One record's slot: the rank of the brick's Morton code (x, y, z interleaved,
// x first) among the codes of the brick grid.  Walking down the octree, the
// codes before this one at a level are those of the children in front of the
// brick's own child, each a box whose part inside the grid is a product of
// three extents.  (Sorting the codes on the host took 1 ms for 33^3 bricks
// and delayed the upload; this is one thread per brick.)
__device__ __forceinline__ long long inside(int o, int h, int n) { return min(max(n - o, 0), h); }

__global__ void brick_slots_kernel(BrickGeometry g, uint4 *__restrict__ bricks) {
    const int brick = blockIdx.x * blockDim.x + threadIdx.x;
    if (brick >= g.nbricks) return;
    const int b[3] = {brick / (g.nb[2] * g.nb[1]), (brick / g.nb[2]) % g.nb[1], brick % g.nb[2]};
    int o[3] = {0, 0, 0};
    long long before = 0;
    const int top = 31 - __clz(max(max(g.nb[0], g.nb[1]), g.nb[2]));
    for (int level = top; level >= 0; --level) {
        const int h = 1 << level;
        long long lo[3], own[3], all[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = inside(o[a], h, g.nb[a]);
            const long long hi = inside(o[a] + h, h, g.nb[a]);
            const bool up = (b[a] >> level) & 1;
            own[a] = up ? hi : lo[a];
            all[a] = lo[a] + hi;
            lo[a] = up ? lo[a] : 0;  // the half in front of the own one
            if (up) o[a] += h;
        }
        before += lo[0] * all[1] * all[2] + own[0] * (lo[1] * all[2] + own[1] * lo[2]);
    }
    bricks[brick].x = (uint32_t)before;
}

// Records of one storage type, built in groups of kStep along x: float one by
// one; uint8 and float16, whose values are halves exactly, in pairs of halves.
template <typename T> struct Lanes;

template <> struct Lanes<float> {
    static constexpr int kStep = 1;
    using Word = float;
    static __device__ __forceinline__ float load(const float *p) { return __ldg(p); }
    static __device__ __forceinline__ Word word(float cur, float) { return cur; }
    // the word of two texels taken from the low lanes of two words
    static __device__ __forceinline__ Word join(Word a, Word) { return a; }
    static __device__ __forceinline__ Word diff(Word p, Word m) { return __fsub_rn(p, m); }
    static __device__ __forceinline__ Word scaled(Word d, Word s) { return __fmul_rn(d, s); }
    static __device__ __forceinline__ Word scales(float a, float) { return a; }
    static __device__ __forceinline__ void range(Word w, bool, Word &lo, Word &hi) {
        lo = fminf(lo, w);
        hi = (w != w || hi != hi) ? w + hi : fmaxf(hi, w);  // NaN sticks
    }
    static __device__ __forceinline__ Word lo_start() { return __int_as_float(0x7f800000); }
    static __device__ __forceinline__ Word hi_start() { return -__int_as_float(0x7f800000); }
    static __device__ __forceinline__ float lo_float(Word w) { return w; }
    static __device__ __forceinline__ float hi_float(Word w) { return w; }
    static __device__ __forceinline__ void records(Word v, Word g0, Word g1, Word g2, float4 *out, int, bool) {
        const float3 n = GradientArith<float>::finish(g0, g1, g2);
        *out = make_float4(v, n.x, n.y, n.z);
    }
    // a record of four stored values
    static __device__ __forceinline__ void quads(Word a, Word b, Word c, Word d, float4 *out, int, bool) {
        *out = make_float4(a, b, c, d);
    }
};

__device__ __forceinline__ __half2 halves(uint32_t u) {
    __half2 h;
    memcpy(&h, &u, sizeof(h));
    return h;
}

struct HalfLanes {
    static constexpr int kStep = 2;
    using Word = uint32_t;
    static __device__ __forceinline__ Word join(Word a, Word b) { return __byte_perm(a, b, 0x5410); }
    static __device__ __forceinline__ Word diff(Word p, Word m) { return half_bits(__hsub2(halves(p), halves(m))); }
    static __device__ __forceinline__ Word scaled(Word d, Word s) { return half_bits(__hmul2(halves(d), halves(s))); }
    static __device__ __forceinline__ Word scales(float a, float b) { return half_bits(__floats2half2_rn(a, b)); }
    static __device__ __forceinline__ void range(Word w, bool both, Word &lo, Word &hi) {
        const __half2 v = halves(both ? w : __byte_perm(w, w, 0x1010));
        lo = half_bits(__hmin2(halves(lo), v));
        hi = half_bits(__hmax2_nan(halves(hi), v));  // NaN sticks
    }
    static __device__ __forceinline__ Word lo_start() { return 0x7c007c00u; }
    static __device__ __forceinline__ Word hi_start() { return 0xfc00fc00u; }
    static __device__ __forceinline__ float lo_float(Word w) {
        const float2 f = __half22float2(halves(w));
        return fminf(f.x, f.y);
    }
    static __device__ __forceinline__ float hi_float(Word w) {
        const float2 f = __half22float2(halves(w));
        return (f.x != f.x || f.y != f.y) ? f.x + f.y : fmaxf(f.x, f.y);
    }
    // two records `stride` apart from component words {c(x), c(x + 1)}
    static __device__ __forceinline__ void quads(Word v, Word n0, Word n1, Word n2, float4 *out, int stride,
                                                 bool both) {
        const float2 f = __half22float2(halves(v)), a = __half22float2(halves(n0)), b = __half22float2(halves(n1)),
                     c = __half22float2(halves(n2));
        out[0] = make_float4(f.x, a.x, b.x, c.x);
        if (both) out[stride] = make_float4(f.y, a.y, b.y, c.y);
    }
    static __device__ __forceinline__ void quads(Word v, Word n0, Word n1, Word n2, uint2 *out, int stride, bool both) {
        out[0] = make_uint2(__byte_perm(v, n0, 0x5410), __byte_perm(n1, n2, 0x5410));
        if (both) out[stride] = make_uint2(__byte_perm(v, n0, 0x7632), __byte_perm(n1, n2, 0x7632));
    }
};

template <> struct Lanes<__half> : HalfLanes {
    static __device__ __forceinline__ uint32_t load(const __half *p) {
        return __ldg(reinterpret_cast<const unsigned short *>(p));
    }
    static __device__ __forceinline__ Word word(uint32_t cur, uint32_t next) { return cur | (next << 16); }
    static __device__ __forceinline__ void normals(Word g0, Word g1, Word g2, Word n[3]) {
        const __half2 g[3] = {halves(g0), halves(g1), halves(g2)};
        __half2 h[3];
        if (f16_halves(g[0], g[1], g[2], h)) {
#pragma unroll
            for (int a = 0; a < 3; ++a) n[a] = half_bits(h[a]);
        } else {  // a flat place (0 / 0 = NaN, g / 0 = inf, as numpy has it), or infinities
            const float2 ss = f16_square_sum(g[0], g[1], g[2]);
            const float2 len = __half22float2(__floats2half2_rn(__fsqrt_rn(ss.x), __fsqrt_rn(ss.y)));
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float2 f = __half22float2(g[a]);
                n[a] = half_bits(__floats2half2_rn(__fdiv_rn(f.x, len.x), __fdiv_rn(f.y, len.y)));
            }
        }
    }
    template <typename Rec>
    static __device__ __forceinline__ void records(Word v, Word g0, Word g1, Word g2, Rec *out, int stride, bool both) {
        Word n[3];
        normals(g0, g1, g2, n);
        quads(v, n[0], n[1], n[2], out, stride, both);
    }
};

template <> struct Lanes<uint8_t> : HalfLanes {
    static __device__ __forceinline__ uint32_t load(const uint8_t *p) { return __ldg(p); }
    // 1024 + u is the half with u in its low mantissa bits
    static __device__ __forceinline__ Word word(uint32_t cur, uint32_t next) {
        return half_bits(__hsub2(halves(cur | (next << 16) | 0x64006400u), halves(0x64006400u)));
    }
    static __device__ __forceinline__ void records(Word v, Word g0, Word g1, Word g2, uint2 *out, int stride,
                                                   bool both) {
        const float2 a = __half22float2(halves(g0)), b = __half22float2(halves(g1)), c = __half22float2(halves(g2));
        __half2 h[3];
        if (!u8_halves(a, b, c, h)) {
            const float3 p = GradientArith<uint8_t>::finish(a.x, b.x, c.x);
            const float3 q = GradientArith<uint8_t>::finish(a.y, b.y, c.y);
            h[0] = __floats2half2_rn(p.x, q.x);
            h[1] = __floats2half2_rn(p.y, q.y);
            h[2] = __floats2half2_rn(p.z, q.z);
        }
        quads(v, half_bits(h[0]), half_bits(h[1]), half_bits(h[2]), out, stride, both);
    }
    static __device__ __forceinline__ void records(Word v, Word g0, Word g1, Word g2, float4 *out, int stride,
                                                   bool both) {
        const float2 f = __half22float2(halves(v)), a = __half22float2(halves(g0)), b = __half22float2(halves(g1)),
                     c = __half22float2(halves(g2));
        const float3 p = GradientArith<uint8_t>::finish(a.x, b.x, c.x);
        out[0] = make_float4(f.x, p.x, p.y, p.z);
        if (!both) return;
        const float3 q = GradientArith<uint8_t>::finish(a.y, b.y, c.y);
        out[stride] = make_float4(f.y, q.x, q.y, q.z);
    }
};

template <int LOG2B> struct BrickShape {
    static constexpr int B = 1 << LOG2B, A = B + 1, Q = A * A, S = B + 3, P = S * S;
    // one thread per (y, z) of a slice of records; 16^3 bricks: 289 of 320
    static constexpr int kThreads = LOG2B == 4 ? 320 : LOG2B == 3 ? 128 : 64;
};

// Writes a brick's {min, max} from the threads' own (a NaN maximum marks the
// brick as never skippable).  All threads of the block call it.
template <int THREADS>
__device__ __forceinline__ void write_range(float lo, float hi, uint4 *brick) {
    __shared__ float s_lo[THREADS / 32], s_hi[THREADS / 32];
    __shared__ int s_nan[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool nan = __any_sync(0xffffffffu, hi != hi);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
        s_lo[warp] = lo;
        s_hi[warp] = hi;
        s_nan[warp] = nan;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        bool any_nan = false;
        for (int w = 0; w < THREADS / 32; ++w) {
            lo = fminf(lo, s_lo[w]);
            hi = fmaxf(hi, s_hi[w]);
            any_nan |= s_nan[w] != 0;
        }
        brick->y = any_nan ? 0x7fc00000u : __float_as_uint(lo);
        brick->z = any_nan ? 0u : __float_as_uint(hi);
        brick->w = 0u;
    }
}

// The layout of volumes without normals, and of cubic volumes (array axes =
// world axes) with device normals (numpy.gradient semantics).  One block per
// brick, bricks [brick0, brick0 + gridDim.x) in x-major order.
//
// What bounds it: the instructions per record (the earlier kernel issued on
// 90 % of cycles at 353 of them; DRAM 11 %).  So a thread owns one (y, z)
// of the brick and walks x: all its indices are set up once, the texels of a
// slice and of the next one are fixed offsets apart, and the x neighbour of
// one step is the one of the step after next.  uint8 and float16 texels are
// staged as pairs of halves {x, x + 1}, so that one packed instruction does
// two records.  NORMALS: compute them; else a record is the quad of values
// {(y, z), (y + 1, z), (y, z + 1), (y + 1, z + 1)}, so that a sample takes two
// loads instead of eight (643x361 frames of 201x150x173 float32: 42.8 / 43.7 /
// 71.2 -> 36.5 / 40.0 / 58.2 us).  Records of a slice are
// stored contiguously by neighbouring threads.  Voxel (x, y, z) along world
// axes lives at z + D*(y + H*x) of the (D,H,W) C-order buffer (the GL texture
// of size (D,H,W) read through the z/y/x swizzle, volume.frag.glsl:90).
// Measured: 512^3 in 33^3 bricks of 17^3 half records, float16 1720 -> 557 us,
// uint8 1722 -> 457 us; 256^3 in bricks of 9^3 float records, uint8 338 -> 152 us,
// float32 249 -> 121 us.  16^3 bricks: 4 blocks per SM (48 registers, with spills:
// 64 bytes for float16, 168 for float32 with normals); 3 (64 registers) and 5
// (32) are slower: 512^3 float16 557 us against 796 and 744, 200^3 float32 51
// us against 59 with 3 (without normals 43 against 46).
template <typename T, int LOG2B, typename Rec, bool NORMALS>
__global__ void __launch_bounds__(BrickShape<LOG2B>::kThreads, LOG2B == 4 ? 4 : 1)
build_walk_kernel(BrickGeometry g, const T *__restrict__ vol, int brick0, Rec *__restrict__ records,
                  uint4 *__restrict__ bricks) {
    using Sh = BrickShape<LOG2B>;
    using L = Lanes<T>;
    using Word = typename L::Word;
    constexpr int B = Sh::B, A = Sh::A, Q = Sh::Q, S = Sh::S, P = Sh::P;
    __shared__ Word sw[S * P];
    const int brick = brick0 + blockIdx.x;
    const int bz = brick % g.nb[2], by = (brick / g.nb[2]) % g.nb[1], bx = brick / (g.nb[2] * g.nb[1]);
    // staged texels: b*B - 2 + r on each axis, r in [0, S), clamped to the
    // volume; word (rx, ry, rz) holds texel rx and, in pairs, texel rx + 1
    const int ox = bx * B - 2, oy = by * B - 2, oz = bz * B - 2;
    const uint32_t slice = (uint32_t)g.ext[1] * (uint32_t)g.ext[2];
    for (int q = threadIdx.x; q < P; q += Sh::kThreads) {
        const int y = min(max(oy + q / S, 0), g.ext[1] - 1), z = min(max(oz + q % S, 0), g.ext[2] - 1);
        const T *src = vol + ((uint32_t)y * (uint32_t)g.ext[2] + (uint32_t)z);
        auto at = [&](int r) { return L::load(src + (uint32_t)min(max(ox + r, 0), g.ext[0] - 1) * (size_t)slice); };
        auto cur = at(0);
#pragma unroll
        for (int r = 0; r < S; ++r) {
            const auto next = r + 1 < S && L::kStep == 2 ? at(r + 1) : cur;
            sw[r * P + q] = L::word(cur, next);
            cur = L::kStep == 2 ? next : (r + 1 < S ? at(r + 1) : cur);
        }
    }
    __syncthreads();
    Word lo = L::lo_start(), hi = L::hi_start();
    const uint32_t slot = bricks[brick].x;
    Rec *out = records + (size_t)slot * brick_records(LOG2B) + threadIdx.x;
    if (threadIdx.x < Q) {
        const int ly = threadIdx.x / A, lz = threadIdx.x % A;
        // local indices of the volume's first and last texel: record l holds
        // texel clamp(b*B - 1 + l)
        const int fx = bx == 0 ? 1 : -9, fy = by == 0 ? 1 : -9, fz = bz == 0 ? 1 : -9;
        const int ex = g.ext[0] - bx * B, ey = g.ext[1] - by * B, ez = g.ext[2] - bz * B;
        if (fx < 0 && fy < 0 && fz < 0 && ex > B && ey > B && ez > B) {
            // every record and every neighbour lies inside the volume
            const Word *c = sw + (S + ly + 1) * S + lz + 1;
            Word xm = c[-P];
            const Word half = L::scales(0.5f, 0.5f);
#pragma unroll
            for (int l = 0; l < A; l += L::kStep, c += L::kStep * P, out += L::kStep * Q) {
                const Word v = c[0], xp = c[P];
                const bool both = l + 1 < A;
                L::range(v, both, lo, hi);
                if (NORMALS) {
                    const Word g0 = L::scaled(L::diff(xp, xm), half);
                    const Word g1 = L::scaled(L::diff(c[S], c[-S]), half);
                    const Word g2 = L::scaled(L::diff(c[1], c[-1]), half);
                    xm = L::kStep == 2 ? xp : v;
                    L::records(v, g0, g1, g2, out, Q, both);
                } else {
                    L::quads(v, c[S], c[1], c[S + 1], out, Q, both);
                }
            }
        } else {
            // a brick at the volume's faces: clamped texels, and one-sided
            // differences on them
            auto clampl = [](int l, int f, int e) { return min(max(l, f), e); };
            const int y = clampl(ly, fy, ey), z = clampl(lz, fz, ez);
            const int ym = y == fy ? y : y - 1, yp = y == ey ? y : y + 1;
            const int zm = z == fz ? z : z - 1, zp = z == ez ? z : z + 1;
            const float hy = ym == y || yp == y ? 1.0f : 0.5f, hz = zm == z || zp == z ? 1.0f : 0.5f;
            const Word sy = L::scales(hy, hy), sz = L::scales(hz, hz);
            auto at = [&](int xa, int xb, int yy, int zz) {
                const int o = (yy + 1) * S + zz + 1;
                return L::join(sw[(xa + 1) * P + o], sw[(xb + 1) * P + o]);
            };
            for (int l = 0; l < A; l += L::kStep, out += L::kStep * Q) {
                const bool both = l + 1 < A;
                const int xa = clampl(l, fx, ex), xb = clampl(min(l + 1, A - 1), fx, ex);
                const Word v = at(xa, xb, y, z);
                L::range(v, true, lo, hi);
                if (NORMALS) {
                    const bool fa = xa == fx || xa == ex, fb = xb == fx || xb == ex;
                    const Word g0 = L::scaled(L::diff(at(xa == ex ? xa : xa + 1, xb == ex ? xb : xb + 1, y, z),
                                                      at(xa == fx ? xa : xa - 1, xb == fx ? xb : xb - 1, y, z)),
                                              L::scales(fa ? 1.0f : 0.5f, fb ? 1.0f : 0.5f));
                    const Word g1 = L::scaled(L::diff(at(xa, xb, yp, z), at(xa, xb, ym, z)), sy);
                    const Word g2 = L::scaled(L::diff(at(xa, xb, y, zp), at(xa, xb, y, zm)), sz);
                    L::records(v, g0, g1, g2, out, Q, both);
                } else {
                    const int y1 = clampl(ly + 1, fy, ey), z1 = clampl(lz + 1, fz, ez);
                    L::quads(v, at(xa, xb, y1, z), at(xa, xb, y, z1), at(xa, xb, y1, z1), out, Q, both);
                }
            }
        }
    }
    write_range<Sh::kThreads>(L::lo_float(lo), L::hi_float(hi), bricks + brick);
}

constexpr int kLayoutThreads = 256;

// n / d for n < 2^31 by one multiplication (Granlund & Montgomery 1994).
struct FastDiv {
    uint32_t d, m, s;
    explicit FastDiv(uint32_t div) : d(div), s(0) {
        while ((1ull << s) < d) ++s;
        m = (uint32_t)(((1ull << 32) * ((1ull << s) - d)) / d + 1);
    }
    __device__ __forceinline__ uint32_t quot(uint32_t n) const { return (__umulhi(n, m) + n) >> s; }
};

// The layout of the other volumes: given normals (read from `nrm`, indexed
// like the voxels: manager.py:123-125), and device normals of non-cubic
// volumes, whose array axes are not the world axes (the neighbours come from
// global memory).  One block per brick; a thread per record.
template <typename T, int LOG2B, typename Rec>
__global__ void __launch_bounds__(kLayoutThreads)
build_bricks_kernel(BrickGeometry g, const T *__restrict__ vol, int D, int H, int W, FastDiv by_w, FastDiv by_h,
                    const float *__restrict__ nrm, Rec *__restrict__ records, uint4 *__restrict__ bricks) {
    constexpr int B = 1 << LOG2B, A = B + 1, R = A * A * A;
    const int brick = blockIdx.x;
    const int bz = brick % g.nb[2], by = (brick / g.nb[2]) % g.nb[1], bx = brick / (g.nb[2] * g.nb[1]);
    const uint32_t slot = bricks[brick].x;
    float lo = __int_as_float(0x7f800000), hi = -lo;
    bool nan = false;
    for (int rec = threadIdx.x; rec < R; rec += kLayoutThreads) {
        const int lz = rec % A, ly = (rec / A) % A, lx = rec / (A * A);
        // record l of the brick holds texel clamp(b*B - 1 + l)
        const int x = min(max(bx * B - 1 + lx, 0), g.ext[0] - 1);
        const int y = min(max(by * B - 1 + ly, 0), g.ext[1] - 1);
        const int z = min(max(bz * B - 1 + lz, 0), g.ext[2] - 1);
        const uint32_t src = (uint32_t)z + (uint32_t)g.ext[2] * ((uint32_t)y + (uint32_t)g.ext[1] * (uint32_t)x);
        const float val = raw_value<T>(vol, src);
        nan |= val != val;
        lo = fminf(lo, val);
        hi = fmaxf(hi, val);
        float3 n;
        if (nrm) {
            n = make_float3(nrm[3 * (size_t)src + 0], nrm[3 * (size_t)src + 1], nrm[3 * (size_t)src + 2]);
        } else {
            // array position (a, b, c) of flat element src in the (D,H,W) array
            const uint32_t ab = by_w.quot(src), a = by_h.quot(ab);
            const int c = (int)(src - ab * by_w.d), b = (int)(ab - a * by_h.d);
            const uint32_t sa = (uint32_t)H * (uint32_t)W;
            const float am = (int)a > 0 ? raw_value<T>(vol, src - sa) : 0.0f;
            const float ap = (int)a < D - 1 ? raw_value<T>(vol, src + sa) : 0.0f;
            const float bm = b > 0 ? raw_value<T>(vol, src - W) : 0.0f, bp = b < H - 1 ? raw_value<T>(vol, src + W) : 0.0f;
            const float cm = c > 0 ? raw_value<T>(vol, src - 1) : 0.0f, cp = c < W - 1 ? raw_value<T>(vol, src + 1) : 0.0f;
            n = GradientArith<T>::finish(GradientArith<T>::axis(am, val, ap, (int)a, D),
                                         GradientArith<T>::axis(bm, val, bp, b, H),
                                         GradientArith<T>::axis(cm, val, cp, c, W));
        }
        records[(size_t)slot * R + rec] = make_record<Rec>(val, n);
    }
    write_range<kLayoutThreads>(lo, nan ? __int_as_float(0x7fc00000) : hi, bricks + brick);
}

// A float survives float -> half -> float bit for bit (NaN: as some NaN).
__device__ __forceinline__ bool half_exact(float x, unsigned short &h) {
    const __half hv = __float2half_rn(x);
    h = __half_as_ushort(hv);
    const float back = __half2float(hv);
    if (x != x) return back != back;
    return __float_as_uint(back) == __float_as_uint(x);
}

// Compact records: {value, nx, ny, nz} as four halves in one 8-byte record,
// each rounded to nearest.  The march decodes them exactly, so a volume
// whose records all survive the round trip renders the same images from
// either form.  *inexact gets bit 0 if some value does not survive it, bit 1
// if some normal component does not.
__global__ void compact_records_kernel(const float4 *__restrict__ in, uint2 *__restrict__ out, long long n,
                                       int *__restrict__ inexact) {
    unsigned bad = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float4 r = in[i];
        unsigned short h0, h1, h2, h3;
        const bool v_ok = half_exact(r.x, h0);
        const bool x_ok = half_exact(r.y, h1);
        const bool y_ok = half_exact(r.z, h2);
        const bool z_ok = half_exact(r.w, h3);
        bad |= (v_ok ? 0u : 1u) | ((x_ok && y_ok && z_ok) ? 0u : 2u);
        out[i] = make_uint2((uint32_t)h0 | ((uint32_t)h1 << 16), (uint32_t)h2 | ((uint32_t)h3 << 16));
    }
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (bad && (threadIdx.x & 31) == 0) atomicOr(inexact, (int)bad);
}

__device__ __forceinline__ float4 record_at(const float4 *r, size_t i) { return r[i]; }
__device__ __forceinline__ float4 record_at(const uint2 *r, size_t i) {
    const uint2 q = r[i];
    return make_float4(__half2float(__ushort_as_half((unsigned short)(q.x & 0xffffu))),
                       __half2float(__ushort_as_half((unsigned short)(q.x >> 16))),
                       __half2float(__ushort_as_half((unsigned short)(q.y & 0xffffu))),
                       __half2float(__ushort_as_half((unsigned short)(q.y >> 16))));
}

// Scatter the normals held in the records back to (D,H,W,3): one thread per
// texel, reading the record of local index (k+1) % B in brick (k+1) / B.
template <int LOG2B, typename Rec>
__global__ void read_normals_kernel(BrickGeometry g, int D, int H, int W,
                                    const uint4 *__restrict__ bricks,
                                    const Rec *__restrict__ records, float *__restrict__ out) {
    constexpr int B = 1 << LOG2B, A = B + 1, R = A * A * A;
    const long long total = (long long)D * H * W;
    for (long long src = blockIdx.x * (long long)blockDim.x + threadIdx.x; src < total;
         src += (long long)gridDim.x * blockDim.x) {
        // flat texel index src = z + D*(y + H*x) (world axes)
        const int z = (int)(src % D);
        const int y = (int)((src / D) % H);
        const int x = (int)(src / ((long long)D * H));
        const int kx = x + 1, ky = y + 1, kz = z + 1;
        const int id = ((kx >> LOG2B) * g.nb[1] + (ky >> LOG2B)) * g.nb[2] + (kz >> LOG2B);
        const int rec = ((kx & (B - 1)) * A + (ky & (B - 1))) * A + (kz & (B - 1));
        const float4 v = record_at(records, (size_t)bricks[id].x * R + rec);
        out[3 * src + 0] = v.y;
        out[3 * src + 1] = v.z;
        out[3 * src + 2] = v.w;
    }
}

template <typename T, int LOG2B, typename Rec>
cudaError_t build_typed(const BrickGeometry &g, const void *vol, const int dims[3], const float *nrm,
                        int normals_mode, int brick0, int nbricks, Rec *records, uint4 *bricks, cudaStream_t st) {
    // one block per brick: short blocks, so that render kernels on streams
    // of higher priority get SMs as soon as any layout block retires
    const bool cubic = dims[0] == dims[1] && dims[1] == dims[2];
    constexpr int threads = BrickShape<LOG2B>::kThreads;
    const T *v = (const T *)vol;
    if (normals_mode == PVR_NORMALS_NONE)
        build_walk_kernel<T, LOG2B, Rec, false><<<nbricks, threads, 0, st>>>(g, v, brick0, records, bricks);
    else if (normals_mode == PVR_NORMALS_DEVICE && cubic)
        build_walk_kernel<T, LOG2B, Rec, true><<<nbricks, threads, 0, st>>>(g, v, brick0, records, bricks);
    else
        build_bricks_kernel<T, LOG2B, Rec><<<nbricks, kLayoutThreads, 0, st>>>(
            g, v, dims[0], dims[1], dims[2], FastDiv(dims[2]), FastDiv(dims[1]),
            normals_mode == PVR_NORMALS_GIVEN ? nrm : nullptr, records, bricks);
    return cudaGetLastError();
}

template <int LOG2B>
cudaError_t build_log2(const BrickGeometry &g, int dtype, const void *vol, const int dims[3],
                       const float *nrm, int normals_mode, int brick0, int nbricks, void *records, bool half,
                       uint4 *bricks, cudaStream_t st) {
    if (dtype == PVR_F32)  // float32 values are not halves: float records only
        return build_typed<float, LOG2B, float4>(g, vol, dims, nrm, normals_mode, brick0, nbricks, (float4 *)records,
                                                 bricks, st);
    if (dtype == PVR_U8)
        return half ? build_typed<uint8_t, LOG2B, uint2>(g, vol, dims, nrm, normals_mode, brick0, nbricks,
                                                         (uint2 *)records, bricks, st)
                    : build_typed<uint8_t, LOG2B, float4>(g, vol, dims, nrm, normals_mode, brick0, nbricks,
                                                          (float4 *)records, bricks, st);
    return half ? build_typed<__half, LOG2B, uint2>(g, vol, dims, nrm, normals_mode, brick0, nbricks,
                                                    (uint2 *)records, bricks, st)
                : build_typed<__half, LOG2B, float4>(g, vol, dims, nrm, normals_mode, brick0, nbricks,
                                                     (float4 *)records, bricks, st);
}

}  // namespace

BrickGeometry make_brick_geometry(const int dims_dhw[3], int log2b) {
    BrickGeometry g;
    g.log2b = log2b;
    g.ext[0] = dims_dhw[2];  // world x <-> W
    g.ext[1] = dims_dhw[1];  // world y <-> H
    g.ext[2] = dims_dhw[0];  // world z <-> D
    // k + 1 ranges over [0, extent]
    for (int a = 0; a < 3; ++a) g.nb[a] = (g.ext[a] >> log2b) + 1;
    g.nbricks = g.nb[0] * g.nb[1] * g.nb[2];
    return g;
}

cudaError_t launch_brick_slots(const BrickGeometry &g, uint4 *bricks, cudaStream_t st) {
    brick_slots_kernel<<<(g.nbricks + 127) / 128, 128, 0, st>>>(g, bricks);
    return cudaGetLastError();
}

cudaError_t launch_build_records(const BrickGeometry &g, int dtype, const void *vol, const int dims[3],
                                 const float *nrm, int normals_mode, int brick0, int nbricks, void *records, bool half,
                                 uint4 *bricks, cudaStream_t st) {
    if (half && dtype == PVR_F32) return cudaErrorInvalidValue;
    if (nbricks <= 0) return cudaSuccess;
    switch (g.log2b) {
    case 2:
        return build_log2<2>(g, dtype, vol, dims, nrm, normals_mode, brick0, nbricks, records, half, bricks, st);
    case 4:
        return build_log2<4>(g, dtype, vol, dims, nrm, normals_mode, brick0, nbricks, records, half, bricks, st);
    default:
        return build_log2<3>(g, dtype, vol, dims, nrm, normals_mode, brick0, nbricks, records, half, bricks, st);
    }
}

template <typename Rec>
void read_normals_typed(const BrickGeometry &g, const int dims[3], const uint4 *bricks, const Rec *records,
                        float *out, int blocks, cudaStream_t st) {
    switch (g.log2b) {
    case 2: read_normals_kernel<2><<<blocks, 256, 0, st>>>(g, dims[0], dims[1], dims[2], bricks, records, out); break;
    case 4: read_normals_kernel<4><<<blocks, 256, 0, st>>>(g, dims[0], dims[1], dims[2], bricks, records, out); break;
    default: read_normals_kernel<3><<<blocks, 256, 0, st>>>(g, dims[0], dims[1], dims[2], bricks, records, out);
    }
}

cudaError_t launch_read_normals(const BrickGeometry &g, const int dims[3], const uint4 *bricks,
                                const void *records, bool compact, float *out, cudaStream_t st) {
    const long long total = (long long)dims[0] * dims[1] * dims[2];
    int blocks = (int)std::min<long long>((total + 255) / 256, 152LL * 64);
    if (compact) read_normals_typed(g, dims, bricks, (const uint2 *)records, out, blocks, st);
    else read_normals_typed(g, dims, bricks, (const float4 *)records, out, blocks, st);
    return cudaGetLastError();
}

cudaError_t launch_compact_records(const float4 *records, uint2 *out, long long n, int *inexact,
                                   cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int blocks = (int)std::min<long long>((n + 255) / 256, 152LL * 16);
    compact_records_kernel<<<blocks, 256, 0, st>>>(records, out, n, inexact);
    return cudaGetLastError();
}

}  // namespace pvr
