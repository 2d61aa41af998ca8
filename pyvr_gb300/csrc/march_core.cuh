// The ray-march kernels: pyvr/shaders/volume.frag.glsl:main as CUDA, run as
// a persistent kernel over a batch of renders, as a kernel of one render (one
// block per tile), and as one of a small render with several lanes per ray.
//
// A batch's work is a queue of pixel tiles over every job (one job = one
// render with its own volume, LUT, camera, light, config and size).  The job
// table is the kernel's parameter block, so frame constants are read through
// the constant cache as in a single-render kernel.  Each 256-thread block
// pops a tile with one atomic, stages the tile's RGBA LUT (plus the LUT's
// "clear entry" prefix counts) in shared memory when the job changes, then
// marches one ray per thread; the other kernels stage it once per block, of
// 256 threads or (single renders of half records) 128.  Warps cover 8x4-pixel
// sub-tiles so the rays of a warp are spatially close and their trilinear
// footprints share cache lines.  Voxels and normals are read from the bricked
// texel records of layout.cu: each sample is 8 vector loads (without normals
// 2) at fixed offsets from one record address.  Paired channels go through the packed FP32x2 pipe,
// which rounds each lane exactly like the scalar instruction; an add that
// consumes a packed product is always a scalar __fadd_rn, so no
// product/add pair can be fused into one rounding.
//
// The march reproduces the reference loop (frag:87-119) exactly, with two
// shortcuts that change no output bit:
//  - the ray's texture coordinate is monotone in the step index along each
//    axis (the position advances by repeated addition of one float step),
//    so the steps whose coordinate is valid (frag:92) form one contiguous
//    run; once the ray has left it, or provably cannot enter it, every
//    remaining iteration would be a no-op and the loop ends;
//  - a sample in a brick whose value range maps only to LUT entries with
//    alpha exactly 0 (and a finite colour) adds exactly +0 to every
//    accumulator, so its fetches and shading are skipped; the position
//    still advances by the same float additions.  The LUT entry range is
//    exact: a lerp fmaf(t, b-a, a) with t in [0,1) stays within [a, b], so
//    a sample lies in the brick's value range, and the scale and the LUT
//    coordinate are monotone float operations evaluated as for a sample.
//
// A volume's records are 16-byte floats, or 8-byte halves (layout.cu); the
// half form decodes to floats, so the arithmetic is the same either way.
//
// Two arithmetics (pvr_set_arithmetic), chosen per launch:
//  - exact: every operation rounded as the CPU oracle rounds it (no FMA
//    contraction except the texture lerps, exp by pvr_expf, a correctly
//    rounded rsqrt), so a frame equals the oracle's bit for bit;
//  - fast (the default): the position recurrence, the validity test, the
//    texture addressing, the lerps and the LUT addressing are the exact
//    arithmetic's, so the same samples are taken from the same texels; the
//    shading tail fuses products into FMAs, takes exp(-x) as one hardware
//    ex2 of x*log2(e) and 1/|n| as one hardware rsqrt (relative errors
//    about 2^-22), and dots n with the light before scaling by 1/|n|.  The
//    images stay within 1 LSB per RGBA8 channel of the exact ones (tested
//    at the configurations' full sizes).
#pragma once

#include "pvr_device.cuh"
#include "pvr_internal.h"

namespace pvr {

__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// {value, nx, ny, nz}; without normals a quad of values (layout.cu)
template <bool COMPACT> struct RecordOf { using T = float4; };
template <> struct RecordOf<true> { using T = uint2; };

// two halves (low, high) of a 32-bit word as floats, in one conversion
__device__ __forceinline__ float2 half_pair(uint32_t b) {
    __half2 h;
    memcpy(&h, &b, sizeof(h));
    return __half22float2(h);
}

// How the lerps of a sample's records are written: the same two roundings per
// lerp and lane in each.  Packed: two lanes per instruction.  Mixed: the first
// lerp's difference b - a takes b as a half (one instruction of a half and a
// float), so that only a is converted.  MixedScalar: the same, one lane per
// instruction, which needs no register pairs.  Half records in the single
// kernel (us, three 512^2 orbit frames of 16^3 bricks / 1024^2 of 512^3):
// scalar without the mixed difference at 40 registers 74 / 128 / 142 / 676,
// MixedScalar at 40 (it spills) 77 / 139 / 156 / 686, at 48 79 / 119 / 130 /
// 636, packed Mixed at 48 (spills) 82 / 130 / 135 / 655.  The split kernel at
// 48: packed (spills) 123 / 291, MixedScalar 113 / 286 (192^2, 256^2 of 512^3).
// The batch kernels at 48, two comparisons on two GPUs: packed 1498, Mixed
// 1441; and Mixed 1390, MixedScalar 1440.
enum LerpForm { kLerpPacked = 0, kLerpMixed = 1, kLerpMixedScalar = 2 };

template <int LERP>
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float t) {
    if (LERP == kLerpMixedScalar) return make_float2(lerp_tex(a.x, b.x, t), lerp_tex(a.y, b.y, t));
    return lerp_tex2(a, b, t);
}
template <int LERP>
__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float t) {
    const float2 x = lerp2<LERP>(lo2(a), lo2(b), t), y = lerp2<LERP>(hi2(a), hi2(b), t);
    return make_float4(x.x, x.y, y.x, y.y);
}
// half h (the low 16 bits) - c, rounded once
__device__ __forceinline__ float sub_half(uint32_t h, float c) {
    float d;
    asm("sub.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"((unsigned short)h), "f"(c));
    return d;
}
// {value, nx, ny, nz} between two records
template <int LERP>
__device__ __forceinline__ float4 lerp_rec(float4 a, float4 b, float t) { return lerp4<LERP>(a, b, t); }
template <int LERP>
__device__ __forceinline__ float4 lerp_rec(uint2 a, uint2 b, float t) {
    const float2 a0 = half_pair(a.x), a1 = half_pair(a.y);
    if (LERP != kLerpPacked) {
        const float2 d0 = make_float2(sub_half(b.x, a0.x), sub_half(b.x >> 16, a0.y));
        const float2 d1 = make_float2(sub_half(b.y, a1.x), sub_half(b.y >> 16, a1.y));
        if (LERP == kLerpMixedScalar)
            return make_float4(fmaf(t, d0.x, a0.x), fmaf(t, d0.y, a0.y), fmaf(t, d1.x, a1.x), fmaf(t, d1.y, a1.y));
        const float2 x = __ffma2_rn(dup2(t), d0, a0), y = __ffma2_rn(dup2(t), d1, a1);
        return make_float4(x.x, x.y, y.x, y.y);
    }
    const float2 b0 = half_pair(b.x), b1 = half_pair(b.y);
    return lerp4<LERP>(make_float4(a0.x, a0.y, a1.x, a1.y), make_float4(b0.x, b0.y, b1.x, b1.y), t);
}
// A record without normals is the quad of values {(y, z), (y + 1, z),
// (y, z + 1), (y + 1, z + 1)}: its lerp along z, lanes y and y + 1.
template <int LERP>
__device__ __forceinline__ float2 lerp_quad(float4 q, float t) { return lerp2<LERP>(lo2(q), hi2(q), t); }
template <int LERP>
__device__ __forceinline__ float2 lerp_quad(uint2 q, float t) {
    const float2 a = half_pair(q.x);
    if (LERP == kLerpMixed)
        return __ffma2_rn(dup2(t), make_float2(sub_half(q.y, a.x), sub_half(q.y >> 16, a.y)), a);
    return lerp2<LERP>(a, half_pair(q.y), t);
}

template <bool SMEM>
__device__ __forceinline__ int prefix_entry(const int *p, int i) {
    if (SMEM) return p[i];
    return __ldg(p + i);
}

// LUT entry index of density d: floor(d*size - 0.5) clamped to the table,
// as texture(transfer_function_lut, vec2(d, 0.5)) addresses it (frag:96).
// fl = floor(coordinate); NaN and negative coordinates give entry 0.
__device__ __forceinline__ int lut_index(float fl, float lmax) {
    return (int)fminf(fmaxf(fl, 0.0f), lmax);
}

// What one sample adds before its transmittance: (r, g) and (b, alpha).
struct Source {
    float2 rg, ba;
};

// Front-to-back compositing (frag:112-115):
// acc.c += (1 - acc.a) * (c * light * alpha), acc.a += (1 - acc.a) * alpha
template <bool FAST>
__device__ __forceinline__ void composite(const Source &s, float2 &acc_rg, float2 &acc_ba) {
    const float2 tr = dup2(__fadd_rn(1.0f, -acc_ba.y));
    if (FAST) {
        acc_rg = __ffma2_rn(tr, s.rg, acc_rg);
        acc_ba = __ffma2_rn(tr, s.ba, acc_ba);
        return;
    }
    const float2 add_rg = __fmul2_rn(tr, s.rg);
    const float2 add_ba = __fmul2_rn(tr, s.ba);
    acc_rg = make_float2(__fadd_rn(acc_rg.x, add_rg.x), __fadd_rn(acc_rg.y, add_rg.y));
    acc_ba = make_float2(__fadd_rn(acc_ba.x, add_ba.x), __fadd_rn(acc_ba.y, add_ba.y));
}

// Shading of one in-box sample (frag:93-110).  p: the record of the
// footprint's lower corner; fx, fy, fz: the filter fractions.
template <int LOG2B, bool NORMALS, bool SMEM_LUT, bool FAST, int LERP, typename Rec>
__device__ __forceinline__ Source shade_sample(const MarchFrame &f, const Rec *__restrict__ p,
                                               float fx, float fy, float fz, const float4 *lut) {
    constexpr int ROW = brick_apron(LOG2B), SLICE = ROW * ROW;
    float density;
    float n[3];
    if (NORMALS) {
        const Rec r000 = __ldg(p);
        const Rec r001 = __ldg(p + 1);
        const Rec r010 = __ldg(p + ROW);
        const Rec r011 = __ldg(p + ROW + 1);
        const Rec r100 = __ldg(p + SLICE);
        const Rec r101 = __ldg(p + SLICE + 1);
        const Rec r110 = __ldg(p + SLICE + ROW);
        const Rec r111 = __ldg(p + SLICE + ROW + 1);
        // texture(volume_texture, tex.zyx) and texture(normal_volume, ...):
        // lerp along z, then y, then x; lanes (value, nx) and (ny, nz)
        const float4 v = lerp4<LERP>(lerp4<LERP>(lerp_rec<LERP>(r000, r001, fz), lerp_rec<LERP>(r010, r011, fz), fy),
                                     lerp4<LERP>(lerp_rec<LERP>(r100, r101, fz), lerp_rec<LERP>(r110, r111, fz), fy),
                                     fx);
        density = __fmul_rn(v.x, f.value_scale);
        n[0] = v.y;
        n[1] = v.z;
        n[2] = v.w;
    } else {
        const Rec q0 = __ldg(p), q1 = __ldg(p + SLICE);
        const float2 zz0 = lerp_quad<LERP>(q0, fz), zz1 = lerp_quad<LERP>(q1, fz);
        const float2 yy = lerp2<LERP>(make_float2(zz0.x, zz1.x), make_float2(zz0.y, zz1.y), fy);
        density = __fmul_rn(lerp_tex(yy.x, yy.y, fx), f.value_scale);
        // the reference's unbound normal sampler reads the R32F volume
        // texture: normal = (density, 0, 0)
        n[0] = density;
        n[1] = 0.0f;
        n[2] = 0.0f;
    }

    // texture(transfer_function_lut, vec2(density, 0.5)) (frag:96): entries
    // floor(lu) and floor(lu) + 1, each clamped to the table, and the lerp
    // weight lu - floor(lu)
    const float lu = FAST ? fmaf(density, f.flut_size, -0.5f) : __fadd_rn(__fmul_rn(density, f.flut_size), -0.5f);
    const float lfl = floorf(lu);
    const float la = __fadd_rn(lu, -lfl);
    float4 A, B;
    if (SMEM_LUT) {
        // the staged table has an apron entry at either end (stage_lut), so one
        // clamped index addresses both entries: -1 and 0 below the table (or
        // for NaN), size - 1 and size above it
        const float4 *e = lut + (int)fminf(fmaxf(lfl, -1.0f), f.flut_max);
        A = e[0];
        B = e[1];
    } else {
        A = __ldg(lut + lut_index(lfl, f.flut_max));
        B = __ldg(lut + lut_index(__fadd_rn(lfl, 1.0f), f.flut_max));
    }
    const float2 crg = lerp2<LERP>(lo2(A), lo2(B), la);
    const float2 cba = lerp2<LERP>(hi2(A), hi2(B), la);  // (blue, alpha_tf)

    if (FAST) {
        // alpha = 1 - exp(-alpha_tf * step/ref) (frag:101)
        const float alpha = __fadd_rn(1.0f, -ex2_approx(-__fmul_rn(cba.y, f.alpha_k2)));
        // Lambert term (frag:107-110): dot(n, L) / |n|; a zero (or NaN)
        // normal gives 0
        const float n2 = fmaf(n[0], n[0], fmaf(n[1], n[1], __fmul_rn(n[2], n[2])));
        const float dl = fmaf(n[0], f.light_dir[0], fmaf(n[1], f.light_dir[1], __fmul_rn(n[2], f.light_dir[2])));
        const float di = n2 > 0.0f ? fmaxf(__fmul_rn(dl, rsqrt_approx(n2)), 0.0f) : 0.0f;
        const float la_ = __fmul_rn(fmaf(f.diffuse, di, f.ambient), alpha);
        return {__fmul2_rn(crg, dup2(la_)), make_float2(__fmul_rn(cba.x, la_), alpha)};
    }

    // Beer-Lambert opacity correction (frag:101)
    const float alpha = __fadd_rn(1.0f, -pvr_expf(-__fmul_rn(cba.y, f.alpha_k)));

    // Lambert term (frag:107-110); a zero (or NaN) normal gives 0
    const float n2 = __fadd_rn(__fadd_rn(__fmul_rn(n[0], n[0]), __fmul_rn(n[1], n[1])), __fmul_rn(n[2], n[2]));
    float di = 0.0f;
    if (n2 > 0.0f) {
        // normalize(n) = n * rsqrt(n.n), the reciprocal square root rounded
        // once (correctly rounded: equal to RN(1/sqrt(x)) evaluated in double)
        const float inv = rsqrt_rn(n2);
        const float d = __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(n[0], inv), f.light_dir[0]),
                                            __fmul_rn(__fmul_rn(n[1], inv), f.light_dir[1])),
                                  __fmul_rn(__fmul_rn(n[2], inv), f.light_dir[2]));
        di = fmaxf(d, 0.0f);
    }
    const float light = __fadd_rn(f.ambient, __fmul_rn(f.diffuse, di));
    return {__fmul2_rn(__fmul2_rn(crg, dup2(light)), dup2(alpha)),
            make_float2(__fmul_rn(__fmul_rn(cba.x, light), alpha), alpha)};
}

__device__ __forceinline__ uint32_t blend_rgba8(float2 rg, float2 ba) {
    // SRC_ALPHA / ONE_MINUS_SRC_ALPHA over a cleared UNORM8 target.
    const float a = fminf(fmaxf(ba.y, 0.0f), 1.0f);
    const uint32_t r = (uint32_t)rintf(__fmul_rn(__fmul_rn(fminf(fmaxf(rg.x, 0.0f), 1.0f), a), 255.0f));
    const uint32_t g = (uint32_t)rintf(__fmul_rn(__fmul_rn(fminf(fmaxf(rg.y, 0.0f), 1.0f), a), 255.0f));
    const uint32_t b = (uint32_t)rintf(__fmul_rn(__fmul_rn(fminf(fmaxf(ba.x, 0.0f), 1.0f), a), 255.0f));
    const uint32_t al = (uint32_t)rintf(__fmul_rn(__fmul_rn(a, a), 255.0f));
    return r | (g << 8) | (b << 16) | (al << 24);
}

// Is a sample of this brick exactly transparent under the job's LUT?
// m = the brick's (min, max) stored values.
template <bool SMEM_LUT, bool FAST>
__device__ __forceinline__ bool brick_clear(const MarchFrame &f, float2 m, const int *prefix) {
    if (!(m.x == m.x)) return false;  // NaN in the brick
    const float d0 = __fmul_rn(m.x, f.value_scale), d1 = __fmul_rn(m.y, f.value_scale);
    const float dlo = fminf(d0, d1), dhi = fmaxf(d0, d1);
    if (!(dlo == dlo && dhi == dhi)) return false;
    // the LUT coordinates of the extreme densities, rounded as the march
    // rounds them (FAST: one FMA); both roundings are monotone in d
    const float clo = FAST ? fmaf(dlo, f.flut_size, -0.5f) : __fadd_rn(__fmul_rn(dlo, f.flut_size), -0.5f);
    const float chi = FAST ? fmaf(dhi, f.flut_size, -0.5f) : __fadd_rn(__fmul_rn(dhi, f.flut_size), -0.5f);
    const int ilo = lut_index(floorf(clo), f.flut_max);
    const int ihi = lut_index(__fadd_rn(floorf(chi), 1.0f), f.flut_max);
    return prefix_entry<SMEM_LUT>(prefix, ihi + 1) == prefix_entry<SMEM_LUT>(prefix, ilo);
}

// One pixel's ray of volume.frag.glsl:main (lines 70-122).  PACKED: the x and
// y coordinates in packed instructions (their frame constants then take six
// registers); scalar ones read the constants from the parameter bank.
template <int LOG2B, int UNROLL, bool NORMALS, bool SMEM_LUT, bool COMPACT, bool FAST, int LERP, bool PACKED>
__device__ __forceinline__ void march_ray(const JobDesc &job, int px, int py, const float4 *lut,
                                          const int *prefix, float2 &acc_rg, float2 &acc_ba,
                                          unsigned &n_skipped, unsigned &n_shaded) {
    constexpr int B = 1 << LOG2B, ROW = brick_apron(LOG2B), SLICE = ROW * ROW;
    constexpr int RECS = brick_records(LOG2B);
    const MarchFrame &f = job.f;
    float pos[3], dstep[3];
    if (!setup_ray(f, px, py, pos, dstep)) return;
    // (x, y) lanes packed, z scalar; per lane the reference expressions
    float2 pxy = make_float2(pos[0], pos[1]);
    float pz = pos[2];
    const float2 dxy = make_float2(dstep[0], dstep[1]);
    const float dz = dstep[2];
    const float2 nbmin_xy = make_float2(-f.bmin[0], -f.bmin[1]);
    const float2 inv_xy = make_float2(f.inv_ext[0], f.inv_ext[1]);
    const float2 fext_xy = make_float2(f.fext[0], f.fext[1]);
    const float nbmin_z = -f.bmin[2], inv_z = f.inv_ext[2], fext_z = f.fext[2];
    const int nb1 = f.nb[1], nb2 = f.nb[2];
    bool entered = false;
    int cur_brick = -1;
    bool clear = false;
    using Rec = typename RecordOf<COMPACT>::T;
    const Rec *bp = static_cast<const Rec *>(job.records);
    int i = 0;
    for (;;) {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            if (!(i < f.max_steps && acc_ba.y < 0.99f)) return;
            // world_to_texture_coords (frag:25-27, 88)
            const float2 txy = PACKED ? __fmul2_rn(__fadd2_rn(pxy, nbmin_xy), inv_xy)
                                      : make_float2(__fmul_rn(__fadd_rn(pxy.x, -f.bmin[0]), f.inv_ext[0]),
                                                    __fmul_rn(__fadd_rn(pxy.y, -f.bmin[1]), f.inv_ext[1]));
            const float tz = __fmul_rn(__fadd_rn(pz, nbmin_z), inv_z);
            const bool valid = txy.x >= 0.0f && txy.x <= 1.0f && txy.y >= 0.0f &&
                               txy.y <= 1.0f && tz >= 0.0f && tz <= 1.0f;
            if (valid) {
                entered = true;
                // texel coordinate u = t*size - 0.5, lower texel k = floor(u)
                const float2 sxy = PACKED ? __fmul2_rn(txy, fext_xy)
                                          : make_float2(__fmul_rn(txy.x, f.fext[0]), __fmul_rn(txy.y, f.fext[1]));
                const float ux = __fadd_rn(sxy.x, -0.5f), uy = __fadd_rn(sxy.y, -0.5f);
                const float uz = __fadd_rn(__fmul_rn(tz, fext_z), -0.5f);
                const float flx = floorf(ux), fly = floorf(uy), flz = floorf(uz);
                const int kx = (int)flx + 1, ky = (int)fly + 1, kz = (int)flz + 1;
                const int id = ((kx >> LOG2B) * nb1 + (ky >> LOG2B)) * nb2 + (kz >> LOG2B);
                if (id != cur_brick) {
                    cur_brick = id;
                    const uint4 bi = __ldg(job.bricks + id);
                    bp = static_cast<const Rec *>(job.records) + (size_t)bi.x * RECS;
                    clear = job.skip &&
                            brick_clear<SMEM_LUT, FAST>(f, make_float2(__uint_as_float(bi.y),
                                                                       __uint_as_float(bi.z)),
                                                        prefix);
                }
                if (!clear) {
                    ++n_shaded;
                    const int j = (kx & (B - 1)) * SLICE + (ky & (B - 1)) * ROW + (kz & (B - 1));
                    composite<FAST>(shade_sample<LOG2B, NORMALS, SMEM_LUT, FAST, LERP>(
                                        f, bp + j, __fadd_rn(ux, -flx), __fadd_rn(uy, -fly), __fadd_rn(uz, -flz), lut),
                                    acc_rg, acc_ba);
                } else {
                    ++n_skipped;
                }
            } else {
                const bool never = entered || (txy.x < 0.0f && dxy.x <= 0.0f) ||
                                   (txy.x > 1.0f && dxy.x >= 0.0f) ||
                                   (txy.y < 0.0f && dxy.y <= 0.0f) ||
                                   (txy.y > 1.0f && dxy.y >= 0.0f) || (tz < 0.0f && dz <= 0.0f) ||
                                   (tz > 1.0f && dz >= 0.0f);
                if (never) return;
            }
            // current_world_pos += ray_dir * step_size (frag:118)
            pxy = __fadd2_rn(pxy, dxy);
            pz = __fadd_rn(pz, dz);
            ++i;
        }
    }
}

// The pixel of a lane in its warp's 8x4 block, in Z-order.  The L1 data pipe
// serves a 16-byte gather in passes of 8 lanes and an 8-byte gather in passes
// of 16, each taking longer the more 128-byte lines its lanes touch (it is
// 80-88 % busy on the large frames): in Z-order a pass covers 4x2 or 4x4
// pixels instead of 8x1 or 8x2.  Measured against row order: a 1024^2 frame
// of 256^3 uint8 with float records 538 -> 497 us, a 512^2 frame of 384^3
// with half records 84.7 -> 79.8 us.
__device__ __forceinline__ int lane_x(int lane) { return (lane & 1) | ((lane >> 1) & 2) | ((lane >> 2) & 4); }
__device__ __forceinline__ int lane_y(int lane) { return ((lane >> 1) & 1) | ((lane >> 2) & 2); }

// Stages a job's LUT with an apron entry at either end (s_lut[0] = entry 0,
// s_lut[1 + i] = entry i, s_lut[1 + size] = entry size - 1) and its prefix
// counts in shared memory.
__device__ __forceinline__ void stage_lut(float4 *s_lut, int *s_prefix, const JobDesc &job) {
    const int size = job.f.lut_size;
    for (int k = threadIdx.x; k < size + 2; k += blockDim.x) s_lut[k] = job.lut[min(max(k - 1, 0), size - 1)];
    for (int k = threadIdx.x; k <= size; k += blockDim.x) s_prefix[k] = job.prefix[k];
}

// Writes the lane's pixel (writes: it has one) and adds the warp's sample
// counts.
__device__ __forceinline__ void store_pixel(const JobDesc &job, int px, int py, bool writes, float2 acc_rg,
                                            float2 acc_ba, unsigned n_inbox, unsigned n_shaded, int lane) {
    if (writes) {
        const long long idx = (long long)py * job.f.width + px;
        if (job.out8) job.out8[idx] = blend_rgba8(acc_rg, acc_ba);
        if (job.outf) job.outf[idx] = make_float4(acc_rg.x, acc_rg.y, acc_ba.x, acc_ba.y);
    }
    if (job.counters) {
        unsigned long long a = n_inbox, b = n_shaded;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0 && a) {
            atomicAdd(job.counters, a);
            atomicAdd(job.counters + 1, b);
        }
    }
}

template <int LOG2B, int UNROLL, bool NORMALS, bool SMEM_LUT, bool COMPACT, bool FAST, int LERP, bool PACKED>
__device__ __forceinline__ void march_tile(const JobDesc &job, int px, int py, const float4 *lut,
                                           const int *prefix, int lane) {
    const bool in_image = px < job.f.width && py < job.f.height;
    float2 acc_rg = make_float2(0.0f, 0.0f), acc_ba = make_float2(0.0f, 0.0f);
    unsigned n_skipped = 0, n_shaded = 0;
    if (in_image)
        march_ray<LOG2B, UNROLL, NORMALS, SMEM_LUT, COMPACT, FAST, LERP, PACKED>(job, px, py, lut, prefix, acc_rg,
                                                                                 acc_ba, n_skipped, n_shaded);
    store_pixel(job, px, py, in_image, acc_rg, acc_ba, n_shaded + n_skipped, n_shaded, lane);
}

// Persistent batch kernel of one variant: normals or not, LUT staged in
// shared memory or read from global memory, float or half records, exact or
// fast arithmetic (the launcher groups a batch's jobs by variant, so that
// each kernel carries one march and stays within its register budget).  The
// job table is the kernel's own parameter block (read through the constant
// cache).  Dynamic shared memory (SMEM_LUT): p.lut_smem_entries + 2 float4
// entries (a LUT and its apron) and p.lut_smem_entries + 1 prefix counts;
// p.lut_smem_entries is at least every job's LUT size.
template <int LOG2B, int UNROLL, bool NORMALS, bool SMEM_LUT, bool COMPACT, bool FAST>
__global__ void __launch_bounds__(kBatchThreads, COMPACT ? 5 : 4)
march_batch_kernel(const __grid_constant__ BatchParams p) {
    extern __shared__ float4 s_dyn[];
    float4 *s_lut = s_dyn;
    int *s_prefix = reinterpret_cast<int *>(s_dyn + p.lut_smem_entries + 2);
    __shared__ int s_tile, s_job_idx;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warps_x = p.tile_w >> 3;
    const int sub_x = (warp % warps_x) * 8 + lane_x(lane);
    const int sub_y = (warp / warps_x) * 4 + lane_y(lane);
    int cur_job = -1;
    for (;;) {
        if (threadIdx.x == 0) {
            const int t = atomicAdd(p.work, 1);
            int lo = 0, hi = p.njobs - 1;  // last job whose first tile is <= t
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (p.tile_base[mid] <= t) lo = mid; else hi = mid - 1;
            }
            s_tile = t;
            s_job_idx = lo;
        }
        __syncthreads();
        const int t = s_tile, j = s_job_idx;
        if (t >= p.total_tiles) break;
        const JobDesc &job = p.jobs[j];
        if (SMEM_LUT && j != cur_job) {
            // stage the job's LUT (the previous tile's readers passed the
            // barrier at the end of the last round)
            stage_lut(s_lut, s_prefix, job);
            __syncthreads();
            cur_job = j;
        }
        const int local = t - job.tile_base;
        const int px = (local % job.tiles_x) * p.tile_w + sub_x;
        const int py = (local / job.tiles_x) * p.tile_h + sub_y;
        march_tile<LOG2B, UNROLL, NORMALS, SMEM_LUT, COMPACT, FAST, COMPACT ? kLerpMixed : kLerpPacked, false>(
            job, px, py, SMEM_LUT ? s_lut + 1 : job.lut, SMEM_LUT ? s_prefix : job.prefix, lane);
        __syncthreads();  // s_tile / the staged LUT are rewritten next round
    }
}

// Single-job kernel: one block per tile of one render; the job descriptor
// is the parameter block itself (static offsets), as in a plain frame kernel.
// One instantiation per variant (normals, LUT in shared memory, half
// records, arithmetic), chosen on the host: each gets its own register
// allocation.  SMEM_LUT requires job.f.lut_size <= p.lut_smem_entries.  All
// normals variants have 48 registers and 40 warps per SM; half records mostly
// in blocks of 128 threads on half a tile (single_threads in batch.cu).
template <int LOG2B, int UNROLL, bool NORMALS, bool SMEM_LUT, bool COMPACT, bool FAST>
__global__ void __launch_bounds__(kBatchThreads, NORMALS ? 5 : 6)
march_single_kernel(const __grid_constant__ SingleParams p) {
    extern __shared__ float4 s_dyn[];
    float4 *s_lut = s_dyn;
    int *s_prefix = reinterpret_cast<int *>(s_dyn + p.lut_smem_entries + 2);
    const JobDesc &job = p.job;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warps_x = p.tile_w >> 3;
    if (SMEM_LUT) {
        stage_lut(s_lut, s_prefix, job);
        __syncthreads();
    }
    const int t = blockIdx.x;
    const int px = (t % job.tiles_x) * p.tile_w + (warp % warps_x) * 8 + lane_x(lane);
    const int py = (t / job.tiles_x) * p.tile_h + (warp / warps_x) * 4 + lane_y(lane);
    march_tile<LOG2B, UNROLL, NORMALS, SMEM_LUT, COMPACT, FAST, COMPACT ? kLerpMixedScalar : kLerpPacked, true>(
        job, px, py, SMEM_LUT ? s_lut + 1 : job.lut, SMEM_LUT ? s_prefix : job.prefix, lane);
}

// The march of one small render with SPLIT lanes per ray: lane q of a ray
// evaluates the samples q, q + SPLIT, ..., and all its lanes composite them
// in order, so every rounding is the one-lane march's.  What a sample adds
// (Source) does not depend on the samples before it; samples evaluated
// beyond the ray's end are dropped.
//
// A frame of few pixels does not fill the chip: 256^2 are 2048 warps of rays,
// 3.4 per scheduler, each a serial chain of gathers and shading per sample
// (issue 37 %).  Here it is SPLIT times the warps with 1/SPLIT of the chain.
// Each group of samples costs 4 * SPLIT shuffles and as many compositing
// steps, so a frame that fills the chip is faster with one lane per ray
// (split_lanes in batch.cu).  A warp is 4x2 (SPLIT 4) or 4x4 pixels.
template <int LOG2B, int SPLIT, bool NORMALS, bool SMEM_LUT, bool COMPACT, bool FAST>
__global__ void __launch_bounds__(kBatchThreads, split_blocks_per_sm(COMPACT))
march_split_kernel(const __grid_constant__ SingleParams p) {
    constexpr int B = 1 << LOG2B, ROW = brick_apron(LOG2B), SLICE = ROW * ROW;
    constexpr int RECS = brick_records(LOG2B);
    constexpr unsigned kAll = 0xffffffffu, kGroup = (1u << SPLIT) - 1;
    using Rec = typename RecordOf<COMPACT>::T;
    extern __shared__ float4 s_dyn[];
    float4 *s_lut = s_dyn;
    int *s_prefix = reinterpret_cast<int *>(s_dyn + p.lut_smem_entries + 2);
    const JobDesc &job = p.job;
    const MarchFrame &f = job.f;
    if (SMEM_LUT) {
        stage_lut(s_lut, s_prefix, job);
        __syncthreads();
    }
    const float4 *lut = SMEM_LUT ? s_lut + 1 : job.lut;
    const int *prefix = SMEM_LUT ? s_prefix : job.prefix;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & (SPLIT - 1), ray = lane / SPLIT;
    // the warp's block of pixels in Z-order: 4x2 or 4x4
    const int t = blockIdx.x;
    const int px = (t % job.tiles_x) * split_tile_w(SPLIT) + (warp & 1) * 4 + ((ray & 1) | ((ray >> 1) & 2));
    const int py = (t / job.tiles_x) * split_tile_h(SPLIT) + (warp >> 1) * (8 / SPLIT) +
                   (((ray >> 1) & 1) | ((ray >> 2) & 2));
    const bool in_image = px < f.width && py < f.height;
    float pos[3] = {}, d[3] = {};
    bool done = !in_image || !setup_ray(f, px, py, pos, d);
    for (int k = 0; k < q; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) pos[a] = __fadd_rn(pos[a], d[a]);
    __syncwarp();
    float2 acc_rg = make_float2(0.0f, 0.0f), acc_ba = make_float2(0.0f, 0.0f);
    unsigned n_inbox = 0, n_shaded = 0;
    bool entered = false, clear = false;
    int cur_brick = -1;
    const Rec *bp = nullptr;
    for (int i = 0; __any_sync(kAll, !done); i += SPLIT) {
        float tc[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) tc[a] = __fmul_rn(__fadd_rn(pos[a], -f.bmin[a]), f.inv_ext[a]);
        const bool valid = tc[0] >= 0.0f && tc[0] <= 1.0f && tc[1] >= 0.0f && tc[1] <= 1.0f && tc[2] >= 0.0f &&
                           tc[2] <= 1.0f;
        // the ray ends here if it has been in the box before, or cannot reach it
        bool ends = i + q >= f.max_steps;
        bool never = false;
        if (!valid)
#pragma unroll
            for (int a = 0; a < 3; ++a)
                never = never || (tc[a] < 0.0f && d[a] <= 0.0f) || (tc[a] > 1.0f && d[a] >= 0.0f);
        ends = ends || never;
        Source s = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
        bool shaded = false;
        if (valid && !done && !ends) {
            int k[3];
            float fr[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float u = __fadd_rn(__fmul_rn(tc[a], f.fext[a]), -0.5f), fl = floorf(u);
                k[a] = (int)fl + 1;
                fr[a] = __fadd_rn(u, -fl);
            }
            const int id = ((k[0] >> LOG2B) * f.nb[1] + (k[1] >> LOG2B)) * f.nb[2] + (k[2] >> LOG2B);
            if (id != cur_brick) {
                cur_brick = id;
                const uint4 bi = __ldg(job.bricks + id);
                bp = static_cast<const Rec *>(job.records) + (size_t)bi.x * RECS;
                clear = job.skip && brick_clear<SMEM_LUT, FAST>(f, make_float2(__uint_as_float(bi.y),
                                                                               __uint_as_float(bi.z)), prefix);
            }
            if (!clear) {
                const int j = (k[0] & (B - 1)) * SLICE + (k[1] & (B - 1)) * ROW + (k[2] & (B - 1));
                s = shade_sample<LOG2B, NORMALS, SMEM_LUT, FAST, COMPACT ? kLerpMixedScalar : kLerpPacked>(
                    f, bp + j, fr[0], fr[1], fr[2], lut);
                shaded = true;
            }
        }
        // per ray, one bit per sample of the group (the same on all its lanes):
        // in the box, shaded, and the first one at which the ray ends
        const unsigned base = lane & ~(SPLIT - 1);
        const unsigned in = (__ballot_sync(kAll, valid) >> base) & kGroup;
        const unsigned lit = (__ballot_sync(kAll, shaded) >> base) & kGroup;
        unsigned stop = (__ballot_sync(kAll, ends) >> base) & kGroup;
        const unsigned after = entered ? kGroup : ~((in & (0u - in)) * 2 - 1) & (in ? kGroup : 0u);
        stop |= ~in & after & kGroup;  // outside after having been inside
        const unsigned before = stop ? (stop & (0u - stop)) - 1 : kGroup;  // the samples in front of it
        entered = entered || in != 0;
        unsigned taken = 0;
#pragma unroll
        for (int k = 0; k < SPLIT; ++k) {
            const Source sk = {make_float2(__shfl_sync(kAll, s.rg.x, k, SPLIT), __shfl_sync(kAll, s.rg.y, k, SPLIT)),
                               make_float2(__shfl_sync(kAll, s.ba.x, k, SPLIT), __shfl_sync(kAll, s.ba.y, k, SPLIT))};
            if (!done && acc_ba.y < 0.99f && ((before >> k) & 1)) {
                taken |= 1u << k;
                if ((lit >> k) & 1) composite<FAST>(sk, acc_rg, acc_ba);
            }
        }
        n_inbox += __popc(taken & in);
        n_shaded += __popc(taken & lit);
        done = done || stop != 0 || !(acc_ba.y < 0.99f);
#pragma unroll
        for (int k = 0; k < SPLIT; ++k)
#pragma unroll
            for (int a = 0; a < 3; ++a) pos[a] = __fadd_rn(pos[a], d[a]);
    }
    const bool writes = in_image && q == 0;
    store_pixel(job, px, py, writes, acc_rg, acc_ba, writes ? n_inbox : 0, writes ? n_shaded : 0, lane);
}

template <int LOG2B, int SPLIT, bool FAST>
const void *split_variant_of(int v) {
    switch (v & 7) {
    case 0: return (const void *)march_split_kernel<LOG2B, SPLIT, false, false, false, FAST>;
    case 1: return (const void *)march_split_kernel<LOG2B, SPLIT, true, false, false, FAST>;
    case 2: return (const void *)march_split_kernel<LOG2B, SPLIT, false, true, false, FAST>;
    case 3: return (const void *)march_split_kernel<LOG2B, SPLIT, true, true, false, FAST>;
    case 4: return (const void *)march_split_kernel<LOG2B, SPLIT, false, false, true, FAST>;
    case 5: return (const void *)march_split_kernel<LOG2B, SPLIT, true, false, true, FAST>;
    case 6: return (const void *)march_split_kernel<LOG2B, SPLIT, false, true, true, FAST>;
    default: return (const void *)march_split_kernel<LOG2B, SPLIT, true, true, true, FAST>;
    }
}

template <int LOG2B>
const void *split_kernel_log2(int lanes, int v) {
    if (lanes == 4)
        return (v & kSingleFast) ? split_variant_of<LOG2B, 4, true>(v) : split_variant_of<LOG2B, 4, false>(v);
    return (v & kSingleFast) ? split_variant_of<LOG2B, 2, true>(v) : split_variant_of<LOG2B, 2, false>(v);
}

template <int LOG2B, int UNROLL, bool FAST>
const void *single_variant_of(int v) {
    switch (v & 7) {
    case 0: return (const void *)march_single_kernel<LOG2B, UNROLL, false, false, false, FAST>;
    case 1: return (const void *)march_single_kernel<LOG2B, UNROLL, true, false, false, FAST>;
    case 2: return (const void *)march_single_kernel<LOG2B, UNROLL, false, true, false, FAST>;
    case 3: return (const void *)march_single_kernel<LOG2B, UNROLL, true, true, false, FAST>;
    case 4: return (const void *)march_single_kernel<LOG2B, UNROLL, false, false, true, FAST>;
    case 5: return (const void *)march_single_kernel<LOG2B, UNROLL, true, false, true, FAST>;
    case 6: return (const void *)march_single_kernel<LOG2B, UNROLL, false, true, true, FAST>;
    default: return (const void *)march_single_kernel<LOG2B, UNROLL, true, true, true, FAST>;
    }
}

template <int LOG2B, int UNROLL>
const void *single_variant(int v) {
    return (v & kSingleFast) ? single_variant_of<LOG2B, UNROLL, true>(v) : single_variant_of<LOG2B, UNROLL, false>(v);
}

template <int LOG2B>
const void *single_kernel_log2(const Tuning &t, int variant) {
    if (t.steps_per_iter >= 4) return single_variant<LOG2B, 4>(variant);
    return single_variant<LOG2B, 1>(variant);
}

template <int LOG2B, int UNROLL, bool FAST>
const void *batch_variant_of(int v) {
    switch (v & 7) {
    case 0: return (const void *)march_batch_kernel<LOG2B, UNROLL, false, false, false, FAST>;
    case 1: return (const void *)march_batch_kernel<LOG2B, UNROLL, true, false, false, FAST>;
    case 2: return (const void *)march_batch_kernel<LOG2B, UNROLL, false, true, false, FAST>;
    case 3: return (const void *)march_batch_kernel<LOG2B, UNROLL, true, true, false, FAST>;
    case 4: return (const void *)march_batch_kernel<LOG2B, UNROLL, false, false, true, FAST>;
    case 5: return (const void *)march_batch_kernel<LOG2B, UNROLL, true, false, true, FAST>;
    case 6: return (const void *)march_batch_kernel<LOG2B, UNROLL, false, true, true, FAST>;
    default: return (const void *)march_batch_kernel<LOG2B, UNROLL, true, true, true, FAST>;
    }
}

template <int LOG2B, int UNROLL>
const void *batch_variant(int v) {
    return (v & kSingleFast) ? batch_variant_of<LOG2B, UNROLL, true>(v) : batch_variant_of<LOG2B, UNROLL, false>(v);
}

template <int LOG2B>
const void *batch_kernel_log2(const Tuning &t, int variant) {
    if (t.steps_per_iter >= 4) return batch_variant<LOG2B, 4>(variant);
    return batch_variant<LOG2B, 1>(variant);
}

template <int LOG2B>
int max_blocks_log2(const Tuning &t, int lut_smem_entries, int variant) {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel_log2<LOG2B>(t, variant), kBatchThreads,
                                                  batch_smem_bytes(lut_smem_entries));
    return n;
}

}  // namespace pvr
