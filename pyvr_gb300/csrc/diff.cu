// Differentiable march: gradients of an image loss with respect to the RGBA
// LUT and the voxel values (FP32 volume), for several views of one scene.
//
// Forward: the march of pyvr/shaders/volume.frag.glsl:70-122 with the
// renderer's exact per-sample arithmetic (setup_ray, texel fractions,
// z-then-y-then-x trilinear lerps, LUT lerp, pvr_expf opacity correction,
// Lambert term, front-to-back compositing), so the float image equals the
// renderer's float image.  Per pixel it also keeps the number of loop
// iterations executed; nothing is kept per sample.
//
// Backward: the same march a second time, front to back, with the forward's
// own positions, samples and accumulators (bit for bit).  With T_i = 1 - acc.a
// the transmittance in front of sample i, c_i = light_i * rgb_i and acc_i the
// accumulated colour behind it, what lies beyond sample i is the image minus
// acc_i, so
//   dC/dc_i = T_i alpha_i,
//   dC/dalpha_i = T_i c_i - (C - acc_i) / (1 - alpha_i),
//   dA/dalpha_i = (1 - A) / (1 - alpha_i).
// T_i is exact here (a walk from the last sample to the first has to rebuild
// it by division from 1 - A), and all rays of a warp are at the same step,
// so their gathers and table entries coincide as in the forward.  The last
// sample of a ray has nothing beyond it: C - acc_i is exactly 0 there, and
// dA/dalpha is T_i.
//
// Chain rule down to the leaves: alpha = 1 - exp(-a K) gives
// dalpha/da = K exp(-a K); the LUT lerp rgba = lerp(lut[i0], lut[i1], f)
// gives weights (1 - f, f) to the two entries and d rgba/d density =
// (lut[i1] - lut[i0]) * lut_size; density = value_scale * trilinear(voxels)
// gives each of the 8 corners its trilinear weight.  Normals (given, or
// (density, 0, 0) without a normal volume) are held constant.
//
// What bounds it, and the layout: a sample needs 8 texels of 1 (or, with
// normals, 4) floats.  Gathered from the (D,H,W) and (D,H,W,3) arrays that
// is 8 (32) loads, and the L1 data pipe is their limit (93 % busy).  With
// a workspace (pvr_diff_workspace) each call first packs the volume into
// 16-byte texels, which the march reads with 8 loads (value and normal of a
// texel) or, without normals, 2 (the four (y, z) corners of a texel).
// Measured on 128^3 with normals, 8 views of 512^2, from the scene's arrays and
// walking backward -> now (the profile's launches): forward 985 -> 400 us,
// backward to the LUT 3250 -> 820 us, the packing 13 us of each; 72^3 without
// normals, 3 views of 251x197, backward to voxels and LUT 303 -> 110 us.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "pvr_device.cuh"
#include "pvr_internal.h"

namespace pvr {
namespace {

constexpr int kDiffMaxViews = 32;   // views per launch (more are split)
constexpr int kDiffThreads = 256;   // 16 x 16 pixel tile; warps cover 8 x 4 pixels
constexpr int kDiffTile = 16;
constexpr int kDiffMaxLut = 2048;   // LUT entries (shared-memory gradient)
// LUTs up to this many entries get a gradient table per warp (8 KB each),
// larger ones one per block, whose float atomics cost more than the L1 that
// the tables take: 128^3 with normals, 8 views of 512^2, high opacity, backward
// us with warp tables / one table, 272 entries 2568 / 3156, 384 2546 / 3076,
// 512 2480 / 2925.  Three blocks per SM fit up to about 530 entries.
constexpr int kWarpTableLut = 512;

// Where a sample's texels come from: the scene's arrays (8 or, with normals,
// 32 scalar loads), or packed texels with normals, or packed (y, z) quads of
// values.
enum TexelSource { kLinear = 0, kLinearNormals = 1, kPackedNormals = 2, kPackedQuads = 3 };
__host__ __device__ constexpr bool is_packed(int source) { return source >= kPackedNormals; }

struct DiffParams {
    const float *vol;       // (D, H, W) C order: texel (x, y, z) at (x * H + y) * D + z
    const float *nrm;       // 3 floats per texel, or null
    const float4 *texels;   // packed texels (kPackedNormals, kPackedQuads)
    const float4 *lut;
    float4 *image;          // [view][y][x]
    int *steps;             // [view][y][x] loop iterations executed
    const float4 *gimage;   // dL/dimage
    float4 *glut;           // dL/dlut, accumulated; or null
    float *gvol;            // dL/dvoxel, accumulated; or null
    float4 *gquads;         // dL/dvoxel by (y, z) quads (zeroed; added to gvol afterwards); or null
    int nviews, tiles_x, tiles_y;
    int ext[3];             // texels along world x, y, z (W, H, D)
    MarchFrame f[kDiffMaxViews];
};

// lerp_tex2 with the difference as fma(a, -1, b), which is b - a exactly as
// rounded there: 2 % faster here, where the addition form costs moves.
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float t) {
    return __ffma2_rn(make_float2(t, t), __ffma2_rn(a, make_float2(-1.0f, -1.0f), b), a);
}

struct Sample {
    int k[3];        // lower texel, -1 .. ext - 1
    float fx, fy, fz;
    int j0;          // LUT entry floor(lu) clamped to -1 .. size - 1
    float la;
    float4 A, B;
    float r, g, b;   // LUT colour
    float e;         // exp(-a K)
    float alpha;     // 1 - e
    float light;     // ambient + diffuse * max(dot(n, L), 0)
};

// texture coordinate of a world position (frag:25-27, 88) and its validity
__device__ __forceinline__ bool tex_coords(const MarchFrame &f, const float pos[3], float t[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) t[a] = __fmul_rn(__fadd_rn(pos[a], -f.bmin[a]), f.inv_ext[a]);
    return t[0] >= 0.0f && t[0] <= 1.0f && t[1] >= 0.0f && t[1] <= 1.0f && t[2] >= 0.0f && t[2] <= 1.0f;
}

// once the ray has left the valid run, or cannot reach it, the march ends
__device__ __forceinline__ bool never_valid(const float t[3], const float d[3]) {
    bool nv = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) nv = nv || (t[a] < 0.0f && d[a] <= 0.0f) || (t[a] > 1.0f && d[a] >= 0.0f);
    return nv;
}

// Packed texels: texel clamp(i - 1) of each axis at index i in [0, ext + 1]
// (kPackedNormals), so a footprint is never clamped; quads likewise along x,
// and at (y, z) index (j, l) in [0, ext] the corners {(y, z), (y, z + 1),
// (y + 1, z), (y + 1, z + 1)} of lower texel (j - 1, l - 1).
__host__ __device__ inline long long packed_texels(const int ext[3], bool normals) {
    return (long long)(ext[0] + 2) * (ext[1] + (normals ? 2 : 1)) * (ext[2] + (normals ? 2 : 1));
}

// Also clears the first nquads gradient quads (never more than the texels)
// and the first nglut floats of the LUT gradient.
template <int SOURCE>
__global__ void pack_kernel(const float *__restrict__ vol, const float *__restrict__ nrm, int ex, int ey, int ez,
                            float4 *__restrict__ out, float4 *__restrict__ gquads, int nquads,
                            float *__restrict__ glut, int nglut) {
    const int ny = ey + (SOURCE == kPackedNormals ? 2 : 1), nz = ez + (SOURCE == kPackedNormals ? 2 : 1);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int total = (ex + 2) * ny * nz;
    for (int k = i; k < nglut; k += gridDim.x * blockDim.x) glut[k] = 0.0f;
    if (i >= total) return;
    if (i < nquads) gquads[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int z = i % nz, y = (i / nz) % ny, x = min(max(i / (nz * ny) - 1, 0), ex - 1);
    const int y0 = min(max(y - 1, 0), ey - 1), z0 = min(max(z - 1, 0), ez - 1);
    if (SOURCE == kPackedNormals) {
        const int t = (x * ey + y0) * ez + z0;
        out[i] = make_float4(vol[t], nrm[3 * t + 0], nrm[3 * t + 1], nrm[3 * t + 2]);
    } else {
        const int y1 = min(y, ey - 1), z1 = min(z, ez - 1);
        const float *r0 = vol + (x * ey + y0) * ez, *r1 = vol + (x * ey + y1) * ez;
        out[i] = make_float4(r0[z0], r0[z1], r1[z0], r1[z1]);
    }
}

// dL/dvoxel from the quads: voxel (x, y, z) is the lower and the upper corner
// of two quad indices per axis, and of one more at each clamped face.
__global__ void unpack_grad_kernel(const float4 *__restrict__ quads, int ex, int ey, int ez, bool overwrite,
                                   float *__restrict__ gvol) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ex * ey * ez) return;
    const int z = i % ez, y = (i / ez) % ey, x = i / (ez * ey);
    const int ny = ey + 1, nz = ez + 1;
    float sum = 0.0f;
    for (int qx = x == 0 ? 0 : x + 1; qx <= (x == ex - 1 ? ex + 1 : x + 1); ++qx) {
        for (int qy = y; qy <= y + 1; ++qy)
            for (int qz = z; qz <= z + 1; ++qz) {
                const float4 q = __ldg(quads + (qx * ny + qy) * nz + qz);
                // as lower corner: index c + 1, or 0 on the first texel; as
                // upper corner: index c, or ext on the last
                const bool yl = qy == y + 1 || y == 0, yu = qy == y || y == ey - 1;
                const bool zl = qz == z + 1 || z == 0, zu = qz == z || z == ez - 1;
                sum += (yl && zl ? q.x : 0.0f) + (yl && zu ? q.y : 0.0f) + (yu && zl ? q.z : 0.0f) +
                       (yu && zu ? q.w : 0.0f);
            }
    }
    gvol[i] = overwrite ? sum : gvol[i] + sum;
}

__device__ __forceinline__ int texel(const DiffParams &p, int x, int y, int z) {
    return (x * p.ext[1] + y) * p.ext[2] + z;
}

// The 8 texels of a sample in the scene's own arrays; bits 2, 1 and 0 of the
// index: upper x, y and z.
struct Corners {
    int i[8];
};
__device__ __forceinline__ Corners corners(const DiffParams &p, const Sample &s) {
    int lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = max(s.k[a], 0);
        hi[a] = min(s.k[a] + 1, p.ext[a] - 1);
    }
    Corners c;
#pragma unroll
    for (int k = 0; k < 8; ++k) c.i[k] = texel(p, k & 4 ? hi[0] : lo[0], k & 2 ? hi[1] : lo[1], k & 1 ? hi[2] : lo[2]);
    return c;
}

__device__ __forceinline__ float lerp8(const float v[8], const Sample &s) {
    return lerp_tex(lerp_tex(lerp_tex(v[0], v[1], s.fz), lerp_tex(v[2], v[3], s.fz), s.fy),
                    lerp_tex(lerp_tex(v[4], v[5], s.fz), lerp_tex(v[6], v[7], s.fz), s.fy), s.fx);
}

__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// Stored value and normal at a sample; the lerps are the same per component
// whatever the source.
template <int SOURCE>
__device__ __forceinline__ float fetch(const DiffParams &p, const MarchFrame &f, const Sample &s, float n[3]) {
    if (SOURCE == kPackedNormals) {
        const int sy = p.ext[2] + 2, sx = (p.ext[1] + 2) * sy;
        const float4 *t = p.texels + ((s.k[0] + 1) * sx + (s.k[1] + 1) * sy + (s.k[2] + 1));
        const float4 r000 = __ldg(t), r001 = __ldg(t + 1);
        const float4 r010 = __ldg(t + sy), r011 = __ldg(t + sy + 1);
        t += sx;
        const float4 r100 = __ldg(t), r101 = __ldg(t + 1);
        const float4 r110 = __ldg(t + sy), r111 = __ldg(t + sy + 1);
        const float2 a = lerp2(lerp2(lerp2(lo2(r000), lo2(r001), s.fz),
                                             lerp2(lo2(r010), lo2(r011), s.fz), s.fy),
                                   lerp2(lerp2(lo2(r100), lo2(r101), s.fz),
                                             lerp2(lo2(r110), lo2(r111), s.fz), s.fy), s.fx);
        const float2 b = lerp2(lerp2(lerp2(hi2(r000), hi2(r001), s.fz),
                                             lerp2(hi2(r010), hi2(r011), s.fz), s.fy),
                                   lerp2(lerp2(hi2(r100), hi2(r101), s.fz),
                                             lerp2(hi2(r110), hi2(r111), s.fz), s.fy), s.fx);
        n[0] = a.y;
        n[1] = b.x;
        n[2] = b.y;
        return __fmul_rn(a.x, f.value_scale);
    }
    float density;
    if (SOURCE == kPackedQuads) {
        const int sy = p.ext[2] + 1, sx = (p.ext[1] + 1) * sy;
        const float4 *t = p.texels + ((s.k[0] + 1) * sx + (s.k[1] + 1) * sy + (s.k[2] + 1));
        const float4 q0 = __ldg(t), q1 = __ldg(t + sx);
        const float2 z0 = lerp2(make_float2(q0.x, q0.z), make_float2(q0.y, q0.w), s.fz);
        const float2 z1 = lerp2(make_float2(q1.x, q1.z), make_float2(q1.y, q1.w), s.fz);
        const float2 y = lerp2(make_float2(z0.x, z1.x), make_float2(z0.y, z1.y), s.fy);
        density = __fmul_rn(lerp_tex(y.x, y.y, s.fx), f.value_scale);
    } else {
        const Corners c = corners(p, s);
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __ldg(p.vol + c.i[k]);
        if (SOURCE == kLinearNormals) {
            float m[3][8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
                for (int a = 0; a < 3; ++a) m[a][k] = __ldg(p.nrm + 3 * c.i[k] + a);
#pragma unroll
            for (int a = 0; a < 3; ++a) n[a] = lerp8(m[a], s);
            return __fmul_rn(lerp8(v, s), f.value_scale);
        }
        density = __fmul_rn(lerp8(v, s), f.value_scale);
    }
    // the reference's unbound normal sampler reads the volume
    n[0] = density;
    n[1] = 0.0f;
    n[2] = 0.0f;
    return density;
}

// Everything one in-box sample computes (frag:93-110), with the renderer's
// rounding.  lut: the table in shared memory with an apron entry at either
// end (lut[-1] = lut[0], lut[size] = lut[size - 1]); for the scene's own arrays
// the table itself, since scalar gathers need L1 more: staged, 2048 entries
// took a 104^3 volume's forward from 65 to 72 us (48 registers) and 156 (40).
template <int SOURCE>
__device__ __forceinline__ void eval_sample(const DiffParams &p, const MarchFrame &f, const float t[3],
                                           const float4 *lut, Sample &s) {
    float fr[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float u = __fadd_rn(__fmul_rn(t[a], f.fext[a]), -0.5f);
        const float fl = floorf(u);
        fr[a] = __fadd_rn(u, -fl);
        s.k[a] = (int)fl;  // -1 .. ext-1
    }
    s.fx = fr[0]; s.fy = fr[1]; s.fz = fr[2];
    float n[3];
    const float density = fetch<SOURCE>(p, f, s, n);
    // texture(transfer_function_lut, vec2(density, 0.5)) (frag:96)
    const float lu = __fadd_rn(__fmul_rn(density, f.flut_size), -0.5f);
    const float lfl = floorf(lu);
    s.la = __fadd_rn(lu, -lfl);
    s.j0 = (int)fminf(fmaxf(lfl, -1.0f), f.flut_max);  // NaN: -1
    if (is_packed(SOURCE)) {
        s.A = lut[s.j0];
        s.B = lut[s.j0 + 1];
    } else {
        s.A = __ldg(lut + max(s.j0, 0));
        s.B = __ldg(lut + min(s.j0 + 1, f.lut_size - 1));
    }
    const float2 rg = lerp2(lo2(s.A), lo2(s.B), s.la), ba = lerp2(hi2(s.A), hi2(s.B), s.la);
    s.r = rg.x;
    s.g = rg.y;
    s.b = ba.x;
    s.e = pvr_expf(-__fmul_rn(ba.y, f.alpha_k));
    s.alpha = __fadd_rn(1.0f, -s.e);
    const float n2 = __fadd_rn(__fadd_rn(__fmul_rn(n[0], n[0]), __fmul_rn(n[1], n[1])), __fmul_rn(n[2], n[2]));
    float di = 0.0f;
    if (n2 > 0.0f) {
        const float inv = rsqrt_rn(n2);  // as the renderer: rounded once
        const float d = __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(n[0], inv), f.light_dir[0]),
                                            __fmul_rn(__fmul_rn(n[1], inv), f.light_dir[1])),
                                  __fmul_rn(__fmul_rn(n[2], inv), f.light_dir[2]));
        di = fmaxf(d, 0.0f);
    }
    s.light = __fadd_rn(f.ambient, __fmul_rn(f.diffuse, di));
}

// acc.c += (1 - acc.a) * (c * light * alpha); acc.a += (1 - acc.a) * alpha
__device__ __forceinline__ void composite(const Sample &s, float4 &acc) {
    const float tr = __fadd_rn(1.0f, -acc.w);
    acc.x = __fadd_rn(acc.x, __fmul_rn(tr, __fmul_rn(__fmul_rn(s.r, s.light), s.alpha)));
    acc.y = __fadd_rn(acc.y, __fmul_rn(tr, __fmul_rn(__fmul_rn(s.g, s.light), s.alpha)));
    acc.z = __fadd_rn(acc.z, __fmul_rn(tr, __fmul_rn(__fmul_rn(s.b, s.light), s.alpha)));
    acc.w = __fadd_rn(acc.w, __fmul_rn(tr, s.alpha));
}

// Lanes in Z-order inside the warp's 8x4 pixels, as in the renderer's march:
// the 8 lanes of one pass of a 16-byte gather cover 4x2 pixels.
__device__ __forceinline__ void pixel_of(int tile_in_view, int tiles_x, int &px, int &py) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    px = (tile_in_view % tiles_x) * kDiffTile + (warp & 1) * 8 +
         ((lane & 1) | ((lane >> 1) & 2) | ((lane >> 2) & 4));
    py = (tile_in_view / tiles_x) * kDiffTile + (warp >> 1) * 4 + (((lane >> 1) & 1) | ((lane >> 2) & 2));
}

__device__ __forceinline__ const float4 *stage_diff_lut(const DiffParams &p, float4 *s_lut) {
    const int size = p.f[0].lut_size;
    for (int k = threadIdx.x; k < size + 2; k += kDiffThreads) s_lut[k] = __ldg(p.lut + min(max(k - 1, 0), size - 1));
    return s_lut + 1;
}

// Blocks per SM that the forward's registers allow (0: the compiler's choice):
// the 32 loads of a sample of the scene's arrays with normals need 64
// registers to be in flight together (113 random scenes against the kernel
// before packing: at 48 registers 1.02 times as fast on average, the worst
// 0.78; at 64 1.09, the worst 0.89).
constexpr int forward_blocks(int source) { return source == kLinearNormals ? 4 : source == kLinear ? 5 : 0; }

// Dynamic shared memory (packed sources): the LUT and its apron (lut_size + 2
// entries).
template <int SOURCE>
__global__ void __launch_bounds__(kDiffThreads, forward_blocks(SOURCE))
diff_forward_kernel(const __grid_constant__ DiffParams p) {
    extern __shared__ float4 s_dyn[];
    const float4 *lut = p.lut;
    if (is_packed(SOURCE)) {
        lut = stage_diff_lut(p, s_dyn);
        __syncthreads();
    }
    const int per_view = p.tiles_x * p.tiles_y;
    const int view = blockIdx.x / per_view;
    const MarchFrame &f = p.f[view];
    int px, py;
    pixel_of(blockIdx.x % per_view, p.tiles_x, px, py);
    if (px >= f.width || py >= f.height) return;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int i = 0;
    float pos[3], d[3];
    if (setup_ray(f, px, py, pos, d)) {
        bool entered = false;
        for (;; ++i) {
            if (!(i < f.max_steps && acc.w < 0.99f)) break;
            float t[3];
            if (tex_coords(f, pos, t)) {
                entered = true;
                Sample s;
                eval_sample<SOURCE>(p, f, t, lut, s);
                composite(s, acc);
            } else if (entered || never_valid(t, d)) {
                break;
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) pos[a] = __fadd_rn(pos[a], d[a]);
        }
    }
    const long long idx = ((long long)view * f.height + py) * f.width + px;
    p.image[idx] = acc;
    p.steps[idx] = i;
}

// Adds a sample's voxel gradient (packed sources) to the quads, or without them
// (too small a workspace) to the voxels.
__device__ __forceinline__ void add_voxel_grad(const DiffParams &p, const Sample &s, float gd) {
    const float wx[2] = {1.0f - s.fx, s.fx}, wy[2] = {1.0f - s.fy, s.fy}, wz[2] = {1.0f - s.fz, s.fz};
    if (p.gquads) {
        // one 16-byte reduction per x corner
        const int sy = p.ext[2] + 1, sx = (p.ext[1] + 1) * sy;
        float4 *q = p.gquads + ((s.k[0] + 1) * sx + (s.k[1] + 1) * sy + (s.k[2] + 1));
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const float w0 = gd * wx[a] * wy[0], w1 = gd * wx[a] * wy[1];
            atomicAdd(q + a * sx, make_float4(w0 * wz[0], w0 * wz[1], w1 * wz[0], w1 * wz[1]));
        }
        return;
    }
    int xs[2], ys[2], zs[2];
    xs[0] = max(s.k[0], 0); xs[1] = min(s.k[0] + 1, p.ext[0] - 1);
    ys[0] = max(s.k[1], 0); ys[1] = min(s.k[1] + 1, p.ext[1] - 1);
    zs[0] = max(s.k[2], 0); zs[1] = min(s.k[2] + 1, p.ext[2] - 1);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const float wab = gd * wx[a] * wy[b];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float w = wab * wz[c];
                if (w != 0.0f) atomicAdd(p.gvol + texel(p, xs[a], ys[b], zs[c]), w);
            }
        }
}

// Sums v[0..7] over each group of lanes in `peers` (the lanes of the warp
// with the same key, from __match_any_sync) by a tree over the group's
// ranks; returns true on the group's lowest lane, which then holds the sums.
// All lanes of the warp call it.
__device__ __forceinline__ bool reduce_peers(unsigned peers, float v[8]) {
    const int lane = threadIdx.x & 31;
    int rank = __popc(peers & ((1u << lane) - 1u));
    unsigned above = lane == 31 ? 0u : peers & (0xffffffffu << (lane + 1));
    bool member = true;  // still holds a partial sum of its group
    while (__any_sync(0xffffffffu, member && above != 0u)) {
        const int next = (member && above) ? __ffs(above) - 1 : lane;
        const bool take = member && above != 0u && !(rank & 1);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float t = __shfl_sync(0xffffffffu, v[c], next);
            if (take) v[c] += t;
        }
        // the odd ranks have handed their sums down and leave
        const unsigned leaving = __ballot_sync(0xffffffffu, member && (rank & 1));
        if (member && (rank & 1)) member = false;
        above &= ~leaving;
        rank >>= 1;
    }
    return member;
}

// Adds the warp's voxel gradients (gd of each lane, 0 for none; the scene's own
// arrays as source) to the voxels.  All rays of a warp are at the same step, so neighbouring ones
// mostly add to the same 8 voxels: lanes with the same ones sum first, or
// their atomics queue up (36x47x28 voxels under a 91x634 image: 1395 -> 268 us).
// All lanes of the warp call it.
__device__ __forceinline__ void add_voxel_grads(const DiffParams &p, const Sample &s, float gd) {
    const bool adds = gd != 0.0f;
    if (!__any_sync(0xffffffffu, adds)) return;
    unsigned key = 0xffffffffu - (threadIdx.x & 31);  // no peers
    float v[8] = {};
    if (adds) {
        key = ((unsigned)(s.k[0] + 1) * (p.ext[1] + 1) + (s.k[1] + 1)) * (p.ext[2] + 1) + (s.k[2] + 1);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v[k] = gd * (k & 4 ? s.fx : 1.0f - s.fx) * (k & 2 ? s.fy : 1.0f - s.fy) * (k & 1 ? s.fz : 1.0f - s.fz);
    }
    if (reduce_peers(__match_any_sync(0xffffffffu, key), v) && adds) {
        const Corners c = corners(p, s);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (v[k] != 0.0f) atomicAdd(p.gvol + c.i[k], v[k]);
    }
}

// A warp's rays of one tile.  table: the warp's own LUT gradient (WARP_TABLE:
// entry j of the LUT at table[j + 1], its apron below and above, written
// without atomics: the lanes that write hold different entries), or the
// block's (channel-major floats, added to atomically); null without a LUT
// gradient.  The whole warp runs every step.
template <int SOURCE, bool WARP_TABLE>
__device__ __forceinline__ void backward_rays(const DiffParams &p, const MarchFrame &f, int px, int py,
                                              long long idx, const float4 *lut, float4 *table) {
    int nsteps = px < f.width && py < f.height ? p.steps[idx] : 0;
    float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f), out = g;
    float pos[3] = {}, d[3] = {};
    if (nsteps > 0) {
        g = p.gimage[idx];
        out = p.image[idx];
        if ((g.x == 0.0f && g.y == 0.0f && g.z == 0.0f && g.w == 0.0f) || !setup_ray(f, px, py, pos, d)) nsteps = 0;
    }
    const float t_end = __fadd_rn(1.0f, -out.w);
    const int most = __reduce_max_sync(0xffffffffu, nsteps);
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int i = 0; i < most; ++i) {
        float t[3];
        const bool sampled = tex_coords(f, pos, t) && i < nsteps;
        unsigned key = 0xffff0000u | threadIdx.x;  // no peers
        float v[8], gd = 0.0f;
        Sample s;
        if (sampled) {
            eval_sample<SOURCE>(p, f, t, lut, s);
            const float T = __fadd_rn(1.0f, -acc.w);
            composite(s, acc);
            const float om = 1.0f - s.alpha, inv = om > 0.0f ? rcp_newton(om) : 0.0f;
            const float cr = s.light * s.r, cg = s.light * s.g, cb = s.light * s.b;
            // T * (c - radiance behind) and T * (1 - alpha behind)
            const float br = (out.x - acc.x) * inv, bg = (out.y - acc.y) * inv, bb = (out.z - acc.z) * inv;
            const float ta = i == nsteps - 1 || !(om > 0.0f) ? T : t_end * inv;
            const float dalpha = g.x * (T * cr - br) + g.y * (T * cg - bg) + g.z * (T * cb - bb) + g.w * ta;
            const float kc = T * s.light * s.alpha;
            const float dr = g.x * kc, dg = g.y * kc, db = g.z * kc;
            const float da = dalpha * f.alpha_k * s.e;
            const float w1 = s.la, w0 = 1.0f - s.la;
            v[0] = w0 * dr; v[1] = w0 * dg; v[2] = w0 * db; v[3] = w0 * da;
            v[4] = w1 * dr; v[5] = w1 * dg; v[6] = w1 * db; v[7] = w1 * da;
            key = (unsigned)(s.j0 + 1);
            if (p.gvol) {
                gd = (dr * (s.B.x - s.A.x) + dg * (s.B.y - s.A.y) + db * (s.B.z - s.A.z) +
                      da * (s.B.w - s.A.w)) * f.flut_size * f.value_scale;
                if (is_packed(SOURCE) && gd != 0.0f) add_voxel_grad(p, s, gd);
            }
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = 0.0f;
        }
        if (!is_packed(SOURCE) && p.gvol) add_voxel_grads(p, s, gd);
#pragma unroll
        for (int a = 0; a < 3; ++a) pos[a] = __fadd_rn(pos[a], d[a]);
        if (table) {
            // neighbouring rays of a warp mostly address the same entries: the
            // lanes with the same entries sum their contributions first, and
            // one lane per entry adds them
            const unsigned peers = __match_any_sync(0xffffffffu, key);
            const bool leader = reduce_peers(peers, v) && key < 0xffff0000u;
            if (WARP_TABLE) {
                if (leader) {
                    float4 e = table[key];
                    e.x += v[0]; e.y += v[1]; e.z += v[2]; e.w += v[3];
                    table[key] = e;
                }
                __syncwarp();
                if (leader) {
                    float4 e = table[key + 1];
                    e.x += v[4]; e.y += v[5]; e.z += v[6]; e.w += v[7];
                    table[key + 1] = e;
                }
                __syncwarp();
            } else if (leader) {
                float *s_glut = reinterpret_cast<float *>(table);
                const int n = f.lut_size, i0 = max((int)key - 1, 0), i1 = min((int)key, n - 1);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (v[c] != 0.0f) atomicAdd(s_glut + c * n + i0, v[c]);
                    if (v[4 + c] != 0.0f) atomicAdd(s_glut + c * n + i1, v[4 + c]);
                }
            }
        }
    }
}

// Persistent blocks over the tiles.  Dynamic shared memory: (packed sources)
// the LUT and its apron, then (p.glut) the gradient tables: one of lut_size + 2
// entries per warp, or one channel-major table per block.
template <int SOURCE, bool WARP_TABLE>
__global__ void __launch_bounds__(kDiffThreads)
diff_backward_kernel(const __grid_constant__ DiffParams p) {
    extern __shared__ float4 s_dyn[];
    constexpr int kWarps = kDiffThreads / 32;
    const int size = p.f[0].lut_size, rows = size + 2;
    const float4 *lut = is_packed(SOURCE) ? stage_diff_lut(p, s_dyn) : p.lut;
    float4 *tables = is_packed(SOURCE) ? s_dyn + rows : s_dyn;
    if (p.glut)
        for (int k = threadIdx.x; k < (WARP_TABLE ? kWarps * rows : size); k += kDiffThreads)
            tables[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    float4 *table = !p.glut ? nullptr : WARP_TABLE ? tables + (threadIdx.x >> 5) * rows : tables;
    const int per_view = p.tiles_x * p.tiles_y;
    const int total = per_view * p.nviews;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
        const int view = tile / per_view;
        const MarchFrame &f = p.f[view];
        int px, py;
        pixel_of(tile % per_view, p.tiles_x, px, py);
        backward_rays<SOURCE, WARP_TABLE>(p, f, px, py, ((long long)view * f.height + py) * f.width + px, lut, table);
    }
    if (!p.glut) return;
    __syncthreads();
    float *g = reinterpret_cast<float *>(p.glut);  // (size, 4), entry-major
    const float *flat = reinterpret_cast<const float *>(tables);
    for (int k = threadIdx.x; k < 4 * size; k += kDiffThreads) {
        float sum = 0.0f;
        if (WARP_TABLE) {
            const int e = k >> 2, c = k & 3;
            for (int w = 0; w < kWarps; ++w) {
                const float *t = flat + 4 * w * rows + c;
                sum += t[4 * (e + 1)];
                if (e == 0) sum += t[0];
                if (e == size - 1) sum += t[4 * (size + 1)];
            }
        } else {
            sum = flat[(k & 3) * size + (k >> 2)];
        }
        if (sum != 0.0f) atomicAdd(g + k, sum);
    }
}

int build_params(const pvr_diff_scene *s, int v0, int nv, DiffParams &p) {
    std::memset(&p, 0, sizeof(p));
    p.vol = s->volume;
    p.nrm = s->normals;
    p.lut = reinterpret_cast<const float4 *>(s->lut);
    p.nviews = nv;
    p.tiles_x = (s->width + kDiffTile - 1) / kDiffTile;
    p.tiles_y = (s->height + kDiffTile - 1) / kDiffTile;
    p.ext[0] = s->w;
    p.ext[1] = s->h;
    p.ext[2] = s->d;
    float light_dir[3];
    light_direction(s->light_pos, s->light_target, light_dir);
    for (int k = 0; k < nv; ++k) {
        const pvr_diff_view &v = s->views[v0 + k];
        MarchFrame &f = p.f[k];
        double ip[16], iv[16];
        if (!invert_gl(v.proj, ip)) return fail(PVR_ERR_VALUE, "view %d: projection matrix is singular", v0 + k);
        if (!invert_gl(v.view, iv)) return fail(PVR_ERR_VALUE, "view %d: view matrix is singular", v0 + k);
        for (int i = 0; i < 8; ++i) f.ip[i] = (float)ip[i];
        for (int i = 0; i < 12; ++i) f.iv[i] = (float)iv[i];
        f.width = s->width;
        f.height = s->height;
        for (int a = 0; a < 3; ++a) {
            f.cam[a] = v.camera_pos[a];
            f.bmin[a] = s->min_bounds[a];
            f.bmax[a] = s->max_bounds[a];
            f.inv_ext[a] = 1.0f / (s->max_bounds[a] - s->min_bounds[a]);
            f.ext[a] = p.ext[a];
            f.fext[a] = (float)p.ext[a];
            f.nb[a] = 0;
            f.light_dir[a] = light_dir[a];
        }
        f.step = s->step_size;
        f.alpha_k = s->step_size / s->reference_step_size;
        f.max_steps = s->max_steps;
        f.ambient = s->ambient;
        f.diffuse = s->diffuse;
        f.value_scale = s->value_scale;
        f.lut_size = s->lut_size;
        f.flut_size = (float)s->lut_size;
        f.flut_max = (float)(s->lut_size - 1);
    }
    return PVR_OK;
}

int check_scene(const pvr_diff_scene *s) {
    if (!s) return fail(PVR_ERR_VALUE, "scene is NULL");
    if (!s->volume || !s->lut || !s->views) return fail(PVR_ERR_VALUE, "scene without volume, LUT or views");
    if (s->d < 1 || s->h < 1 || s->w < 1 || (long long)s->d * s->h * s->w > (1LL << 31) / 4)
        return fail(PVR_ERR_VALUE, "volume dims must be positive and under 2^29 voxels");
    if (s->lut_size < 1 || s->lut_size > kDiffMaxLut)
        return fail(PVR_ERR_VALUE, "LUT size must be in 1..%d, got %d", kDiffMaxLut, s->lut_size);
    if (s->width < 1 || s->height < 1 || s->width > 16384 || s->height > 16384)
        return fail(PVR_ERR_VALUE, "image size must be in 1..16384");
    if (s->n_views < 1 || s->n_views > 4096) return fail(PVR_ERR_VALUE, "n_views must be in 1..4096");
    if (!(s->step_size > 0.0f) || !std::isfinite(s->step_size) || !(s->reference_step_size > 0.0f) ||
        !std::isfinite(s->reference_step_size) || s->max_steps < 1)
        return fail(PVR_ERR_VALUE, "invalid step_size / reference_step_size / max_steps");
    for (int a = 0; a < 3; ++a)
        if (!(s->max_bounds[a] > s->min_bounds[a])) return fail(PVR_ERR_VALUE, "max_bounds must exceed min_bounds");
    return PVR_OK;
}

// Packing pays while a texel is read often enough: packing moves 44 bytes per
// texel (about 7 ps), the march saves about 0.2 ns per ray and more.
constexpr int kPackTexelsPerPixel = 16;

long long packed_bytes(const pvr_diff_scene *s, bool normals) {
    const int ext[3] = {s->w, s->h, s->d};
    const long long n = packed_texels(ext, normals);
    const long long pixels = (long long)s->width * s->height * s->n_views;
    if (n > (1LL << 30) || (long long)s->d * s->h * s->w > kPackTexelsPerPixel * pixels) return 0;
    return n * (long long)sizeof(float4);
}

int check_workspace(void *ws, long long bytes) {
    if (ws && (reinterpret_cast<uintptr_t>(ws) & 15)) return fail(PVR_ERR_VALUE, "workspace must be 16-byte aligned");
    if (bytes < 0) return fail(PVR_ERR_VALUE, "workspace bytes must be >= 0");
    return PVR_OK;
}

// Packs the scene's texels into the workspace where that pays and fits, and
// (volume_gradient) clears the gradient quads behind them: where the march
// then reads and adds.  clear_lut: a LUT gradient to clear as well, or null.
struct Packed {
    int source = kLinear;  // or kLinearNormals: set by pack_scene
    const float4 *texels = nullptr;
    float4 *gquads = nullptr;
};
cudaError_t pack_scene(const pvr_diff_scene *s, bool volume_gradient, float *clear_lut, void *ws, long long bytes,
                       cudaStream_t st, Packed &out) {
    const long long need = packed_bytes(s, s->normals != nullptr), more = packed_bytes(s, false);
    const int nglut = clear_lut ? 4 * s->lut_size : 0;
    out.source = s->normals ? kLinearNormals : kLinear;
    if (!ws || need == 0 || bytes < need)
        return nglut ? cudaMemsetAsync(clear_lut, 0, nglut * sizeof(float), st) : cudaSuccess;
    float4 *texels = static_cast<float4 *>(ws);
    const int total = (int)(need / (long long)sizeof(float4)), blocks = (total + 255) / 256;
    out.source = s->normals ? kPackedNormals : kPackedQuads;
    out.texels = texels;
    int nquads = 0;
    if (volume_gradient && bytes >= need + more) {
        out.gquads = texels + total;
        nquads = (int)(more / (long long)sizeof(float4));
    }
    if (s->normals)
        pack_kernel<kPackedNormals><<<blocks, 256, 0, st>>>(s->volume, s->normals, s->w, s->h, s->d, texels,
                                                            out.gquads, nquads, clear_lut, nglut);
    else
        pack_kernel<kPackedQuads><<<blocks, 256, 0, st>>>(s->volume, nullptr, s->w, s->h, s->d, texels, out.gquads,
                                                          nquads, clear_lut, nglut);
    return cudaGetLastError();
}

const void *forward_kernel(int source) {
    switch (source) {
    case kPackedNormals: return (const void *)diff_forward_kernel<kPackedNormals>;
    case kPackedQuads: return (const void *)diff_forward_kernel<kPackedQuads>;
    case kLinearNormals: return (const void *)diff_forward_kernel<kLinearNormals>;
    default: return (const void *)diff_forward_kernel<kLinear>;
    }
}

// Dynamic shared memory of the backward kernel: for packed sources the LUT and
// its apron, and with a LUT gradient as many entries per warp, or for the block.
int backward_smem(int source, int lut_size, bool lut_gradient) {
    const int tables = !lut_gradient ? 0 : lut_size <= kWarpTableLut ? kDiffThreads / 32 : 1;
    return (lut_size + 2) * (int)sizeof(float4) * ((is_packed(source) ? 1 : 0) + tables);
}

template <bool WARP_TABLE>
const void *backward_kernel(int source) {
    switch (source) {
    case kPackedNormals: return (const void *)diff_backward_kernel<kPackedNormals, WARP_TABLE>;
    case kPackedQuads: return (const void *)diff_backward_kernel<kPackedQuads, WARP_TABLE>;
    case kLinearNormals: return (const void *)diff_backward_kernel<kLinearNormals, WARP_TABLE>;
    default: return (const void *)diff_backward_kernel<kLinear, WARP_TABLE>;
    }
}

}  // namespace
}  // namespace pvr

using pvr::fail;

extern "C" int pvr_diff_workspace(const pvr_diff_scene *s, long long *bytes, long long *bytes_volume_gradient) {
    if (!bytes || !bytes_volume_gradient) return fail(PVR_ERR_VALUE, "bytes is NULL");
    *bytes = *bytes_volume_gradient = 0;
    if (int rc = pvr::check_scene(s)) return rc;
    *bytes = pvr::packed_bytes(s, s->normals != nullptr);
    *bytes_volume_gradient = *bytes > 0 ? *bytes + pvr::packed_bytes(s, false) : 0;
    return PVR_OK;
}

extern "C" int pvr_diff_forward_ws(const pvr_diff_scene *s, float *d_image, int *d_steps, void *workspace,
                                   long long workspace_bytes, void *stream) {
    if (int rc = pvr::check_scene(s)) return rc;
    if (!d_image || !d_steps) return fail(PVR_ERR_VALUE, "image / steps buffer is NULL");
    if (int rc = pvr::check_workspace(workspace, workspace_bytes)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const long long frame = (long long)s->width * s->height;
    pvr::Packed packed;
    for (int v0 = 0; v0 < s->n_views; v0 += pvr::kDiffMaxViews) {
        const int nv = std::min(pvr::kDiffMaxViews, s->n_views - v0);
        pvr::DiffParams p;
        if (int rc = pvr::build_params(s, v0, nv, p)) return rc;
        if (v0 == 0) PVR_CUDA(pvr::pack_scene(s, false, nullptr, workspace, workspace_bytes, st, packed));
        p.texels = packed.texels;
        p.image = reinterpret_cast<float4 *>(d_image) + v0 * frame;
        p.steps = d_steps + v0 * frame;
        const int blocks = p.tiles_x * p.tiles_y * nv;
        void *args[] = {&p};
        PVR_CUDA(cudaLaunchKernel(pvr::forward_kernel(packed.source), dim3(blocks), dim3(pvr::kDiffThreads), args,
                                  pvr::is_packed(packed.source) ? (size_t)(s->lut_size + 2) * sizeof(float4) : 0, st));
    }
    return PVR_OK;
}

extern "C" int pvr_diff_forward(const pvr_diff_scene *s, float *d_image, int *d_steps, void *stream) {
    return pvr_diff_forward_ws(s, d_image, d_steps, nullptr, 0, stream);
}

extern "C" int pvr_diff_backward_ws(const pvr_diff_scene *s, const float *d_image, const int *d_steps,
                                    const float *d_grad_image, float *d_grad_lut, float *d_grad_volume, int overwrite,
                                    void *workspace, long long workspace_bytes, void *stream) {
    if (int rc = pvr::check_scene(s)) return rc;
    if (!d_image || !d_steps || !d_grad_image) return fail(PVR_ERR_VALUE, "image / steps / gradient buffer is NULL");
    if (int rc = pvr::check_workspace(workspace, workspace_bytes)) return rc;
    if (!d_grad_lut && !d_grad_volume) return PVR_OK;
    cudaStream_t st = (cudaStream_t)stream;
    int device = 0, sms = 0;
    PVR_CUDA(cudaGetDevice(&device));
    PVR_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const bool warp_table = s->lut_size <= pvr::kWarpTableLut;
    int per_sm = 0, smem = 0;
    pvr::Packed packed;
    const void *kernel = nullptr;
    const long long frame = (long long)s->width * s->height;
    for (int v0 = 0; v0 < s->n_views; v0 += pvr::kDiffMaxViews) {
        const int nv = std::min(pvr::kDiffMaxViews, s->n_views - v0);
        pvr::DiffParams p;
        if (int rc = pvr::build_params(s, v0, nv, p)) return rc;
        if (v0 == 0) {
            PVR_CUDA(pvr::pack_scene(s, d_grad_volume != nullptr, overwrite ? d_grad_lut : nullptr, workspace,
                                     workspace_bytes, st, packed));
            if (overwrite && d_grad_volume && !packed.gquads)
                PVR_CUDA(cudaMemsetAsync(d_grad_volume, 0, (size_t)s->d * s->h * s->w * sizeof(float), st));
            kernel = warp_table ? pvr::backward_kernel<true>(packed.source) : pvr::backward_kernel<false>(packed.source);
            smem = pvr::backward_smem(packed.source, s->lut_size, d_grad_lut != nullptr);
            // more than 48 KB of dynamic shared memory: the limit belongs to the
            // kernel on the current device, not to this call, so every call sets
            // the most that any table takes (a smaller limit would refuse the
            // launch of another thread's larger table)
            if (smem > 48 * 1024)
                PVR_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              pvr::backward_smem(packed.source, warp_table ? pvr::kWarpTableLut : pvr::kDiffMaxLut, true)));
            PVR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, pvr::kDiffThreads, smem));
            per_sm = std::max(1, per_sm);
        }
        p.texels = packed.texels;
        p.image = const_cast<float4 *>(reinterpret_cast<const float4 *>(d_image)) + v0 * frame;
        p.steps = const_cast<int *>(d_steps) + v0 * frame;
        p.gimage = reinterpret_cast<const float4 *>(d_grad_image) + v0 * frame;
        p.glut = reinterpret_cast<float4 *>(d_grad_lut);
        p.gvol = d_grad_volume;
        p.gquads = packed.gquads;
        const int tiles = p.tiles_x * p.tiles_y * nv;
        const int blocks = std::min(tiles, sms * per_sm);
        void *args[] = {&p};
        PVR_CUDA(cudaLaunchKernel(kernel, dim3(blocks), dim3(pvr::kDiffThreads), args, smem, st));
    }
    if (packed.gquads) {
        const int voxels = s->d * s->h * s->w;
        pvr::unpack_grad_kernel<<<(voxels + 255) / 256, 256, 0, st>>>(packed.gquads, s->w, s->h, s->d, overwrite != 0,
                                                                        d_grad_volume);
        PVR_CUDA(cudaGetLastError());
    }
    return PVR_OK;
}

extern "C" int pvr_diff_backward(const pvr_diff_scene *s, const float *d_image, const int *d_steps,
                                 const float *d_grad_image, float *d_grad_lut, float *d_grad_volume,
                                 void *stream) {
    return pvr_diff_backward_ws(s, d_image, d_steps, d_grad_image, d_grad_lut, d_grad_volume, 0, nullptr, 0, stream);
}
