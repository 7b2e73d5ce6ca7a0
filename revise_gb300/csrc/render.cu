// Block ray casting for sm_103a.
//
// Restates renderKernel<FieldMode::Argb> + renderArgb of the reference
// (src/s3dmm_cuda/DenseFieldRenderer_cu.cu:62-215, src/s3dmm_cuda/renderArgb.hpp:30-55,
// cuda_blend.hpp:24-44, cuda_argb_transform.hpp:26-43) without texture
// hardware: bricks are linear arrays in HBM read through the read-only path,
// filtered in FP32 by software trilinear interpolation with clamp addressing
// (a sample whose 8 texels hold a NaN is skipped, as the texture unit's
// weighted sum would be NaN); the transfer function sits in shared memory.
//
// Ray set-up (per-pixel ray, per-block slab test, sample count and positions)
// is written with explicitly rounded operations (__fadd_rn, __fmul_rn, ...)
// so that it cannot be contracted and the CPU oracle reproduces the same
// sample positions bit for bit.  The sample loop keeps the reference's
// indexing: sample k = i-1 for i = 1 .. sampleCount-1, at entry + k*step,
// computed directly (fma) rather than by accumulation.
//
// Kernels:
//   render_block_mode_kernel  one block into an ARGB8 viewport (drop-in form):
//                             reference non-premultiplied blending, ARGB8
//                             read-modify-write per block, any field mode;
//   part_blocks_kernel        all the blocks of a worker's part at once, with
//                             part_composite_kernel the same pixels;
//   frame_render_kernel       batched form: each ray walks the block grid front
//                             to back (3D DDA), marches every block it enters
//                             exactly as above, composites block results with
//                             the over operator in FP32 (premultiplied), and
//                             stops once alpha passes view.alpha_stop;
//   frame_backward_kernel     adjoint of frame_render_kernel w.r.t. the
//                             transfer function and the dense values; re-walks
//                             each ray instead of storing samples.
#include "s3r_internal.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

namespace s3r {
namespace {

constexpr float kAlphaThreshold = 0.996f; // renderArgb.hpp:47
constexpr float kTopHalf = 5.f;           // DenseFieldRenderer_cu.cu:339

struct BlockRay {
    float tau_enter;
    float tau_exit;
    int samples;
    float p0[3];
    float step[3];
    float origin[3];
    float factor;
    uint32_t n;     // vertices per axis, 2^depth+1
    uint32_t pitch; // row pitch of the brick in elements (>= n)
};

// A brick's extent and row pitch: vertex (x, y, z) is element (z n + y) pitch + x.
struct Dim {
    uint32_t n, pitch;
};
__device__ __forceinline__ Dim dim_of(const BlockRay& r) { return Dim{r.n, r.pitch}; }

// a / b correctly rounded from y = 1 / b correctly rounded (Markstein's quotient: one product, its exact
// residual, one correction), for b and a / b well inside the normal range: three fused operations where the
// divisor serves many quotients, against a division's reciprocal, refinement and range test each time.
__device__ __forceinline__ float div_by(float a, float b, float y)
{
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
}

// floor(x) of |x| < 2^22 and the integer, by one addition rounded down that leaves the integer in the low
// mantissa bits: the conversion unit, which float-to-integer, floor and the exponentials of a sample share,
// runs at a fraction of the adders' rate.
__device__ __forceinline__ float floor_small(float x, int& i)
{
    const float r = __fadd_rd(x, 12582912.f); // 1.5 * 2^23
    i = __float_as_int(r) - 0x4b400000;
    return __fsub_rn(r, 12582912.f);
}

__device__ __forceinline__ void pixel_ray(const s3r_view& v, uint32_t vx, uint32_t vy, float org[3], float dir[3])
{
    const float x = __fmul_rn(__fadd_rn(-0.5f, __fdiv_rn(__fadd_rn((float)vx, 0.5f), (float)v.W)), v.cam.w);
    const float y = __fmul_rn(__fadd_rn(-0.5f, __fdiv_rn(__fadd_rn((float)vy, 0.5f), (float)v.H)), v.cam.h);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float ex = __fmul_rn(v.cam.e1[d], x);
        const float ey = __fmul_rn(v.cam.e2[d], y);
        if (v.cam.ortho) {
            org[d] = __fadd_rn(__fadd_rn(v.cam.eye[d], ex), ey);
            dir[d] = v.cam.n[d];
        } else {
            org[d] = v.cam.eye[d];
            dir[d] = __fadd_rn(__fadd_rn(v.cam.n[d], ex), ey);
        }
    }
}

// 1 / dir per axis for block_ray and walk_blocks; an axis the ray hardly moves along is never divided by.
__device__ __forceinline__ void ray_inverse(const float dir[3], float inv[3])
{
#pragma unroll
    for (int d = 0; d < 3; ++d) inv[d] = __frcp_rn(dir[d]);
}

// Slab test and sample set-up (DenseFieldRenderer_cu.cu:81-181). Returns true
// when the block is rendered for this ray.
__device__ __forceinline__ bool block_ray(const s3r_view& v, const float org[3], const float dir[3],
                                          const float inv[3], const RenderBlock& rb, BlockRay& r)
{
    const float* c = rb.center;
    const float h = rb.half;
    float te = 1.f, tx = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (!(fabsf(dir[a]) > 1e-10f)) continue;
        const int b1 = a == 0 ? 1 : 0;
        const int b2 = a == 2 ? 1 : 2;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const float face = side ? __fadd_rn(c[a], h) : __fsub_rn(c[a], h);
            const float tau = div_by(__fsub_rn(face, org[a]), dir[a], inv[a]);
            const float p1 = __fadd_rn(org[b1], __fmul_rn(dir[b1], tau));
            const float p2 = __fadd_rn(org[b2], __fmul_rn(dir[b2], tau));
            if (fabsf(__fsub_rn(p1, c[b1])) <= h && fabsf(__fsub_rn(p2, c[b2])) <= h) {
                const bool enter = (dir[a] > 0.f) == (side == 0);
                if (enter) te = tau;
                else tx = tau;
            }
        }
    }
    if (te < 1.f) te = 1.f;
    r.tau_enter = te;
    r.tau_exit = tx;
    if (!(tx > te)) return false;
    const uint32_t n = (1u << rb.depth) + 1u;
    const float texel = rb.texel;
    const float span = __fsub_rn(tx, te);
    const float dotr = __fadd_rn(__fadd_rn(__fmul_rn(dir[0], dir[0]), __fmul_rn(dir[1], dir[1])),
                                 __fmul_rn(dir[2], dir[2]));
    const float l1 = __fadd_rn(__fadd_rn(fabsf(dir[0]), fabsf(dir[1])), fabsf(dir[2]));
    const float num = __fmul_rn(__fmul_rn(v.quality, span), dotr);
    const float den = __fmul_rn(texel, l1);
    const int s = __float2int_rz(__fdiv_rn(num, den));
    const float dtau = __fdiv_rn(span, (float)s);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        r.step[d] = __fmul_rn(dir[d], dtau);
        r.p0[d] = __fadd_rn(org[d], __fmul_rn(dir[d], te));
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) r.origin[d] = rb.origin[d];
    r.factor = rb.factor;
    r.n = n;
    r.pitch = rb.pitch ? rb.pitch : n;
    r.samples = s;
    return true;
}

// A texel of a brick of format Fmt, decoded to float.
template <int Fmt> struct Brick;
template <> struct Brick<S3R_BRICK_F32> {
    __device__ static float get(const void* b, uint64_t i) { return __ldg(reinterpret_cast<const float*>(b) + i); }
};
template <> struct Brick<S3R_BRICK_F16> {
    __device__ static float get(const void* b, uint64_t i)
    {
        return __half2float(__ldg(reinterpret_cast<const __half*>(b) + i));
    }
};
template <> struct Brick<S3R_BRICK_BF16> {
    __device__ static float get(const void* b, uint64_t i)
    {
        return __bfloat162float(__ldg(reinterpret_cast<const __nv_bfloat16*>(b) + i));
    }
};

// ---------------------------------------------------------------- texture-unit filtering
//
// S3R_FILTER_TEXTURE: the linear filtering the GPU texture unit applies to the
// reference's clamped float textures (measured on this GPU with one-hot
// textures over a lattice of coordinates).  Per axis xb = coordinate - 0.5,
// texels floor(xb) and floor(xb)+1 (clamped), fraction a = floor(frac * 256 +
// 1/2) in 0..256.  1D: weights (256 - a, a) / 256.  3D: the z split is exact
// (zt = 256 - c | c); in each z half xh = rn(a * zt), xl = zt - xh; the y split
// rounds the y-high part under xh (rn(xh * b)) and the y-low part under xl
// (rn(xl * (256 - b))), the rest going to the other side, rn(p) = (p + 128) >> 8.
// A NaN texel makes the sample NaN when its per-axis factors are all nonzero.

struct TexAxis {
    uint32_t i0, i1;
    int32_t a; // 0..256
};

__device__ __forceinline__ TexAxis tex_axis(float tc, int hi)
{
    const float xb = __fsub_rn(tc, 0.5f);
    // xb * 256 is exact, so the one rounding of the fma cannot carry floor() past an integer
    const float q = floorf(__fmaf_rn(xb, 256.f, 0.5f));
    const float fl = floorf(__fmul_rn(q, 0.00390625f));
    TexAxis t;
    t.a = (int32_t)__fmaf_rn(fl, -256.f, q);
    const int lo = (int)fmaxf(fminf(fl, 1e9f), -1e9f);
    t.i0 = (uint32_t)min(max(lo, 0), hi);
    t.i1 = (uint32_t)min(max(lo + 1, 0), hi);
    return t;
}

__device__ __forceinline__ int32_t rn8(int32_t x, int32_t y) { return (x * y + 128) >> 8; }

// Texel coordinate of sample k along axis d (the fetch coordinate of the reference).
__device__ __forceinline__ float sample_tc(const BlockRay& r, int k, int d)
{
    const float p = __fmaf_rn(r.step[d], (float)k, r.p0[d]);
    return __fmul_rn(__fsub_rn(p, r.origin[d]), r.factor);
}

template <int Fmt> struct Brick;

template <int Fmt>
__device__ __forceinline__ bool tex_trilinear_at(const void* brick, Dim g, float tcx, float tcy, float tcz,
                                                 float& val)
{
    const int hi = (int)g.n - 1;
    const TexAxis x = tex_axis(tcx, hi);
    const TexAxis y = tex_axis(tcy, hi);
    const TexAxis z = tex_axis(tcz, hi);
    int32_t w[8];
#pragma unroll
    for (int hz = 0; hz < 2; ++hz) {
        const int32_t zt = hz ? z.a : 256 - z.a;
        const int32_t xh = rn8(x.a, zt), xl = zt - xh;
        const int32_t yhh = rn8(xh, y.a), yll = rn8(xl, 256 - y.a);
        w[3 | (hz << 2)] = yhh;
        w[1 | (hz << 2)] = xh - yhh;
        w[hz << 2] = yll;
        w[2 | (hz << 2)] = xl - yll;
    }
    const uint64_t n64 = g.n, p64 = g.pitch;
    float t[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const uint64_t xi = (q & 1) ? x.i1 : x.i0;
        const uint64_t yi = (q & 2) ? y.i1 : y.i0;
        const uint64_t zi = (q & 4) ? z.i1 : z.i0;
        t[q] = Brick<Fmt>::get(brick, (zi * n64 + yi) * p64 + xi);
    }
    // per-axis factor nonzero: the low texel needs a < 256, the high one a > 0
    const bool lx = x.a < 256, hx = x.a > 0, ly = y.a < 256, hy = y.a > 0, lz = z.a < 256, hz = z.a > 0;
    bool bad = false;
    float acc = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const bool inx = (q & 1) ? hx : lx, iny = (q & 2) ? hy : ly, inz = (q & 4) ? hz : lz;
        if (isnan(t[q])) bad |= inx && iny && inz;
        else acc = __fmaf_rn((float)w[q], t[q], acc);
    }
    if (bad) return false;
    val = __fmul_rn(acc, 0.00390625f);
    return true;
}

template <int Fmt>
__device__ __forceinline__ bool tex_trilinear(const void* brick, const BlockRay& r, int k, float& val)
{
    return tex_trilinear_at<Fmt>(brick, dim_of(r), sample_tc(r, k, 0), sample_tc(r, k, 1), sample_tc(r, k, 2), val);
}

__device__ __forceinline__ float4 tex_tf_lookup(const float4* tf, uint32_t tfn, float v01)
{
    const TexAxis u = tex_axis(__fmul_rn(v01, (float)tfn), (int)tfn - 1);
    const float4 p = tf[u.i0], q = tf[u.i1];
    const float wl = (float)(256 - u.a), wh = (float)u.a;
    float4 c;
    c.x = __fmul_rn(__fmaf_rn(wh, q.x, __fmul_rn(wl, p.x)), 0.00390625f);
    c.y = __fmul_rn(__fmaf_rn(wh, q.y, __fmul_rn(wl, p.y)), 0.00390625f);
    c.z = __fmul_rn(__fmaf_rn(wh, q.z, __fmul_rn(wl, p.z)), 0.00390625f);
    c.w = __fmul_rn(__fmaf_rn(wh, q.w, __fmul_rn(wl, p.w)), 0.00390625f);
    return c;
}

// The transfer function in shared memory as the kernels look it up: P holds tf_n + 2 entries, the table with its first
// and last entry repeated, so that a lookup is one index and two 16-byte loads, without clamping two indices.  Shared
// memory is taken from the L1, which the texels need: kernels whose CTAs fill an SM two at a time also keep D, the
// differences P[j+1] - P[j] (tables of up to kTfDiff entries), the others form them at the lookup.  (8 CTAs with 1000
// entries and their differences each left no L1: 606 -> 1197 us for level 3, depths 3-7, at 1920x1080.)
constexpr uint32_t kTfDiff = 1024;
struct TfTable {
    const float4* p;
    const float4* d; // nullptr: the difference is formed at the lookup
    __device__ const float4* raw() const { return p + 1; }
};
inline __host__ __device__ uint32_t tf_smem_entries(uint32_t tf_n, bool diff)
{
    return diff && tf_n <= kTfDiff ? 2 * tf_n + 3 : tf_n + 2;
}

// All threads of the CTA; ends with a barrier.
template <bool kDiff>
__device__ __forceinline__ TfTable load_tf(float4* sm, const float* tf, uint32_t tf_n, uint32_t tid, uint32_t nthreads)
{
    const float4* g = reinterpret_cast<const float4*>(tf);
    const bool diff = kDiff && tf_n <= kTfDiff;
    for (uint32_t j = tid; j < tf_n + 2; j += nthreads) {
        const float4 a = g[min(max((int)j - 1, 0), (int)tf_n - 1)];
        sm[j] = a;
        if (diff && j <= tf_n) {
            const float4 b = g[min(j, tf_n - 1)];
            sm[tf_n + 2 + j] = make_float4(b.x - a.x, b.y - a.y, b.z - a.z, b.w - a.w);
        }
    }
    __syncthreads();
    return TfTable{sm, diff ? sm + tf_n + 2 : nullptr};
}

// The colour from the padded table: entry j = floor(u) + 1 within [0, tf_n] gives the clamped pair;
// beyond the table the pair is one entry twice, so any finite fraction gives that entry.
__device__ __forceinline__ float4 tf_colour(const TfTable& tf, uint32_t tfn, float v01)
{
    const float u = __fmaf_rn(v01, (float)tfn, -0.5f);
    int j;
    const float fl = floor_small(fminf(fmaxf(u, -1.f), (float)tfn - 0.5f), j);
    const float f = u - fl;
    const float4 p = tf.p[j + 1];
    float4 d;
    if (tf.d) {
        d = tf.d[j + 1];
    } else {
        const float4 q = tf.p[j + 2];
        d = make_float4(q.x - p.x, q.y - p.y, q.z - p.z, q.w - p.w);
    }
    return make_float4(__fmaf_rn(f, d.x, p.x), __fmaf_rn(f, d.y, p.y), __fmaf_rn(f, d.z, p.z), __fmaf_rn(f, d.w, p.w));
}

// The relative value (val - field_min) / span, correctly rounded: by the kept reciprocal where span is far
// from the ends of the float range, else by a division.
struct Relative {
    float lo, span, y;
    bool fast;
    __device__ __forceinline__ float operator()(float val) const
    {
        const float a = __fsub_rn(val, lo);
        return fast ? div_by(a, span, y) : __fdiv_rn(a, span);
    }
    // The texture unit's rule clamps the lookup of an infinite relative value to the table's end, which the kept
    // reciprocal's residual would make a NaN.  (The exact filter's fraction of an infinite value is a NaN either way.)
    __device__ __forceinline__ float clamped(float val) const
    {
        const float q = (*this)(val);
        return fabsf(q) <= 3.402823466e38f ? q : __fdiv_rn(__fsub_rn(val, lo), span);
    }
};
__device__ __forceinline__ Relative relative_of(const s3r_view& v)
{
    const float span = v.field_max - v.field_min;
    return Relative{v.field_min, span, __frcp_rn(span), span > 1e-18f && span < 1e18f};
}

// Whether one of 8 values is NaN, two values per comparison.
__device__ __forceinline__ bool any_nan(const float t[8])
{
    uint32_t bad;
    asm("{\n\t.reg .pred p;\n\t"
        "setp.nan.f32 p, %1, %2;\n\t"
        "setp.nan.or.f32 p, %3, %4, p;\n\t"
        "setp.nan.or.f32 p, %5, %6, p;\n\t"
        "setp.nan.or.f32 p, %7, %8, p;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(bad)
        : "f"(t[0]), "f"(t[1]), "f"(t[2]), "f"(t[3]), "f"(t[4]), "f"(t[5]), "f"(t[6]), "f"(t[7]));
    return bad != 0;
}

__device__ __forceinline__ float layer_exponent(uint32_t depth, uint32_t level, float quality)
{
    return __fmul_rn(__fdiv_rn(1.f, __fmul_rn((float)(1u << (depth + level)), quality)), 100.f);
}

__device__ __forceinline__ float4 argb_to_rgba(uint32_t p)
{
    constexpr float y = 1.f / 255.f;
    return make_float4(div_by((float)((p >> 16) & 0xffu), 255.f, y), div_by((float)((p >> 8) & 0xffu), 255.f, y),
                       div_by((float)(p & 0xffu), 255.f, y), div_by((float)((p >> 24) & 0xffu), 255.f, y));
}

__device__ __forceinline__ uint32_t rgba_to_argb(float4 c)
{
    return ((uint32_t)(c.w * 255.999f) << 24) + ((uint32_t)(c.x * 255.999f) << 16) +
           ((uint32_t)(c.y * 255.999f) << 8) + (uint32_t)(c.z * 255.999f);
}

// ---------------------------------------------------------------- field modes (plain form)
//
// renderKernel<mode> with the reference's render functions (render*.hpp) and
// lighting (cuda_lighting.hpp), on the plain form's ray set-up and sampling.

// Trilinear value of 8 texels (x fastest, then y, then z) at the cell's fractions.
__device__ __forceinline__ float lerp_cell(const float t[8], const float f[3])
{
    const float x00 = __fmaf_rn(f[0], t[1] - t[0], t[0]);
    const float x10 = __fmaf_rn(f[0], t[3] - t[2], t[2]);
    const float x01 = __fmaf_rn(f[0], t[5] - t[4], t[4]);
    const float x11 = __fmaf_rn(f[0], t[7] - t[6], t[6]);
    const float y0 = __fmaf_rn(f[1], x10 - x00, x00);
    const float y1 = __fmaf_rn(f[1], x11 - x01, x01);
    return __fmaf_rn(f[2], y1 - y0, y0);
}

// The 8 texels and fractions of the exact filter at a texel coordinate -- the reference's fetch coordinate: loads
// issued by fetch_cell, value (NaN where one texel is NaN) by cell_value.
struct FieldCell {
    float t[8], f[3];
};
__device__ __forceinline__ void fetch_cell(const float* brick, Dim n, float x, float y, float z, FieldCell& c)
{
    const uint32_t hi = n.n - 1;
    const float tc[3] = {x, y, z};
    int a[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float xb = __fsub_rn(tc[d], 0.5f);
        c.f[d] = __fsub_rn(xb, floor_small(xb, a[d]));
    }
    if ((uint32_t)a[0] < hi && (uint32_t)a[1] < hi && (uint32_t)a[2] < hi) {
        // the cell lies in the brick: four pairs in four rows (32-bit offsets: a brick holds at most 513^3)
        const uint32_t o = ((uint32_t)a[2] * n.n + (uint32_t)a[1]) * n.pitch + (uint32_t)a[0];
        const uint32_t dz = n.n * n.pitch;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            c.t[q] = __ldg(brick + (uint64_t)(o + ((q & 2) ? n.pitch : 0u) + ((q & 4) ? dz : 0u)) + (q & 1));
    } else {
        uint32_t i0[3], i1[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            i0[d] = (uint32_t)min(max(a[d], 0), (int)hi);
            i1[d] = (uint32_t)min(max(a[d], -1) + 1, (int)hi);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
            c.t[q] = __ldg(brick + ((((q & 4) ? i1[2] : i0[2]) * n.n + ((q & 2) ? i1[1] : i0[1])) * n.pitch +
                                  ((q & 1) ? i1[0] : i0[0])));
    }
}
__device__ __forceinline__ float cell_value(const FieldCell& c)
{
    return any_nan(c.t) ? __int_as_float(0x7fc00000) : lerp_cell(c.t, c.f);
}

template <bool kTex> __device__ __forceinline__ float4 tf_rgba(const TfTable& tf, uint32_t tfn, float v01)
{
    if constexpr (kTex) return tex_tf_lookup(tf.raw(), tfn, v01);
    else return tf_colour(tf, tfn, v01);
}

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 f3(const float* p) { return F3{p[0], p[1], p[2]}; }
__device__ __forceinline__ F3 operator+(F3 a, F3 b) { return F3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return F3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 operator*(F3 a, float s) { return F3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ F3 operator*(F3 a, F3 b) { return F3{a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ float dot3(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ F3 normalize3(F3 a) { return a * (1.f / sqrtf(dot3(a, a))); }
__device__ __forceinline__ float clamp01(float x) { return fmaxf(0.f, fminf(1.f, x)); }

// x^100 in double by squaring (x^64 x^32 x^4): eight multiplications, whose
// few-ulp double error almost never reaches the float the result is rounded to;
// a general double pow costs several times that on this GPU's FP64 units.
__device__ __forceinline__ double pow100(double x)
{
    const double x2 = x * x, x4 = x2 * x2, x8 = x4 * x4, x16 = x8 * x8, x32 = x16 * x16, x64 = x32 * x32;
    return x64 * x32 * x4;
}

// Blinn-Phong term of one light (cuda_lighting.hpp:26-50): material ambient 1,
// diffuse = the transfer-function colour, specular 0.5, shininess 100; the
// reference's max(., 0.0) and pow promote to double (the max is exact in float,
// the power is formed in double as above).
__device__ __forceinline__ F3 blinn(F3 N, F3 V, F3 L, const s3r_light& light, F3 kd)
{
    const float diff = fmaxf(dot3(L, N), 0.f);
    const F3 H = normalize3(L + V);
    const float spec = diff > 0.f ? (float)pow100(fmax((double)dot3(H, N), 0.0)) : 0.f;
    return f3(light.ambient) + kd * f3(light.diffuse) * diff + F3{0.5f, 0.5f, 0.5f} * f3(light.specular) * spec;
}

// Where a field-mode march takes its samples from: fetch starts a sample's loads at a texel coordinate (from the
// second field's brick, or the first's), value gives its field value, NaN outside the domain.
//   BrickSampler<kTex>: linear bricks in HBM, filtered in software (kTex: the
//     texture unit's rule, else exact trilinear); the table in shared memory.
//   TextureSampler: the GPU's texture unit itself, as the reference samples --
//     tex3D on a 3-D float array (unnormalized coordinates, linear filtering,
//     clamp) and tex1D on the transfer-function array (normalized, linear,
//     clamp).
// kStepwise: sample positions accumulated step by step from the entry point
// (pos += step), as the reference forms them, because texture filtering's
// 8-bit fractions are sensitive to the last ulp of a position; else entry +
// k * step (one fma), as the oracle and the batched path form them.
// kContracted: the crossing positions of the isosurface modes written as the
// reference writes them (pos + step * t, which nvcc fuses into one fma), else
// rounded twice as the oracle rounds them.
// kTexRule: filtered as the texture unit does, the transfer function too.
// kAhead: sample k + 1 is fetched before sample k is used.  The texture unit's
// rule in software filters in its fetch, and a sample ahead only costs it
// registers (lit volume, 64 blocks of depth 6: 10.0 against 11.0 ms).
template <bool kTex> struct BrickSampler {
    const float* b1;
    const float* b2;
    Dim n;
    TfTable tf;
    uint32_t tfn;
    static constexpr bool kStepwise = kTex, kTexRule = kTex, kContracted = false, kAhead = !kTex;
    using Sample = std::conditional_t<kTex, float, FieldCell>;
    __device__ void fetch(int second, F3 p, Sample& x) const
    {
        if constexpr (!kTex) fetch_cell(second ? b2 : b1, n, p.x, p.y, p.z, x);
        else if (!tex_trilinear_at<S3R_BRICK_F32>(second ? b2 : b1, n, p.x, p.y, p.z, x)) x = __int_as_float(0x7fc00000);
    }
    static __device__ float value(const Sample& x)
    {
        if constexpr (kTex) return x;
        else return cell_value(x);
    }
    __device__ float4 colour(float v01) const { return tf_rgba<kTex>(tf, tfn, v01); }
};

struct TextureSampler {
    cudaTextureObject_t t1, t2, tf;
    static constexpr bool kStepwise = true, kTexRule = true, kContracted = true, kAhead = true;
    using Sample = float;
    __device__ void fetch(int second, F3 p, Sample& x) const { x = tex3D<float>(second ? t2 : t1, p.x, p.y, p.z); }
    static __device__ float value(const Sample& x) { return x; }
    __device__ float4 colour(float v01) const { return tex1D<float4>(tf, v01); }
};

// computeFragColor (cuda_lighting.hpp:52-95): normal from central differences
// of the field at +-0.1 texel, double-sided lighting, colour clamped to [0, 1].
template <class S>
__device__ __forceinline__ float4 frag_color(const S& smp, float4 diffuse, F3 eye, F3 surf, F3 tc,
                                             const s3r_presentation& pr)
{
    constexpr float d = 0.1f;
    auto field = [&](float x, float y, float z) {
        typename S::Sample c;
        smp.fetch(0, F3{x, y, z}, c);
        return S::value(c);
    };
    const F3 a{field(tc.x - d, tc.y, tc.z), field(tc.x, tc.y - d, tc.z), field(tc.x, tc.y, tc.z - d)};
    const F3 b{field(tc.x + d, tc.y, tc.z), field(tc.x, tc.y + d, tc.z), field(tc.x, tc.y, tc.z + d)};
    F3 N = normalize3(a - b);
    const F3 V = normalize3(eye - surf);
    F3 c{0.f, 0.f, 0.f};
    const F3 kd{diffuse.x, diffuse.y, diffuse.z};
    for (uint32_t i = 0; i < pr.light_count; ++i) {
        const F3 L = normalize3(f3(pr.lights[i].pos) - surf);
        if (dot3(L, N) < 0.f) N = F3{-N.x, -N.y, -N.z};
        c = c + blinn(N, V, L, pr.lights[i], kd);
    }
    return make_float4(clamp01(c.x), clamp01(c.y), clamp01(c.z), diffuse.w);
}

// blendBehind / blendAbove (cuda_blend.hpp:24-44), non-premultiplied
__device__ __forceinline__ void blend_behind(float4& acc, float4 col)
{
    const float da = col.w * (1.f - acc.w);
    const float a = acc.w + da;
    if (a > 0.f) {
        // both quotients by one reciprocal; an alpha too small for its reciprocal is divided by
        float ka, kd;
        if (a > 1e-30f) {
            const float y = __frcp_rn(a);
            ka = div_by(acc.w, a, y);
            kd = div_by(da, a, y);
        } else {
            ka = acc.w / a;
            kd = da / a;
        }
        acc.x = acc.x * ka + col.x * kd;
        acc.y = acc.y * ka + col.y * kd;
        acc.z = acc.z * ka + col.z * kd;
    }
    acc.w = a;
}

__device__ __forceinline__ uint32_t blend_above_argb(uint32_t pix, float4 acc)
{
    float4 ex = argb_to_rgba(pix);
    const float da = ex.w * (1.f - acc.w);
    const float a = acc.w + da;
    if (a > 0.f) {
        const float kd = da / a, ki = acc.w / a;
        ex.x = ex.x * kd + acc.x * ki;
        ex.y = ex.y * kd + acc.y * ki;
        ex.z = ex.z * kd + acc.z * ki;
    }
    ex.w = a;
    return rgba_to_argb(ex);
}

// findInterval (cuda_findInterval.hpp:26-43): i with levels[i-1] <= v < levels[i]
__device__ __forceinline__ int find_interval(float v, const float* levels, uint32_t count)
{
    if (v < levels[0]) return 0;
    if (v >= levels[count - 1]) return (int)count;
    int i1 = 0, i2 = (int)count;
    while (i2 - i1 > 1) {
        const int i = (i1 + i2) >> 1;
        if (v < levels[i]) i2 = i;
        else i1 = i;
    }
    return i2;
}

// What one block contributes to one pixel in a field mode.
struct ModeOut {
    enum : uint32_t { kNone, kBlend, kMax, kClear } kind;
    float4 acc; // kBlend: non-premultiplied colour and alpha gathered front to back in the block
    float t;    // kMax: (max value - field min) / span
};

// s3r_render_block_argb's march: MODE_ARGB, but a sample is left out where one of its texels is NaN, not where its value
// is (infinite texels filter to a NaN, which shows).  The two are told apart by the NaN that stands for "outside".
constexpr int kPlainArgb = 8;
__device__ __forceinline__ bool is_outside(float v) { return __float_as_uint(v) == 0x7fc00000u; }

// The per-pixel march of one block in a field mode (renderKernel<mode>,
// DenseFieldRenderer_cu.cu:62-215 and render*.hpp): max intensity gives the
// block's maximum above the threshold; the colour modes (Argb, ArgbLight,
// DomainVoxels) and the isosurface modes the colour gathered with blendBehind;
// multi-level modes with no level clear the pixel.
template <class S, int kMode = -1>
__device__ __forceinline__ ModeOut march_block_mode(const s3r_view& v, const s3r_presentation& pr, const S& smp,
                                                    const BlockRay& r, uint32_t depth)
{
    ModeOut out{ModeOut::kNone, make_float4(0.f, 0.f, 0.f, 0.f), 0.f};
    const Relative rel = relative_of(v);
    const float span = rel.span;
    const F3 eye = f3(v.cam.eye);
    const F3 step{r.step[0], r.step[1], r.step[2]};
    // sample k's position: with the texture filter accumulated step by step from
    // the entry point as the reference does (increase(pos, step)), because the
    // texture unit's 8-bit fractions make it sensitive to the last ulp of the
    // position; with the exact filter entry + k * step (one fma), as the oracle
    // and the batched path form it.  Every loop below visits k = 0, 1, 2, ... in
    // order, carrying the accumulated position from one iteration to the next
    // (advance), so that consecutive samples' fetches are independent of one
    // another and can be in flight together.
    F3 seq{r.p0[0], r.p0[1], r.p0[2]};
    auto advance = [&]() {
        if constexpr (S::kStepwise)
            seq = F3{__fadd_rn(seq.x, r.step[0]), __fadd_rn(seq.y, r.step[1]), __fadd_rn(seq.z, r.step[2])};
    };
    auto pos_of = [&](int k) {
        if constexpr (S::kStepwise) {
            return seq; // the caller has advanced to sample k
        } else {
            return F3{__fmaf_rn(r.step[0], (float)k, r.p0[0]), __fmaf_rn(r.step[1], (float)k, r.p0[1]),
                      __fmaf_rn(r.step[2], (float)k, r.p0[2])};
        }
    };
    auto tc_of = [&](F3 p) {
        return F3{__fmul_rn(__fsub_rn(p.x, r.origin[0]), r.factor), __fmul_rn(__fsub_rn(p.y, r.origin[1]), r.factor),
                  __fmul_rn(__fsub_rn(p.z, r.origin[2]), r.factor)};
    };
    // the sample that comes next: its position and, where a fetch is loads alone, these in flight
    F3 pn;
    typename S::Sample ahead;
    auto open = [&](int k) {
        pn = pos_of(k);
        if constexpr (S::kAhead) smp.fetch(0, tc_of(pn), ahead);
    };
    auto value = [&](typename S::Sample& x, F3 p) {
        if constexpr (!S::kAhead) smp.fetch(0, tc_of(p), x);
        return S::value(x);
    };
    constexpr float kMax = 0.996f; // AlphaThreshold / AlphaMaxThreshold
    // kMode >= 0: the mode is fixed at compile time (one kernel per mode, as renderKernel<mode> is), so
    // only its branch is compiled in and the registers are that mode's
    const uint32_t mode = kMode == kPlainArgb ? (uint32_t)S3R_MODE_ARGB : kMode >= 0 ? (uint32_t)kMode : pr.mode;
    if (mode == S3R_MODE_MAX_INTENSITY) {
        // renderMaxIntensityProjection.hpp:30-50; the pixel holds float bits
        float maxv = v.field_min - span;
        // nothing ends this loop early: the compiler unrolls it and issues several samples' loads at once (64 blocks of
        // depth 6 through textures, 64 launches: 0.58 ms, 1.31 with the next sample opened by hand)
        for (int i = 1; i < r.samples; ++i, advance()) {
            typename S::Sample x;
            smp.fetch(0, tc_of(pos_of(i - 1)), x);
            const float val = S::value(x);
            if (val >= v.threshold && maxv < val) maxv = val;
        }
        if (maxv < v.field_min) return out;
        out.kind = ModeOut::kMax;
        out.t = (maxv - v.field_min) / span;
        return out;
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (mode == S3R_MODE_ARGB || mode == S3R_MODE_ARGB_LIGHT || mode == S3R_MODE_DOMAIN_VOXELS) {
        const float of = (v.threshold - v.field_min) / span;
        const float il = layer_exponent(depth, v.level, v.quality);
        float4 dom = make_float4(0.f, 0.f, 0.f, 0.f);
        if (mode == S3R_MODE_DOMAIN_VOXELS) {
            // renderDomainVoxels.hpp:41-42: one colour, the table's middle
            dom = smp.colour(0.5f);
            dom.w = 1.f - powf(1.f - dom.w * of, il);
        }
        open(0);
        for (int i = 1; i < r.samples; ++i) {
            const F3 p = pn;
            typename S::Sample x = ahead;
            if (i + 1 < r.samples) {
                advance();
                open(i);
            }
            const float val = value(x, p);
            if (kMode == kPlainArgb ? is_outside(val) : isnan(val)) continue;
            float4 col;
            if (mode == S3R_MODE_DOMAIN_VOXELS) {
                col = dom;
            } else {
                col = smp.colour(S::kTexRule ? rel.clamped(val) : rel(val));
                col.w = 1.f - powf(1.f - col.w * of, il);
                if (mode == S3R_MODE_ARGB_LIGHT) {
                    // renderArgbLight.hpp:44-56: only visible enough samples are lit
                    if (!(col.w >= 0.00001f)) continue;
                    col = frag_color(smp, col, eye, p, tc_of(p), pr);
                }
            }
            blend_behind(acc, col);
            if (acc.w > kMax) break;
        }
        out.kind = ModeOut::kBlend;
        out.acc = acc;
        return out;
    }
    // isosurface modes: v1 at the entry point, v2 at samples 1 .. sampleCount-1; the
    // crossing is placed at pos + step * t from the later sample, as the reference does
    const bool multi = mode == S3R_MODE_ISOSURFACES || mode == S3R_MODE_VALUE_ON_ISOSURFACES;
    const bool secondary = mode == S3R_MODE_VALUE_ON_ISOSURFACE || mode == S3R_MODE_VALUE_ON_ISOSURFACES;
    const uint32_t nl = pr.level_count;
    if (multi && nl < 1) {
        out.kind = ModeOut::kClear; // renderIsosurfaces.hpp:36-38
        return out;
    }
    auto surface_colour = [&](float level, F3 xpos) {
        float4 dif;
        if (secondary) {
            typename S::Sample x;
            smp.fetch(1, tc_of(xpos), x);
            const float vs = S::value(x);
            dif = smp.colour((vs - pr.secondary_min) / (pr.secondary_max - pr.secondary_min));
        } else {
            dif = smp.colour((level - v.field_min) / span);
        }
        dif.w *= pr.isosurface_opacity;
        return frag_color(smp, dif, eye, xpos, tc_of(xpos), pr);
    };
    auto xpos_of = [&](F3 p, float t) {
        if constexpr (S::kContracted) return F3{p.x + step.x * t, p.y + step.y * t, p.z + step.z * t};
        else
            return F3{__fadd_rn(p.x, __fmul_rn(step.x, t)), __fadd_rn(p.y, __fmul_rn(step.y, t)),
                      __fadd_rn(p.z, __fmul_rn(step.z, t))};
    };
    open(0);
    float v1 = value(ahead, pn);
    if (r.samples > 1) {
        advance();
        open(1);
    }
    if (!multi) {
        const float thr = v.threshold;
        for (int i = 1; i < r.samples; ++i) {
            const F3 p = pn;
            typename S::Sample x = ahead;
            if (i + 1 < r.samples) {
                advance();
                open(i + 1);
            }
            const float v2 = value(x, p);
            if (!isnan(v1) && !isnan(v2) && (v1 - thr) * (v2 - thr) < 0.f) {
                const float t = (thr - v1) / (v2 - v1);
                blend_behind(acc, surface_colour(thr, xpos_of(p, t)));
                if (acc.w > kMax) break;
            }
            v1 = v2;
        }
    } else {
        // renderIsosurfaces.hpp:34-106 / renderValueOnIsosurfaces.hpp
        int iint = isnan(v1) ? -1 : find_interval(v1, pr.levels, nl);
        for (int i = 1; i < r.samples; ++i) {
            const F3 p = pn;
            typename S::Sample x = ahead;
            if (i + 1 < r.samples) {
                advance();
                open(i + 1);
            }
            const float v2 = value(x, p);
            if (isnan(v2)) {
                iint = -1;
                v1 = __int_as_float(0x7fc00000);
                continue;
            }
            if (isnan(v1)) {
                v1 = v2;
                iint = find_interval(v1, pr.levels, nl);
                continue;
            }
            int il, dl;
            if (v2 < v1) {
                if (iint == 0) {
                    v1 = v2;
                    continue;
                }
                il = iint - 1;
                dl = -1;
            } else {
                if (iint == (int)nl) {
                    v1 = v2;
                    continue;
                }
                il = iint;
                dl = 1;
            }
            while (il >= 0 && il < (int)nl) {
                const float level = pr.levels[il];
                if ((v1 - level) * (v2 - level) < 0.f) {
                    const float t = (level - v1) / (v2 - v1);
                    blend_behind(acc, surface_colour(level, xpos_of(p, t)));
                    iint += dl;
                    il += dl;
                } else {
                    break;
                }
            }
            if (acc.w > kMax) break;
            v1 = v2;
        }
    }
    out.kind = ModeOut::kBlend;
    out.acc = acc;
    return out;
}

// A block's contribution to one pixel of the ARGB8 viewport, as renderKernel<mode> stores it.
__device__ __forceinline__ void store_mode_pixel(uint32_t* px, const ModeOut& o)
{
    if (o.kind == ModeOut::kMax) {
        // renderMaxIntensityProjection.hpp:30-50; the pixel holds float bits
        const float prev = __uint_as_float(*px);
        if (!isnan(prev) && prev > o.t) return;
        *px = __float_as_uint(o.t);
    } else if (o.kind == ModeOut::kBlend) {
        *px = blend_above_argb(*px, o.acc);
    } else if (o.kind == ModeOut::kClear) {
        *px = 0u;
    }
}

template <bool kTex, int kMode>
__global__ void render_block_mode_kernel(const s3r_view v, const s3r_presentation pr, const float* __restrict__ brick,
                                         const float* __restrict__ brick2, const RenderBlock rb,
                                         const float* __restrict__ tf_g, uint32_t* __restrict__ viewport)
{
    extern __shared__ float4 tf_sm[];
    const TfTable tf = load_tf<false>(tf_sm, tf_g, v.tf_n, threadIdx.y * blockDim.x + threadIdx.x, blockDim.x * blockDim.y);
    const int32_t xx = blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t yy = blockIdx.y * blockDim.y + threadIdx.y;
    if (xx >= rb.rect[2] || yy >= rb.rect[3]) return;
    const uint32_t vx = (uint32_t)(rb.rect[0] + xx), vy = (uint32_t)(rb.rect[1] + yy);
    if (vx >= v.W || vy >= v.H) return;
    float org[3], dir[3];
    pixel_ray(v, vx, vy, org, dir);
    BlockRay r;
    float inv[3];
    ray_inverse(dir, inv);
    if (!block_ray(v, org, dir, inv, rb, r)) return;
    const BrickSampler<kTex> smp{brick, brick2, dim_of(r), tf, v.tf_n};
    store_mode_pixel(&viewport[(size_t)(v.H - 1 - vy) * v.W + vx],
                     march_block_mode<BrickSampler<kTex>, kMode>(v, pr, smp, r, rb.depth));
}

// The per-pixel ray and the block's sampling set-up written with plain float
// operators in the order of DenseFieldRenderer_cu.cu:72-181 (ray = n + e1 x +
// e2 y, face points eye + ray tau, the dot product of the sample count), so
// that nvcc fuses the same products into the same fmas as in the reference's
// kernel and the samples land where the reference's land.  The texture-unit
// path uses them; the other kernels round every step explicitly, as the
// oracle does.
__device__ __forceinline__ void pixel_ray_fused(const s3r_view& v, uint32_t vx, uint32_t vy, float org[3],
                                                float dir[3])
{
    const float x = (-0.5f + ((float)vx + 0.5f) / (float)v.W) * v.cam.w;
    const float y = (-0.5f + ((float)vy + 0.5f) / (float)v.H) * v.cam.h;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (v.cam.ortho) {
            org[d] = v.cam.eye[d] + v.cam.e1[d] * x + v.cam.e2[d] * y;
            dir[d] = v.cam.n[d];
        } else {
            org[d] = v.cam.eye[d];
            dir[d] = v.cam.n[d] + v.cam.e1[d] * x + v.cam.e2[d] * y;
        }
    }
}

__device__ __forceinline__ bool block_ray_fused(const s3r_view& v, const float org[3], const float dir[3],
                                                const RenderBlock& rb, BlockRay& r)
{
    const float* c = rb.center;
    const float h = rb.half;
    float te = 1.f, tx = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (!(fabsf(dir[a]) > 1e-10f)) continue;
        const int b1 = a == 0 ? 1 : 0;
        const int b2 = a == 2 ? 1 : 2;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const float face = side ? c[a] + h : c[a] - h;
            const float tau = (face - org[a]) / dir[a];
            const float p1 = org[b1] + dir[b1] * tau;
            const float p2 = org[b2] + dir[b2] * tau;
            if (fabsf(p1 - c[b1]) <= h && fabsf(p2 - c[b2]) <= h) {
                const bool enter = (dir[a] > 0.f) == (side == 0);
                if (enter) te = tau;
                else tx = tau;
            }
        }
    }
    if (te < 1.f) te = 1.f;
    r.tau_enter = te;
    r.tau_exit = tx;
    if (!(tx > te)) return false;
    const uint32_t n = (1u << rb.depth) + 1u;
    const float dotr = dir[0] * dir[0] + dir[1] * dir[1] + dir[2] * dir[2];
    const int s = (int)(v.quality * (tx - te) * dotr / (rb.texel * (fabsf(dir[0]) + fabsf(dir[1]) + fabsf(dir[2]))));
    const float dtau = (tx - te) / (float)s;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        r.step[d] = dir[d] * dtau;
        r.p0[d] = org[d] + dir[d] * te;
        r.origin[d] = rb.origin[d];
    }
    r.factor = rb.factor;
    r.n = n;
    r.pitch = n;
    r.samples = s;
    return true;
}

// Pixel tile of one CTA of the texture-unit kernel, per field mode: the fastest of 8x4 .. 64x1 and 16x16
// tiles measured on the 64-block depth-6 workload at 1920x1080 (the texture fetches dominate; 8x8 tiles
// keep a CTA's rays close together, the single-isosurface modes do best with 32x2).
__host__ __device__ constexpr uint32_t tex_tile_x(uint32_t mode)
{
    return (mode == S3R_MODE_ISOSURFACE || mode == S3R_MODE_VALUE_ON_ISOSURFACE) ? 32u : 8u;
}
__host__ __device__ constexpr uint32_t tex_tile_y(uint32_t mode)
{
    return (mode == S3R_MODE_ISOSURFACE || mode == S3R_MODE_VALUE_ON_ISOSURFACE) ? 2u : 8u;
}

// One block in any field mode sampled through the texture unit (the field and
// the transfer function as texture objects), on the fused ray set-up above.
template <int kMode>
__global__ void render_block_texture_kernel(const s3r_view v, const s3r_presentation pr, const TextureSampler smp,
                                            const RenderBlock rb, uint32_t* __restrict__ viewport)
{
    const int32_t xx = blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t yy = blockIdx.y * blockDim.y + threadIdx.y;
    if (xx >= rb.rect[2] || yy >= rb.rect[3]) return;
    const uint32_t vx = (uint32_t)(rb.rect[0] + xx), vy = (uint32_t)(rb.rect[1] + yy);
    if (vx >= v.W || vy >= v.H) return;
    float org[3], dir[3];
    pixel_ray_fused(v, vx, vy, org, dir);
    BlockRay r;
    if (!block_ray_fused(v, org, dir, rb, r)) return;
    store_mode_pixel(&viewport[(size_t)(v.H - 1 - vy) * v.W + vx], march_block_mode<TextureSampler, kMode>(v, pr, smp, r,
                                                                                                       rb.depth));
}

// ---------------------------------------------------------------- a part's blocks at once
//
// A worker's image part is its blocks blended back to front into an ARGB8 viewport, each block's result rounded to
// bytes before the next is blended: an order per pixel, and nothing else, ties the blocks together.  One launch marches
// all the blocks (part_blocks_kernel): a pixel of a block's view rectangle whose ray the block contributes to appends
// its result and the block's place in the back-to-front order to the pixel's list, and part_composite_kernel blends
// every pixel's list in that order with the arithmetic, byte for byte, of one launch per block.  A launch per block
// leaves most of the SMs idle (a block of a level covers a few thousand pixels and its rays take as long as any): 512
// blocks of depth 3 to 7 at 1920x1080 took 9.7 ms in launches of 19 us each, 64 of depth 6 through the texture unit
// 2.0 ms.

// The CTA's block and its tile within it: the last block whose running CTA count is at or below `cta`, by 32 probes at
// a time (every warp finds it for itself).
__device__ __forceinline__ uint32_t find_part_block(const uint32_t* first, uint32_t n, uint32_t cta, uint32_t lane)
{
    uint32_t lo = 0, hi = n; // first[lo] <= cta < first[hi]
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32, probe = lo + (lane + 1) * step;
        const bool below = probe < hi && first[probe] <= cta;
        const uint32_t k = (uint32_t)__popc(__ballot_sync(0xffffffffu, below));
        hi = min(hi, lo + (k + 1) * step);
        lo += k * step;
    }
    return lo;
}

// kFilter: 0 exact, 1 the texture unit's rule in software (both on bricks in memory), 2 the texture unit.
template <int kFilter, int kMode>
__global__ void part_blocks_kernel(const s3r_view v, const s3r_presentation pr, const PartArgs a)
{
    extern __shared__ float4 tf_sm[];
    const uint32_t tid = threadIdx.y * blockDim.x + threadIdx.x;
    const uint32_t b = find_part_block(a.first, a.nblocks, blockIdx.x, tid & 31);
    const PartRef ref = a.refs[b];
    const RenderBlock rb = ref.rb;
    TfTable tf{nullptr, nullptr};
    if constexpr (kFilter != 2) tf = load_tf<false>(tf_sm, a.tf, v.tf_n, tid, blockDim.x * blockDim.y);
    // the rows of the block's rectangle that fall into this strip of the part
    const int32_t y0 = max(rb.rect[1], a.y0), y1 = min(rb.rect[1] + rb.rect[3], a.y0 + a.h);
    const uint32_t tile = blockIdx.x - a.first[b];
    const uint32_t tiles_x = ((uint32_t)rb.rect[2] + blockDim.x - 1) / blockDim.x;
    const int32_t x = rb.rect[0] + (int32_t)((tile % tiles_x) * blockDim.x + threadIdx.x);
    const int32_t y = y0 + (int32_t)((tile / tiles_x) * blockDim.y + threadIdx.y);
    if (x >= rb.rect[0] + rb.rect[2] || y >= y1 || x >= (int32_t)v.W || y >= (int32_t)v.H) return;
    float org[3], dir[3];
    BlockRay r;
    ModeOut o;
    if constexpr (kFilter == 2) {
        pixel_ray_fused(v, (uint32_t)x, (uint32_t)y, org, dir);
        if (!block_ray_fused(v, org, dir, rb, r)) return;
        const TextureSampler smp{(cudaTextureObject_t)ref.src1, (cudaTextureObject_t)ref.src2,
                                 (cudaTextureObject_t)a.tf_tex};
        o = march_block_mode<TextureSampler, kMode>(v, pr, smp, r, rb.depth);
    } else {
        pixel_ray(v, (uint32_t)x, (uint32_t)y, org, dir);
        float inv[3];
        ray_inverse(dir, inv);
        if (!block_ray(v, org, dir, inv, rb, r)) return;
        const BrickSampler<kFilter == 1> smp{reinterpret_cast<const float*>(ref.src1),
                                             reinterpret_cast<const float*>(ref.src2), dim_of(r), tf, v.tf_n};
        o = march_block_mode<BrickSampler<kFilter == 1>, kMode>(v, pr, smp, r, rb.depth);
    }
    if (o.kind == ModeOut::kNone) return;
    // a block whose samples are all transparent leaves the pixel's bytes as they are
    if (o.kind == ModeOut::kBlend && o.acc.w == 0.f) return;
    const uint64_t pix = (uint64_t)(y - a.y0) * (uint32_t)a.w + (uint32_t)(x - a.x0), npix = (uint64_t)a.w * a.h;
    const uint32_t slot = atomicAdd(&a.count[pix], 1u);
    if (slot >= a.cap) {
        *a.overflow = 1; // the caller renders the part block by block instead
        return;
    }
    if (o.kind == ModeOut::kMax) o.acc.x = o.t;
    a.result[slot * npix + pix] = o.acc;
    a.order[slot * npix + pix] = (uint16_t)ref.order;
}

// One thread per pixel of the strip: its list put in order (an insertion sort of the places, a handful of them), then
// blended into the viewport.
constexpr uint32_t kCompositeThreads = 128;
__global__ void __launch_bounds__(kCompositeThreads) part_composite_kernel(const PartArgs a, uint32_t* __restrict__ viewport,
                                                                           uint32_t W, uint32_t H, uint32_t kind)
{
    extern __shared__ uint32_t keys[]; // [cap][thread]: order << 16 | slot
    const uint64_t npix = (uint64_t)a.w * a.h, pix = (uint64_t)blockIdx.x * kCompositeThreads + threadIdx.x;
    if (pix >= npix) return;
    const uint32_t n = min(a.count[pix], a.cap);
    if (n == 0) return;
    uint32_t* key = keys + threadIdx.x;
    for (uint32_t i = 0; i < n; ++i) {
        const uint32_t k = ((uint32_t)a.order[i * npix + pix] << 16) | i;
        uint32_t j = i;
        for (; j > 0 && key[(j - 1) * kCompositeThreads] > k; --j) key[j * kCompositeThreads] = key[(j - 1) * kCompositeThreads];
        key[j * kCompositeThreads] = k;
    }
    const uint32_t x = (uint32_t)a.x0 + (uint32_t)(pix % (uint32_t)a.w), y = (uint32_t)a.y0 + (uint32_t)(pix / (uint32_t)a.w);
    uint32_t* px = &viewport[(size_t)(H - 1 - y) * W + x];
    uint32_t out = *px;
    for (uint32_t i = 0; i < n; ++i) {
        const float4 acc = a.result[(key[i * kCompositeThreads] & 0xffffu) * npix + pix];
        ModeOut o;
        o.kind = (decltype(o.kind))kind;
        o.acc = acc;
        o.t = acc.x;
        store_mode_pixel(&out, o);
    }
    *px = out;
}

// ---------------------------------------------------------------- batched form

// Front-to-back walk of the (2^level)^3 block grid along one ray (Amanatides-Woo).
struct BlockWalk {
    int m;
    int c0, c1, c2, s0, s1, s2;
    float tx0, tx1, tx2, td0, td1, td2, t1;

    // The ray's first block; false when it misses the grid.
    __device__ __forceinline__ bool begin(const float org[3], const float dir[3], const float inv[3], uint32_t level)
    {
        m = 1 << level;
        const float cell = (2.f * kTopHalf) / (float)m;
        // entry/exit of the whole cube [-5, 5]^3, restricted to tau >= 1 (the screen plane)
        float t0 = 1.f;
        t1 = 3.4e38f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (fabsf(dir[a]) > 1e-10f) {
                float ta = (-kTopHalf - org[a]) * inv[a], tb = (kTopHalf - org[a]) * inv[a];
                if (ta > tb) { const float t = ta; ta = tb; tb = t; }
                t0 = fmaxf(t0, ta);
                t1 = fminf(t1, tb);
            } else if (org[a] < -kTopHalf || org[a] > kTopHalf) {
                return false;
            }
        }
        if (!(t1 > t0)) return false;
        // start cell: the one holding the entry point itself (clamped onto the grid);
        // starting any distance inside would skip the first block's segment on rays
        // that enter close to a block boundary
        const float tm = t0;
        // start cell, step direction, next boundary crossing and crossing period per axis
        auto setup = [&](int a, int& c, int& st, float& tmax, float& tdel) {
            const float pm = __fmaf_rn(dir[a], tm, org[a]);
            c = min(max((int)floorf((pm + kTopHalf) / cell), 0), m - 1);
            if (dir[a] > 1e-10f) {
                st = 1;
                tmax = div_by((-kTopHalf + cell * (float)(c + 1)) - org[a], dir[a], inv[a]);
                tdel = div_by(cell, dir[a], inv[a]);
            } else if (dir[a] < -1e-10f) {
                st = -1;
                tmax = div_by((-kTopHalf + cell * (float)c) - org[a], dir[a], inv[a]);
                tdel = div_by(-cell, dir[a], inv[a]);
            } else {
                st = 0;
                tmax = 3.4e38f;
                tdel = 3.4e38f;
            }
        };
        setup(0, c0, s0, tx0, td0);
        setup(1, c1, s1, tx1, td1);
        setup(2, c2, s2, tx2, td2);
        return true;
    }

    __device__ __forceinline__ uint32_t cell() const
    {
        return (uint32_t)c0 + (uint32_t)m * ((uint32_t)c1 + (uint32_t)m * (uint32_t)c2);
    }

    // On to the next block of the ray; false when it has left the grid.  (Every step moves one index towards
    // its end of the grid, an axis the ray does not move along never being chosen before the exit, so a walk
    // visits at most 3 m - 2 blocks.)
    __device__ __forceinline__ bool next()
    {
        if (tx0 <= tx1 && tx0 <= tx2) {
            if (tx0 >= t1) return false;
            c0 += s0;
            tx0 += td0;
            return c0 >= 0 && c0 < m;
        }
        if (tx1 <= tx2) {
            if (tx1 >= t1) return false;
            c1 += s1;
            tx1 += td1;
            return c1 >= 0 && c1 < m;
        }
        if (tx2 >= t1) return false;
        c2 += s2;
        tx2 += td2;
        return c2 >= 0 && c2 < m;
    }
};

// Calls f(block cell) for every block one ray passes, front to back; f returns false to stop.
template <class F>
__device__ __forceinline__ void walk_blocks(const float org[3], const float dir[3], const float inv[3],
                                            uint32_t level, F&& f)
{
    BlockWalk w;
    if (!w.begin(org, dir, inv, level)) return;
    for (int guard = 0; guard < 3 * w.m + 3; ++guard) {
        if (!f(w.cell())) return;
        if (!w.next()) return;
    }
}

__device__ __forceinline__ bool pixel_in_rect(const int32_t* rc, uint32_t vx, uint32_t vy)
{
    return (int32_t)vx >= rc[0] && (int32_t)vx < rc[0] + rc[2] && (int32_t)vy >= rc[1] && (int32_t)vy < rc[1] + rc[3];
}

struct Premul {
    float r, g, b, a;
};

// The 8 texels of a sample issued as independent loads (32-bit offsets: a brick holds at most 513^3 vertices)
// with the cell's fractions: x fastest, then y, then z.
template <int Fmt> struct Texels {
    float t[8];
    float f[3];
};

// Sample k of the ray in its block.  kTogether (the rays of a warp march one block): inside the
// brick the cell's 8 texels are four pairs in four rows, and a sample in the outer half texel (a ray's first one, on
// the block's face) takes the clamped indices.  Rays in different blocks meet their faces at different times, so
// there every sample takes the clamped indices (320 x 240 pixels of a level-2 set: 109 us against 115 us).
template <int Fmt, bool kTogether>
__device__ __forceinline__ void fetch_texels(const void* brick, const BlockRay& r, int k, Texels<Fmt>& x)
{
    const uint32_t hi = r.n - 1;
    const float kf = (float)k;
    int a[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float p = __fmaf_rn(r.step[d], kf, r.p0[d]);
        const float tc = __fmul_rn(__fsub_rn(p, r.origin[d]), r.factor);
        const float xb = __fsub_rn(tc, 0.5f);
        x.f[d] = __fsub_rn(xb, floor_small(xb, a[d]));
    }
    if (kTogether && (uint32_t)a[0] < hi && (uint32_t)a[1] < hi && (uint32_t)a[2] < hi) {
        const uint32_t o = ((uint32_t)a[2] * r.n + (uint32_t)a[1]) * r.pitch + (uint32_t)a[0];
        const uint32_t dz = r.n * r.pitch;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            x.t[q] = Brick<Fmt>::get(brick, (uint64_t)(o + ((q & 2) ? r.pitch : 0u) + ((q & 4) ? dz : 0u)) + (q & 1));
    } else {
        uint32_t i0[3], i1[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            i0[d] = (uint32_t)min(max(a[d], 0), (int)hi);
            i1[d] = (uint32_t)min(max(a[d] + 1, 0), (int)hi);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t xi = (q & 1) ? i1[0] : i0[0];
            const uint32_t yi = (q & 2) ? i1[1] : i0[1];
            const uint32_t zi = (q & 4) ? i1[2] : i0[2];
            x.t[q] = Brick<Fmt>::get(brick, (zi * r.n + yi) * r.pitch + xi);
        }
    }
}

// Trilinear value of fetched texels; false when one of them is NaN (outside the domain).
template <int Fmt> __device__ __forceinline__ bool filter_texels(const Texels<Fmt>& x, float& val)
{
    if (any_nan(x.t)) return false;
    val = lerp_cell(x.t, x.f);
    return true;
}

// March one block along a ray (premultiplied, block-local early termination).
// Exact filter: software-pipelined over two sets of texels -- sample k+1's loads
// are issued before sample k is filtered, looked up and composited, so a ray
// keeps two samples' loads in flight; the arithmetic and its order are the
// per-block kernel's.  What bounds it is the issue of the sample's instructions
// (and, before floor_small and div_by, the conversion unit).
template <int Fmt, bool kTex, bool kTogether>
__device__ __forceinline__ Premul march_block(const s3r_view& v, const BlockRay& r, const void* brick, float scale,
                                              float offset, uint32_t depth, const TfTable& tf, const Relative& rel,
                                              float of, uint32_t& taken)
{
    const float il = layer_exponent(depth, v.level, v.quality);
    Premul acc{0.f, 0.f, 0.f, 0.f};
    auto blend = [&](float4 col) {
        const float a = __fsub_rn(1.f, __powf(__fmaf_rn(-col.w, of, 1.f), il));
        const float w = __fmul_rn(__fsub_rn(1.f, acc.a), a);
        acc.r = __fmaf_rn(w, col.x, acc.r);
        acc.g = __fmaf_rn(w, col.y, acc.g);
        acc.b = __fmaf_rn(w, col.z, acc.b);
        acc.a = __fadd_rn(acc.a, w);
        return acc.a > kAlphaThreshold;
    };
    if constexpr (!kTex) {
        if (r.samples < 2) return acc;
        Texels<Fmt> ca, cb;
        // true: the block is opaque
        auto sample = [&](const Texels<Fmt>& x) {
            float val;
            if (!filter_texels<Fmt>(x, val)) return false;
            if (Fmt != S3R_BRICK_F32) val = __fmaf_rn(scale, val, offset);
            return blend(tf_colour(tf, v.tf_n, rel(val)));
        };
        fetch_texels<Fmt, kTogether>(brick, r, 0, ca);
        const int last = r.samples - 1; // samples 0 .. last-1
        int k = 0;                      // the samples taken (a float would stop counting at 2^24)
        while (true) {
            ++k;
            if (k < last) fetch_texels<Fmt, kTogether>(brick, r, k, cb);
            if (sample(ca) || k >= last) break;
            ++k;
            if (k < last) fetch_texels<Fmt, kTogether>(brick, r, k, ca);
            if (sample(cb) || k >= last) break;
        }
        taken += (uint32_t)k;
        return acc;
    } else {
        for (int i = 1; i < r.samples; ++i) {
            ++taken;
            float val;
            if (!tex_trilinear<Fmt>(brick, r, i - 1, val)) continue;
            if (Fmt != S3R_BRICK_F32) val = __fmaf_rn(scale, val, offset);
            if (blend(tex_tf_lookup(tf.raw(), v.tf_n, rel.clamped(val)))) break;
        }
        return acc;
    }
}

// march_block with `lanes` consecutive lanes (2, 4 or 8) to a ray: lane `sub` fetches, filters and looks up samples
// sub, sub + lanes, ...; the samples' colours then go around by shuffles and every lane of the ray composites them in
// order, so the result is march_block's bit for bit.  A ray's chain of samples is that much shorter, for a third more
// instructions in all; a warp's 32 lanes call it together (last: samples to take, 0 for no ray).
template <int Fmt, bool kTex>
__device__ __forceinline__ Premul march_block_lanes(const s3r_view& v, const BlockRay& r, int last, const void* brick,
                                                    float scale, float offset, uint32_t depth, const TfTable& tf,
                                                    const Relative& rel, float of, uint32_t lanes, uint32_t sub,
                                                    uint32_t& taken)
{
    const float il = layer_exponent(depth, v.level, v.quality);
    Premul acc{0.f, 0.f, 0.f, 0.f};
    bool open = last > 0;
    int k0 = 0; // the group's first sample
    Texels<Fmt> cur, nxt;
    if constexpr (!kTex)
        if ((int)sub < last) fetch_texels<Fmt, true>(brick, r, (int)sub, cur);
    while (__any_sync(0xffffffffu, open)) {
        const int k = k0 + (int)sub, next = k + (int)lanes;
        if constexpr (!kTex)
            if (open && next < last) fetch_texels<Fmt, true>(brick, r, next, nxt);
        // a sample outside the domain blends as nothing: all zero
        float4 col = make_float4(0.f, 0.f, 0.f, 0.f);
        if (open && k < last) {
            float val;
            bool in;
            if constexpr (kTex) in = tex_trilinear<Fmt>(brick, r, k, val);
            else in = filter_texels<Fmt>(cur, val);
            if (in) {
                if (Fmt != S3R_BRICK_F32) val = __fmaf_rn(scale, val, offset);
                col = kTex ? tex_tf_lookup(tf.raw(), v.tf_n, rel.clamped(val)) : tf_colour(tf, v.tf_n, rel(val));
                col.w = __fsub_rn(1.f, __powf(__fmaf_rn(-col.w, of, 1.f), il));
            }
        }
#pragma unroll 2
        for (uint32_t j = 0; j < lanes; ++j) {
            const float cr = __shfl_sync(0xffffffffu, col.x, j, lanes), cg = __shfl_sync(0xffffffffu, col.y, j, lanes),
                        cb = __shfl_sync(0xffffffffu, col.z, j, lanes), a = __shfl_sync(0xffffffffu, col.w, j, lanes);
            if (open) {
                const float w = __fmul_rn(__fsub_rn(1.f, acc.a), a);
                acc.r = __fmaf_rn(w, cr, acc.r);
                acc.g = __fmaf_rn(w, cg, acc.g);
                acc.b = __fmaf_rn(w, cb, acc.b);
                acc.a = __fadd_rn(acc.a, w);
                ++k0;
                if (sub == 0) ++taken;
                open = !(acc.a > kAlphaThreshold) && k0 < last;
            }
        }
        if constexpr (!kTex) cur = nxt;
    }
    return acc;
}

// One pixel ray per R consecutive lanes: the ray's block sequence (the DDA
// order) is cut into R contiguous runs, lane r composites run r, and the R
// premultiplied partial results are merged front to back with shuffles (the
// over operator is associative).  With R > 1 a ray stops early only inside its
// run, so R = 1 is used when view.alpha_stop < 1.
template <int Fmt, int R, bool kTex>
__global__ void frame_render_kernel(FrameArgs fa)
{
    extern __shared__ float4 tf_sm[];
    const s3r_view v = *fa.view;
    const uint32_t nthreads = blockDim.x * blockDim.y;
    const uint32_t tid = threadIdx.y * blockDim.x + threadIdx.x;
    const uint32_t seg = threadIdx.x % R;
    const uint32_t px_per_row = blockDim.x / R;
    const uint32_t vx = blockIdx.x * px_per_row + threadIdx.x / R;
    const uint32_t vy = blockIdx.y * blockDim.y + threadIdx.y;
    {
        // CTAs whose pixels no block covers only clear their pixels
        const int4 cv = *reinterpret_cast<const int4*>(fa.cover);
        const int32_t x0 = blockIdx.x * px_per_row, y0 = blockIdx.y * blockDim.y;
        if (x0 >= cv.z || x0 + (int32_t)px_per_row <= cv.x || y0 >= cv.w || y0 + (int32_t)blockDim.y <= cv.y) {
            if (seg == 0 && vx < v.W && vy < v.H) {
                const size_t o = (size_t)(v.H - 1 - vy) * v.W + vx;
                if (fa.rgba) reinterpret_cast<float4*>(fa.rgba)[o] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (fa.argb) fa.argb[o] = 0u;
            }
            return;
        }
    }
    const TfTable tf = load_tf<false>(tf_sm, fa.tf, v.tf_n, tid, nthreads);
    const Relative rel = relative_of(v);
    uint32_t taken = 0;
    Premul acc{0.f, 0.f, 0.f, 0.f};
    const bool inside = vx < v.W && vy < v.H;
    if (inside) {
        float org[3], dir[3];
        pixel_ray(v, vx, vy, org, dir);
        float inv[3];
        ray_inverse(dir, inv);
        const float of = (v.threshold - v.field_min) / (v.field_max - v.field_min);
        int lo = 0, hi = 1 << 30;
        if (R > 1) {
            int n = 0;
            walk_blocks(org, dir, inv, v.level, [&](uint32_t) {
                ++n;
                return true;
            });
            const int chunk = (n + R - 1) / R;
            lo = (int)seg * chunk;
            hi = lo + chunk;
        }
        int idx = 0;
        walk_blocks(org, dir, inv, v.level, [&](uint32_t b) {
            if (idx >= hi) return false;
            if (idx++ < lo) return true;
            const RenderBlock* rb = &fa.table[b];
            const uint32_t depth = rb->depth;
            if (depth == 0xffffffffu) return true;
            const int4 rc = *reinterpret_cast<const int4*>(rb->rect);
            const int32_t rca[4] = {rc.x, rc.y, rc.z, rc.w};
            if (!pixel_in_rect(rca, vx, vy)) return true;
            BlockRay r;
            if (!block_ray(v, org, dir, inv, *rb, r)) return true;
            const char* base = reinterpret_cast<const char*>(fa.bricks);
            const size_t esz = Fmt == S3R_BRICK_F32 ? 4 : 2;
            float scale = 1.f, offset = 0.f;
            if (Fmt != S3R_BRICK_F32) {
                const float2 so = fa.scale_offset[rb->block];
                scale = so.x;
                offset = so.y;
            }
            const Premul p =
                march_block<Fmt, kTex, false>(v, r, base + rb->brick_off * esz, scale, offset, depth, tf, rel, of, taken);
            const float T = __fsub_rn(1.f, acc.a);
            acc.r = __fmaf_rn(T, p.r, acc.r);
            acc.g = __fmaf_rn(T, p.g, acc.g);
            acc.b = __fmaf_rn(T, p.b, acc.b);
            acc.a = __fmaf_rn(T, p.a, acc.a);
            return !(acc.a > v.alpha_stop);
        });
    }
    // merge the runs front to back: lane seg (a multiple of 2*off) takes lane seg+off behind it
#pragma unroll
    for (int off = 1; off < R; off <<= 1) {
        const float br = __shfl_down_sync(0xffffffffu, acc.r, off, R);
        const float bg = __shfl_down_sync(0xffffffffu, acc.g, off, R);
        const float bb = __shfl_down_sync(0xffffffffu, acc.b, off, R);
        const float ba = __shfl_down_sync(0xffffffffu, acc.a, off, R);
        if ((seg & (2 * off - 1)) == 0) {
            const float T = __fsub_rn(1.f, acc.a);
            acc.r = __fmaf_rn(T, br, acc.r);
            acc.g = __fmaf_rn(T, bg, acc.g);
            acc.b = __fmaf_rn(T, bb, acc.b);
            acc.a = __fmaf_rn(T, ba, acc.a);
        }
    }
    if (inside && seg == 0) {
        const size_t o = (size_t)(v.H - 1 - vy) * v.W + vx;
        float4 out = make_float4(0.f, 0.f, 0.f, acc.a);
        if (acc.a > 0.f) {
            const float inv = 1.f / acc.a;
            out.x = acc.r * inv;
            out.y = acc.g * inv;
            out.z = acc.b * inv;
        }
        if (fa.rgba) reinterpret_cast<float4*>(fa.rgba)[o] = out;
        if (fa.argb) fa.argb[o] = rgba_to_argb(out);
    }
    if (fa.samples) {
        unsigned long long t = taken;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if ((tid & 31) == 0 && t) atomicAdd(fa.samples, t);
    }
}

// Non-premultiplied RGBA and ARGB32 of a composited ray, row-flipped as the reference stores pixels.
__device__ __forceinline__ void write_pixel(const FrameArgs& fa, const s3r_view& v, uint32_t vx, uint32_t vy,
                                            const Premul& acc)
{
    const size_t o = (size_t)(v.H - 1 - vy) * v.W + vx;
    float4 out = make_float4(0.f, 0.f, 0.f, acc.a);
    if (acc.a > 0.f) {
        const float inv = 1.f / acc.a;
        out.x = acc.r * inv;
        out.y = acc.g * inv;
        out.z = acc.b * inv;
    }
    if (fa.rgba) reinterpret_cast<float4*>(fa.rgba)[o] = out;
    if (fa.argb) fa.argb[o] = rgba_to_argb(out);
}

// ---------------------------------------------------------------- block-major form

// Front-to-back rank of block (ix, iy, iz) on a ray of direction dir.  Along a
// ray every block index moves monotonically in the direction of its component's
// sign, one step at a time, so this sum grows by exactly one per block the ray
// passes: the blocks of a ray sort front to back by it, and a ray meets at most
// 3m - 2 ranks (m blocks per axis).
__device__ __forceinline__ uint32_t ray_rank(const float dir[3], uint32_t ix, uint32_t iy, uint32_t iz, uint32_t m)
{
    return (dir[0] < 0.f ? m - 1 - ix : ix) + (dir[1] < 0.f ? m - 1 - iy : iy) + (dir[2] < 0.f ? m - 1 - iz : iz);
}

// Whether the per-ray walk (walk_blocks) meets this block on the ray, block_ray having found that the ray passes it.
// It does wherever the middle of the ray's segment lies inside the block by more than the walk's rounding; only a ray
// that grazes the block -- along a face, past an edge -- is walked to see which of the blocks around it the walk takes.
// A crossing time is a quotient (two roundings, and one of its numerator) and up to m sums of a period: off by at most
// (m + 4) 2^-24 of the time itself; two of them are compared, which is as far along the ray as |dir| times that, and
// twice as much is asked for.
__device__ __forceinline__ bool on_walk(const s3r_view& v, const float org[3], const float dir[3], const float inv[3],
                                        const RenderBlock& rb, const BlockRay& r, uint32_t cell)
{
    const float way = fmaxf(fmaxf(fabsf(dir[0]), fabsf(dir[1])), fabsf(dir[2])) * r.tau_exit;
    const float tm = 0.5f * (r.tau_enter + r.tau_exit),
                room = rb.half - (1e-5f + (float)((1u << v.level) + 4u) * 2.3841858e-7f * way); // 2^-22
    bool inside = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) inside &= fabsf(__fmaf_rn(dir[d], tm, org[d]) - rb.center[d]) < room;
    if (inside) return true;
    bool met = false;
    walk_blocks(org, dir, inv, v.level, [&](uint32_t b) {
        met = b == cell;
        return !met;
    });
    return met;
}

// Block-major ray cast: the work items are the warp-sized pixel tiles of every
// block's view rectangle, blocks in decreasing depth (most samples per ray
// first); each warp of a persistent grid takes items from a work-queue counter on
// its own, fetching the next item while it marches the current one.  A lane
// marches its pixel's ray through the item's block exactly as frame_render_kernel
// does (pixel_ray, block_ray, march_block) and stores the premultiplied result at
// the block's front-to-back rank on that ray, marking the rank in the pixel's
// mask; a zero result changes no composite and is not stored.  The lanes of an
// item read one brick, their rays cross it side by side (similar sample counts),
// and the deep blocks' items spread over every SM -- the per-ray walk's lanes
// instead each hold their own block sequence.  frame_composite_kernel then blends
// every pixel's results in rank order with frame_render_kernel's arithmetic.
// kLanes: an item of a block whose rays would take longer than the whole frame's
// share of a warp has 2, 4 or 8 lanes to a ray (SegArgs::items).  A kernel of its
// own: with both marches in it the one with one lane to a ray has too few
// registers (64 blocks of depth 6 at 1920x1080: 336 us instead of 278).
constexpr uint32_t kSegThreads = 512; // warps on their own items, sharing a transfer-function table
template <int Fmt, bool kTex, bool kLanes>
__global__ void __launch_bounds__(kSegThreads, 2) frame_segments_kernel(FrameArgs fa, SegArgs sa, uint32_t fx)
{
    extern __shared__ float4 tf_sm[];
    const s3r_view v = *fa.view;
    const uint32_t nthreads = blockDim.x * blockDim.y;
    const uint32_t tid = threadIdx.y * blockDim.x + threadIdx.x;
    const TfTable tf = load_tf<true>(tf_sm, fa.tf, v.tf_n, tid, nthreads);
    const Relative rel = relative_of(v);
    const uint32_t lane = tid & 31u;
    const uint32_t total = *sa.count;
    const uint32_t m = 1u << v.level;
    const int4 cv = *reinterpret_cast<const int4*>(fa.cover);
    const uint32_t cw = (uint32_t)(cv.z - cv.x);
    const uint64_t npix = (uint64_t)cw * (uint32_t)(cv.w - cv.y);
    const float of = (v.threshold - v.field_min) / (v.field_max - v.field_min);
    uint32_t taken = 0;
    auto take = [&](uint32_t& item, uint2& desc) {
        item = 0xffffffffu;
        desc = make_uint2(0u, 0u);
        if (lane == 0) {
            item = atomicAdd(sa.queue, 1u);
            if (item < total) desc = sa.items[item];
        }
    };
    uint32_t item;
    uint2 desc;
    take(item, desc);
    item = __shfl_sync(0xffffffffu, item, 0);
    desc.x = __shfl_sync(0xffffffffu, desc.x, 0);
    desc.y = __shfl_sync(0xffffffffu, desc.y, 0);
    while (item < total) {
        uint32_t next;
        uint2 ndesc;
        take(next, ndesc); // in flight while this item is marched
        const uint32_t cell = desc.x & kSegCellMask, tile = desc.y,
                       log_lanes = kLanes ? desc.x >> kSegLanesShift : 0u;
        const RenderBlock* rb = &fa.table[cell];
        const int4 rc = *reinterpret_cast<const int4*>(rb->rect);
        uint32_t w, h;
        seg_footprint(fx, log_lanes, w, h);
        const uint32_t p = lane >> log_lanes, tiles_x = ((uint32_t)rc.z + w - 1) / w;
        const int32_t x = rc.x + (int32_t)((tile % tiles_x) * w + p % w);
        const int32_t y = rc.y + (int32_t)((tile / tiles_x) * h + p / w);
        float org[3], dir[3];
        BlockRay r;
        bool hit = false;
        if (x < rc.x + rc.z && y < rc.y + rc.w && x >= 0 && y >= 0 && x < (int32_t)v.W && y < (int32_t)v.H) {
            pixel_ray(v, (uint32_t)x, (uint32_t)y, org, dir);
            float inv[3];
            ray_inverse(dir, inv);
            hit = block_ray(v, org, dir, inv, *rb, r);
            if (hit && sa.walk) hit = on_walk(v, org, dir, inv, *rb, r, cell);
        }
        const char* brick = reinterpret_cast<const char*>(fa.bricks) + rb->brick_off * (Fmt == S3R_BRICK_F32 ? 4 : 2);
        float scale = 1.f, offset = 0.f;
        if (Fmt != S3R_BRICK_F32) {
            const float2 so = fa.scale_offset[rb->block];
            scale = so.x;
            offset = so.y;
        }
        Premul acc{0.f, 0.f, 0.f, 0.f};
        if (kLanes && log_lanes) {
            const uint32_t lanes = 1u << log_lanes, sub = lane & (lanes - 1);
            acc = march_block_lanes<Fmt, kTex>(v, r, hit ? r.samples - 1 : 0, brick, scale, offset,
                                               rb->depth, tf, rel, of, lanes, sub, taken);
            hit = hit && sub == 0;
        } else if (hit) {
            acc = march_block<Fmt, kTex, true>(v, r, brick, scale, offset, rb->depth, tf, rel, of, taken);
        }
        if (hit && !(acc.r == 0.f && acc.g == 0.f && acc.b == 0.f && acc.a == 0.f)) {
            const uint32_t ix = cell % m, iy = (cell / m) % m, iz = cell / (m * m);
            const uint32_t k = ray_rank(dir, ix, iy, iz, m);
            const uint64_t pix = (uint64_t)(y - cv.y) * cw + (uint32_t)(x - cv.x);
            sa.seg[(uint64_t)k * npix + pix] = make_float4(acc.r, acc.g, acc.b, acc.a);
            atomicOr(&sa.mask[(uint64_t)(k >> 6) * npix + pix], 1ull << (k & 63));
        }
        item = __shfl_sync(0xffffffffu, next, 0);
        desc.x = __shfl_sync(0xffffffffu, ndesc.x, 0);
        desc.y = __shfl_sync(0xffffffffu, ndesc.y, 0);
    }
    if (fa.samples) {
        unsigned long long t = taken;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0 && t) atomicAdd(fa.samples, t);
    }
}

// The work items of a view from its list of blocks, a CTA to a block: a few writes each, in place of a list that the
// host fills and copies (270 000 items, 2.2 MB, for 512 blocks at 1920 x 1080).
__global__ void seg_items_kernel(const uint2* __restrict__ list, uint2* __restrict__ items)
{
    const uint2 b = list[blockIdx.x];
    const uint32_t n = list[blockIdx.x + 1].y - b.y;
    for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) items[b.y + t] = make_uint2(b.x, t);
}

// Front-to-back blend of every pixel's block results in rank order -- the
// order frame_render_kernel's walk meets the blocks in -- with its arithmetic
// and its alpha_stop rule; clears the masks and the work-queue counter for the
// next frame.
__global__ void frame_composite_kernel(FrameArgs fa, SegArgs sa)
{
    const s3r_view v = *fa.view;
    const uint64_t at = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (at == 0) *sa.queue = 0u;
    if (at >= (uint64_t)v.W * v.H) return;
    const uint32_t x = (uint32_t)(at % v.W), y = (uint32_t)(at / v.W);
    const int4 cv = *reinterpret_cast<const int4*>(fa.cover);
    const uint32_t cw = (uint32_t)(cv.z - cv.x);
    const uint64_t npix = (uint64_t)cw * (uint32_t)(cv.w - cv.y);
    const uint64_t pix = (uint64_t)((int32_t)y - cv.y) * cw + (uint32_t)((int32_t)x - cv.x);
    const bool covered = (int32_t)x >= cv.x && (int32_t)x < cv.z && (int32_t)y >= cv.y && (int32_t)y < cv.w;
    unsigned long long bits[kSegMaskWords];
#pragma unroll
    for (uint32_t w = 0; w < kSegMaskWords; ++w) {
        bits[w] = 0ull;
        if (covered && w < sa.words) {
            bits[w] = sa.mask[w * npix + pix];
            if (bits[w]) sa.mask[w * npix + pix] = 0ull;
        }
    }
    Premul acc{0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (uint32_t w = 0; w < kSegMaskWords; ++w) {
        while (bits[w] && !(acc.a > v.alpha_stop)) {
            const uint32_t k = 64 * w + (uint32_t)(__ffsll((long long)bits[w]) - 1);
            bits[w] &= bits[w] - 1;
            const float4 p = sa.seg[(uint64_t)k * npix + pix];
            const float T = __fsub_rn(1.f, acc.a);
            acc.r = __fmaf_rn(T, p.x, acc.r);
            acc.g = __fmaf_rn(T, p.y, acc.g);
            acc.b = __fmaf_rn(T, p.z, acc.b);
            acc.a = __fmaf_rn(T, p.w, acc.a);
        }
    }
    write_pixel(fa, v, x, y, acc);
}

// Batched field modes (F32 bricks): one lane per ray walks the blocks front
// to back, each block marched as render_block_mode_kernel marches it
// (march_block_mode), and the blocks' contributions are combined in float: the
// colour modes' block results composited front to back (premultiplied) with
// no ARGB8 rounding between blocks, max intensity the maximum over the
// blocks, and a multi-level mode without levels clears the pixel (what lies
// behind the first block it meets is erased, as the per-block path erases it).
// A kernel per mode and filter, as renderKernel<mode> is (with the mode known at run time: 128 registers and spills).
// What bounds it is the march's instructions and rays of a warp that meet surfaces at different samples; lit
// isosurfaces, 64 blocks of depth 6, 1280x720: 557 us at first, 314 with the cell's fast path, 304 per mode with 8 x 4
// pixels a warp (16 x 2: 343), 275 with the next sample in flight; 5 and 6 CTAs an SM 292 and 303.
template <bool kTex, int kMode>
__global__ void __launch_bounds__(128, 4) frame_render_mode_kernel(FrameArgs fa, const s3r_presentation pr, const float* __restrict__ bricks2)
{
    extern __shared__ float4 tf_sm[];
    const s3r_view v = *fa.view;
    const uint32_t nthreads = blockDim.x * blockDim.y;
    const uint32_t tid = threadIdx.y * blockDim.x + threadIdx.x;
    const TfTable tf = load_tf<false>(tf_sm, fa.tf, v.tf_n, tid, nthreads);
    const uint32_t vx = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t vy = blockIdx.y * blockDim.y + threadIdx.y;
    if (vx >= v.W || vy >= v.H) return;
    constexpr bool mip = kMode == S3R_MODE_MAX_INTENSITY;
    Premul acc{0.f, 0.f, 0.f, 0.f};
    bool have_max = false;
    float best = 0.f;
    const int4 cv = *reinterpret_cast<const int4*>(fa.cover);
    if ((int32_t)vx >= cv.x && (int32_t)vx < cv.z && (int32_t)vy >= cv.y && (int32_t)vy < cv.w) {
        float org[3], dir[3];
        pixel_ray(v, vx, vy, org, dir);
        float inv[3];
        ray_inverse(dir, inv);
        const float* bricks = reinterpret_cast<const float*>(fa.bricks);
        walk_blocks(org, dir, inv, v.level, [&](uint32_t b) {
            const RenderBlock* rb = &fa.table[b];
            const uint32_t depth = rb->depth;
            if (depth == 0xffffffffu) return true;
            const int4 rc = *reinterpret_cast<const int4*>(rb->rect);
            const int32_t rca[4] = {rc.x, rc.y, rc.z, rc.w};
            if (!pixel_in_rect(rca, vx, vy)) return true;
            BlockRay r;
            if (!block_ray(v, org, dir, inv, *rb, r)) return true;
            const BrickSampler<kTex> smp{bricks + rb->brick_off, bricks2 ? bricks2 + rb->brick_off : nullptr, dim_of(r),
                                         tf, v.tf_n};
            const ModeOut o = march_block_mode<BrickSampler<kTex>, kMode>(v, pr, smp, r, depth);
            if (o.kind == ModeOut::kMax) {
                if (!have_max || o.t > best) best = o.t;
                have_max = true;
            } else if (o.kind == ModeOut::kBlend) {
                const float T = __fsub_rn(1.f, acc.a);
                acc.r = __fmaf_rn(T, __fmul_rn(o.acc.x, o.acc.w), acc.r);
                acc.g = __fmaf_rn(T, __fmul_rn(o.acc.y, o.acc.w), acc.g);
                acc.b = __fmaf_rn(T, __fmul_rn(o.acc.z, o.acc.w), acc.b);
                acc.a = __fmaf_rn(T, o.acc.w, acc.a);
            } else if (o.kind == ModeOut::kClear) {
                return false;
            }
            return mip || !(acc.a > v.alpha_stop);
        });
    }
    const size_t o = (size_t)(v.H - 1 - vy) * v.W + vx;
    if (mip) {
        if (fa.rgba)
            reinterpret_cast<float4*>(fa.rgba)[o] =
                have_max ? make_float4(best, best, best, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (fa.argb) fa.argb[o] = have_max ? __float_as_uint(best) : 0x7fc00000u;
        return;
    }
    write_pixel(fa, v, vx, vy, acc);
}

// ---------------------------------------------------------------- adjoint

__device__ __forceinline__ bool filter_cell(const float f[3], const float t[8], float& val)
{
    if (any_nan(t)) return false;
    val = lerp_cell(t, f);
    return true;
}

// A sample's cell in an F32 brick: its low corner (before clamping) and fractions, and its 8 texels.
struct GradCell {
    int a[3];
    float f[3];
    float t[8];
};

__device__ __forceinline__ bool inside_brick(const int a[3], uint32_t hi)
{
    return (uint32_t)a[0] < hi && (uint32_t)a[1] < hi && (uint32_t)a[2] < hi;
}

// Offset of corner q (x | y << 1 | z << 2) of a cell that reaches over the brick's edge, by the clamped indices.
__device__ __forceinline__ uint32_t clamped_corner(const int a[3], Dim g, int q)
{
    const int hi = (int)g.n - 1;
    const int x = min(max(a[0] + (q & 1), 0), hi), y = min(max(a[1] + ((q >> 1) & 1), 0), hi),
              z = min(max(a[2] + (q >> 2), 0), hi);
    return ((uint32_t)z * g.n + (uint32_t)y) * g.pitch + (uint32_t)x;
}

__device__ __forceinline__ void fetch_grad_cell(const float* brick, const BlockRay& r, int k, GradCell& c)
{
    const float kf = (float)k;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float p = __fmaf_rn(r.step[d], kf, r.p0[d]);
        const float tc = __fmul_rn(__fsub_rn(p, r.origin[d]), r.factor);
        const float xb = __fsub_rn(tc, 0.5f);
        c.f[d] = __fsub_rn(xb, floor_small(xb, c.a[d]));
    }
    if (inside_brick(c.a, r.n - 1)) {
        const uint32_t o = ((uint32_t)c.a[2] * r.n + (uint32_t)c.a[1]) * r.pitch + (uint32_t)c.a[0];
        const uint32_t dz = r.n * r.pitch;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            c.t[q] = __ldg(brick + (uint64_t)(o + ((q & 2) ? r.pitch : 0u) + ((q & 4) ? dz : 0u)) + (q & 1));
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) c.t[q] = __ldg(brick + clamped_corner(c.a, dim_of(r), q));
    }
}

// The dense-value gradients of a ray's current cell, kept in registers while the ray moves from cell to cell: a step
// of one along an axis hands the shared face's four sums on and only the face left behind goes to memory, so that a
// sample costs four to seven reductions instead of eight.  A ray moves one way along each axis, so corners are counted
// along the ray: bit a of q is 0 for the face it entered by, and stride[a] leads from that face to the other one.
struct CellGradient {
    float g[8];
    int a[3];       // the cell's low corner
    float* p;       // corner 0
    int stride[3];

    __device__ __forceinline__ void begin(const float step[3], float* dense, int pitch, int dz)
    {
        p = dense;
        stride[0] = step[0] < 0.f ? -1 : 1;
        stride[1] = step[1] < 0.f ? -pitch : pitch;
        stride[2] = step[2] < 0.f ? -dz : dz;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (stride[d] < 0) p -= stride[d];
            a[d] = 0;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) g[q] = 0.f;
    }
    // The corners in `which` (bit q) go to memory.
    __device__ __forceinline__ void put(uint32_t which) const
    {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (((which >> q) & 1u) && g[q] != 0.f)
                atomicAdd(p + (((q & 1) ? stride[0] : 0) + ((q & 2) ? stride[1] : 0) + ((q & 4) ? stride[2] : 0)), g[q]);
    }
    // The ray is now in the (inside) cell `to` of the brick whose gradients start at `dense`: the corners left behind
    // go out, the others move up, without a branch on the axes (a warp's rays cross their faces at different samples;
    // with branches 267 us where this takes 254, and 220 where it takes 201).
    __device__ __forceinline__ void move(const int to[3], float* dense, uint32_t n, uint32_t pitch)
    {
        // steps along the ray: 0 or 1 per axis, or the cell is left altogether
        const int dx = stride[0] < 0 ? a[0] - to[0] : to[0] - a[0], dy = stride[1] < 0 ? a[1] - to[1] : to[1] - a[1],
                  dz = stride[2] < 0 ? a[2] - to[2] : to[2] - a[2];
        if ((dx | dy | dz) == 0) return;
        const bool all = (uint32_t)(dx | dy | dz) > 1u;
        put(all ? 0xffu : ((dx ? 0x55u : 0u) | (dy ? 0x33u : 0u) | (dz ? 0x0fu : 0u)));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const bool moved = all || (d == 0 ? dx : d == 1 ? dy : dz) != 0;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (!(q & (1 << d))) {
                    g[q] = moved ? g[q | (1 << d)] : g[q];
                    g[q | (1 << d)] = moved ? 0.f : g[q | (1 << d)];
                }
        }
        if (all) g[0] = 0.f; // corner 7, out already
        p = dense + (((uint32_t)to[2] * n + (uint32_t)to[1]) * pitch + (uint32_t)to[0]);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (stride[d] < 0) p -= stride[d];
            a[d] = to[d];
        }
    }
    // Adds the sample's gradient by its trilinear weights.
    __device__ __forceinline__ void add(float v, const float f[3])
    {
        float w[3][2];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            w[d][1] = stride[d] < 0 ? 1.f - f[d] : f[d];
            w[d][0] = stride[d] < 0 ? f[d] : 1.f - f[d];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) g[q] = __fmaf_rn(v, w[0][q & 1] * w[1][(q >> 1) & 1] * w[2][q >> 2], g[q]);
    }
};

// For L = 1/2 sum (I - target)^2 with I = (C/A, A) the premultiplied composite
// of the kept samples (front to back, T_k = prod_{j<k} (1 - a_k)):
//   dC/dc_k = T_k a_k,  dC/da_k = T_k c_k - (C - C_{<=k}) / (1 - a_k),
//   dA/da_k = (1 - A) / (1 - a_k),
// a_k = 1 - (1 - alpha_tf * of)^il, c_k / alpha_tf linear in the table
// entries around v01, v01 linear in the trilinear value.  With s_k = gC . c_k
// the gradient of a_k is T_k s_k + Q_k / (1 - a_k), Q_k = gA (1 - A) - gC . (C -
// C_{<=k}), and Q grows by T_k a_k s_k from one sample to the next: one number a
// ray where the composite has three.
//
// What bounds it: the reductions into the dense gradient (about a third of the
// time) and the latency of a ray's chain of samples, at the warps that the
// registers leave room for; the ray, its walk and what only a new block needs are
// kept in shared memory.
constexpr uint32_t kBackwardThreads = 64;
struct BackwardShared {
    BlockWalk walk[kBackwardThreads];
    float ray[9][kBackwardThreads]; // origin, direction, 1 / direction
};

__global__ void __launch_bounds__(kBackwardThreads, 8) frame_backward_kernel(FrameArgs fa)
{
    extern __shared__ float4 sm[];
    __shared__ BackwardShared sh;
    __shared__ s3r_view view_sm;
    const uint32_t tid = threadIdx.y * blockDim.x + threadIdx.x;
    for (uint32_t i = tid; i < sizeof(s3r_view) / 4; i += kBackwardThreads)
        reinterpret_cast<uint32_t*>(&view_sm)[i] = reinterpret_cast<const uint32_t*>(fa.view)[i];
    __syncthreads();
    const s3r_view& v = view_sm;
    const TfTable tf = load_tf<false>(sm, fa.tf, v.tf_n, tid, kBackwardThreads);
    // The transfer-function gradient goes to one of kDtfParts copies in global
    // memory, an RGBA float4 reduction per table entry (fire and forget).  The copy
    // is picked by CTA (modulo kDtfCtaGroups) and by lane (modulo kDtfLaneGroups):
    // neighbouring rays -- neighbouring lanes -- add to the same entry at the same
    // time, and reductions on one address serialize.  (Shared-memory atomics
    // stalled the warps on exactly those collisions.)
    float4* dtf4 = reinterpret_cast<float4*>(fa.dtf_part) +
                   (size_t)(((blockIdx.y * gridDim.x + blockIdx.x) % kDtfCtaGroups) * kDtfLaneGroups +
                            (tid & 31) % kDtfLaneGroups) * v.tf_n;
    const uint32_t vx = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t vy = blockIdx.y * blockDim.y + threadIdx.y;
    if (vx >= v.W || vy >= v.H) return;
    float gC[3] = {0.f, 0.f, 0.f};
    float Q;
    {
        const size_t o = (size_t)(v.H - 1 - vy) * v.W + vx;
        const float4 I = reinterpret_cast<const float4*>(fa.fwd_rgba)[o];
        const float4 gI = reinterpret_cast<const float4*>(fa.dl_drgba)[o];
        const float A = I.w;
        float gA = gI.w;
        if (A > 0.f) {
            const float inv = 1.f / A;
            gC[0] = gI.x * inv;
            gC[1] = gI.y * inv;
            gC[2] = gI.z * inv;
            gA -= (gI.x * I.x + gI.y * I.y + gI.z * I.z) * inv;
        }
        if (gC[0] == 0.f && gC[1] == 0.f && gC[2] == 0.f && gA == 0.f) return;
        Q = gA * (1.f - A) - (gC[0] * (I.x * A) + gC[1] * (I.y * A) + gC[2] * (I.z * A));
    }
    {
        float org[3], dir[3], inv[3];
        pixel_ray(v, vx, vy, org, dir);
        ray_inverse(dir, inv);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            sh.ray[d][tid] = org[d];
            sh.ray[3 + d][tid] = dir[d];
            sh.ray[6 + d][tid] = inv[d];
        }
        BlockWalk w;
        if (!w.begin(org, dir, inv, v.level)) return;
        sh.walk[tid] = w;
    }
    const float inv_span = 1.f / (v.field_max - v.field_min);
    const float of = (v.threshold - v.field_min) / (v.field_max - v.field_min);
    float T = 1.f, accA = 0.f;
    int tf_j = -2; // the table interval of the two sums: entries max(j, 0) and min(j + 1, tf_n - 1); -2: none yet
    float tf_a[4] = {0.f, 0.f, 0.f, 0.f}, tf_b[4] = {0.f, 0.f, 0.f, 0.f};
    auto put_a = [&]() { atomicAdd(&dtf4[max(tf_j, 0)], make_float4(tf_a[0], tf_a[1], tf_a[2], tf_a[3])); };
    auto put_b = [&]() {
        atomicAdd(&dtf4[min(tf_j + 1, (int)v.tf_n - 1)], make_float4(tf_b[0], tf_b[1], tf_b[2], tf_b[3]));
    };
    while (true) {
        asm volatile("" ::: "memory"); // the walk is read back from shared memory, not kept in registers
        const RenderBlock* rb = &fa.table[sh.walk[tid].cell()];
        const uint32_t depth = rb->depth;
        const int4 rc = *reinterpret_cast<const int4*>(rb->rect);
        const int32_t rca[4] = {rc.x, rc.y, rc.z, rc.w};
        BlockRay r;
        bool hit = depth != 0xffffffffu && pixel_in_rect(rca, vx, vy);
        if (hit) {
            const float org[3] = {sh.ray[0][tid], sh.ray[1][tid], sh.ray[2][tid]};
            const float dir[3] = {sh.ray[3][tid], sh.ray[4][tid], sh.ray[5][tid]};
            const float inv[3] = {sh.ray[6][tid], sh.ray[7][tid], sh.ray[8][tid]};
            hit = block_ray(v, org, dir, inv, *rb, r);
        }
        if (hit) {
            const float* brick = reinterpret_cast<const float*>(fa.bricks) + rb->brick_off;
            float* gdense = fa.ddense + rb->brick_off;
            const float il = layer_exponent(depth, v.level, v.quality);
            float Ab = 0.f;
            CellGradient cg;
            cg.begin(r.step, gdense, (int)r.pitch, (int)(r.n * r.pitch));
            // one sample's gradients from its cell; false once the block is opaque
            auto step_sample = [&](const GradCell& cell) -> bool {
                float val;
                if (!filter_cell(cell.f, cell.t, val)) return true;
                // the forward's v01 up to the last ulp (a reciprocal instead of the division), and its colour
                const float u = __fmaf_rn(__fmul_rn(__fsub_rn(val, v.field_min), inv_span), (float)v.tf_n, -0.5f);
                int j;
                // the fraction of the clamped u: beyond the table the pair is one entry twice, and a fraction that grew with
                // the distance would leave the entry's gradient to the difference of two large sums (the product by
                // zero passes the NaN of an infinite value on, as the forward does)
                const float uc = fminf(fmaxf(u, -1.f), (float)v.tf_n - 0.5f);
                const float f = __fmaf_rn(0.f, u, uc) - floor_small(uc, j);
                const float4 p = tf.p[j + 1];
                float4 d;
                if (tf.d) {
                    d = tf.d[j + 1];
                } else {
                    const float4 q = tf.p[j + 2];
                    d = make_float4(q.x - p.x, q.y - p.y, q.z - p.z, q.w - p.w);
                }
                const float base = __fmaf_rn(-__fmaf_rn(f, d.w, p.w), of, 1.f);
                const float pw = __powf(base, il);
                const float a = __fsub_rn(1.f, pw);
                // derivatives need no correctly rounded divisions: fast reciprocals
                const float dadc = base > 0.f ? __fdividef(il * pw, base) * of : 0.f;
                const float wa = T * a;
                const float om = 1.f - a;
                const float inv_om = om > 1e-12f ? __fdividef(1.f, om) : 0.f;
                const float s = gC[0] * __fmaf_rn(f, d.x, p.x) + gC[1] * __fmaf_rn(f, d.y, p.y) +
                                gC[2] * __fmaf_rn(f, d.z, p.z);
                Q = __fmaf_rn(wa, s, Q);
                const float g_col[4] = {gC[0] * wa, gC[1] * wa, gC[2] * wa, (T * s + Q * inv_om) * dadc};
                // transfer-function table: accumulate the two entries of the current
                // interval in registers; when it changes, an entry that the new interval
                // shares (a ray moving to the next one) keeps its sum and only the other
                // one goes to memory
                if (j != tf_j) {
                    const bool up = j == tf_j + 1, down = j == tf_j - 1;
                    if (tf_j != -2) {
                        if (!down) put_a();
                        if (!up) put_b();
                    }
#pragma unroll
                    for (int ch = 0; ch < 4; ++ch) {
                        const float ta = tf_a[ch], tb = tf_b[ch];
                        tf_a[ch] = up ? tb : 0.f;
                        tf_b[ch] = down ? ta : 0.f;
                    }
                    tf_j = j;
                }
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    tf_a[ch] = __fmaf_rn(g_col[ch], 1.f - f, tf_a[ch]);
                    tf_b[ch] = __fmaf_rn(g_col[ch], f, tf_b[ch]);
                }
                // dense values; at the table's ends the colour does not depend on them
                if ((uint32_t)j < v.tf_n - 1) {
                    const float g_v01 = (g_col[0] * d.x + g_col[1] * d.y + g_col[2] * d.z + g_col[3] * d.w) *
                                        (float)v.tf_n;
                    const float g_val = g_v01 * inv_span;
                    if (g_val != 0.f) {
                        if (inside_brick(cell.a, r.n - 1)) {
                            cg.move(cell.a, gdense, r.n, r.pitch);
                            cg.add(g_val, cell.f);
                        } else {
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                const float w = ((q & 1) ? cell.f[0] : 1.f - cell.f[0]) *
                                                ((q & 2) ? cell.f[1] : 1.f - cell.f[1]) *
                                                ((q & 4) ? cell.f[2] : 1.f - cell.f[2]);
                                atomicAdd(&gdense[clamped_corner(cell.a, dim_of(r), q)], g_val * w);
                            }
                        }
                    }
                }
                T *= om;
                Ab = __fadd_rn(Ab, __fmul_rn(__fsub_rn(1.f, Ab), a));
                return !(Ab > kAlphaThreshold);
            };
            // software-pipelined as the forward march, unrolled by two with two
            // buffers: sample i's texels load while sample i-1's gradients form
            GradCell ca, cb;
            if (r.samples > 1) fetch_grad_cell(brick, r, 0, ca);
            const int last = r.samples - 1;
            for (int k = 1; k <= last;) {
                if (k < last) fetch_grad_cell(brick, r, k, cb);
                if (!step_sample(ca) || k >= last) break;
                ++k;
                if (k < last) fetch_grad_cell(brick, r, k, ca);
                if (!step_sample(cb)) break;
                ++k;
            }
            cg.put(0xffu);
            // block composite exactly as the forward kernel forms it
            accA = __fmaf_rn(__fsub_rn(1.f, accA), Ab, accA);
            if (accA > v.alpha_stop) break;
        }
        asm volatile("" ::: "memory");
        BlockWalk w = sh.walk[tid];
        if (!w.next()) break;
        sh.walk[tid] = w;
    }
    if (tf_j != -2) {
        put_a();
        put_b();
    }
}

// dtf[i] += the sum of its kDtfParts copies, one warp per entry-channel of 32 columns: lane l of warp w sums copies
// w, w + 8, ... of column i, so that reads stay coalesced and a column's 512 additions are 8 chains of 64.
__global__ void __launch_bounds__(256) dtf_reduce_kernel(const float* __restrict__ part, float* __restrict__ dtf, uint32_t n)
{
    __shared__ float sums[8][32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    float g = 0.f;
    if (i < n) {
#pragma unroll 8
        for (uint32_t p = w; p < kDtfParts; p += 8) g += part[(size_t)p * n + i];
    }
    sums[w][lane] = g;
    __syncthreads();
    if (w == 0 && i < n) {
        for (uint32_t q = 1; q < 8; ++q) g += sums[q][lane];
        dtf[i] += g;
    }
}

} // namespace

// The walk, the field modes and the per-block kernels take tables of up to kTfPlain entries: 48 KB of shared memory
// and the two repeated entries.  The launch refuses larger ones.
template <class K> cudaError_t allow_table(K kernel, size_t smem)
{
    if (smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(tf_smem_entries(kTfPlain, false) * sizeof(float4)));
}

// f(std::integral_constant<int, mode>) for a field mode known at run time.
template <class F> auto with_mode(uint32_t mode, F&& f)
{
    switch (mode) {
    case S3R_MODE_ISOSURFACE: return f(std::integral_constant<int, S3R_MODE_ISOSURFACE>());
    case S3R_MODE_ISOSURFACES: return f(std::integral_constant<int, S3R_MODE_ISOSURFACES>());
    case S3R_MODE_MAX_INTENSITY: return f(std::integral_constant<int, S3R_MODE_MAX_INTENSITY>());
    case S3R_MODE_ARGB: return f(std::integral_constant<int, S3R_MODE_ARGB>());
    case S3R_MODE_ARGB_LIGHT: return f(std::integral_constant<int, S3R_MODE_ARGB_LIGHT>());
    case S3R_MODE_DOMAIN_VOXELS: return f(std::integral_constant<int, S3R_MODE_DOMAIN_VOXELS>());
    case S3R_MODE_VALUE_ON_ISOSURFACE: return f(std::integral_constant<int, S3R_MODE_VALUE_ON_ISOSURFACE>());
    default: return f(std::integral_constant<int, S3R_MODE_VALUE_ON_ISOSURFACES>());
    }
}

inline s3r_presentation argb_presentation()
{
    s3r_presentation p{};
    p.mode = S3R_MODE_ARGB;
    return p;
}

cudaError_t launch_render_block_mode(const s3r_view* view_host, const s3r_presentation* pres, const float* brick,
                                     const float* brick2, const RenderBlock& rb, const float* tf, uint32_t* viewport,
                                     cudaStream_t s)
{
    if (rb.rect[2] <= 0 || rb.rect[3] <= 0) return cudaSuccess;
    const bool plain = !pres;
    const s3r_presentation argb = argb_presentation();
    if (plain) pres = &argb;
    dim3 block(16, 8);
    dim3 grid((rb.rect[2] + 15) / 16, (rb.rect[3] + 7) / 8);
    const size_t smem = tf_smem_entries(view_host->tf_n, false) * sizeof(float4);
    auto launch = [&](auto kernel) {
        const cudaError_t err = allow_table(kernel, smem);
        if (err != cudaSuccess) return err;
        kernel<<<grid, block, smem, s>>>(*view_host, *pres, brick, brick2, rb, tf, viewport);
        return cudaGetLastError();
    };
    const bool tex = view_host->filter == S3R_FILTER_TEXTURE;
    if (plain)
        return tex ? launch(render_block_mode_kernel<true, kPlainArgb>)
                   : launch(render_block_mode_kernel<false, kPlainArgb>);
    if (tex) return launch(render_block_mode_kernel<true, -1>);
    if (pres->mode == S3R_MODE_ARGB) return launch(render_block_mode_kernel<false, S3R_MODE_ARGB>);
    return launch(render_block_mode_kernel<false, -1>);
}

void part_tile(uint32_t mode, bool texture, uint32_t& w, uint32_t& h)
{
    // in memory: 8 x 4 pixels a warp, whose rays stay close together
    w = texture ? tex_tile_x(mode) : 8u;
    h = texture ? tex_tile_y(mode) : 16u;
}

cudaError_t launch_part(const s3r_view* view_host, const s3r_presentation* pres, const PartArgs& a, uint32_t ctas,
                        bool texture, uint32_t* viewport, cudaStream_t s)
{
    cudaError_t err = cudaMemsetAsync(a.count, 0, (size_t)a.w * a.h * sizeof(uint32_t), s);
    if (err != cudaSuccess || ctas == 0) return err;
    const bool plain = !pres && !texture;
    const s3r_presentation argb = argb_presentation();
    if (!pres) pres = &argb;
    uint32_t tw, th;
    part_tile(pres->mode, texture, tw, th);
    const dim3 block(tw, th);
    const size_t smem = texture ? 0 : tf_smem_entries(view_host->tf_n, false) * sizeof(float4);
    auto launch = [&](auto kernel) {
        const cudaError_t e = allow_table(kernel, smem);
        if (e != cudaSuccess) return e;
        kernel<<<ctas, block, smem, s>>>(*view_host, *pres, a);
        return cudaGetLastError();
    };
    const bool rule = view_host->filter == S3R_FILTER_TEXTURE;
    err = with_mode(pres->mode, [&](auto mode) {
        constexpr int m = decltype(mode)::value;
        if (plain) return rule ? launch(part_blocks_kernel<1, kPlainArgb>) : launch(part_blocks_kernel<0, kPlainArgb>);
        if (texture) return launch(part_blocks_kernel<2, m>);
        return view_host->filter != S3R_FILTER_TEXTURE ? launch(part_blocks_kernel<0, m>)
                                                       : launch(part_blocks_kernel<1, -1>);
    });
    if (err != cudaSuccess) return err;
    const bool multi = pres->mode == S3R_MODE_ISOSURFACES || pres->mode == S3R_MODE_VALUE_ON_ISOSURFACES;
    const uint32_t kind = pres->mode == S3R_MODE_MAX_INTENSITY ? ModeOut::kMax
                          : multi && pres->level_count < 1     ? ModeOut::kClear
                                                               : ModeOut::kBlend;
    const uint64_t npix = (uint64_t)a.w * a.h;
    part_composite_kernel<<<(uint32_t)((npix + kCompositeThreads - 1) / kCompositeThreads), kCompositeThreads,
                            a.cap * kCompositeThreads * sizeof(uint32_t), s>>>(a, viewport, view_host->W, view_host->H,
                                                                               kind);
    return cudaGetLastError();
}

cudaError_t launch_render_block_texture(const s3r_view* view_host, const s3r_presentation* pres, uint64_t field,
                                       uint64_t field2, uint64_t tf_tex, const RenderBlock& rb, uint32_t* viewport,
                                       cudaStream_t s)
{
    if (rb.rect[2] <= 0 || rb.rect[3] <= 0) return cudaSuccess;
    const uint32_t tx = tex_tile_x(pres->mode), ty = tex_tile_y(pres->mode);
    dim3 block(tx, ty);
    dim3 grid((rb.rect[2] + tx - 1) / tx, (rb.rect[3] + ty - 1) / ty);
    const TextureSampler smp{(cudaTextureObject_t)field, (cudaTextureObject_t)field2, (cudaTextureObject_t)tf_tex};
    with_mode(pres->mode, [&](auto mode) {
        render_block_texture_kernel<decltype(mode)::value><<<grid, block, 0, s>>>(*view_host, *pres, smp, rb, viewport);
    });
    return cudaGetLastError();
}

template <int Fmt, bool kTex>
cudaError_t launch_frame_render_fmt(const FrameArgs& a, dim3 grid, dim3 block, size_t smem, uint32_t R, cudaStream_t s)
{
    auto launch = [&](auto kernel) {
        const cudaError_t err = allow_table(kernel, smem);
        if (err != cudaSuccess) return err;
        kernel<<<grid, block, smem, s>>>(a);
        return cudaGetLastError();
    };
    switch (R) {
    case 1: return launch(frame_render_kernel<Fmt, 1, kTex>);
    case 2: return launch(frame_render_kernel<Fmt, 2, kTex>);
    case 4: return launch(frame_render_kernel<Fmt, 4, kTex>);
    default: return launch(frame_render_kernel<Fmt, 8, kTex>);
    }
}

cudaError_t launch_frame_render(const FrameArgs& a, uint32_t W, uint32_t H, uint32_t tf_n, uint32_t fmt,
                                uint32_t tile_shape, uint32_t filter, cudaStream_t s)
{
    // tile_shape: CTA pixel shape (low 2 bits) and lanes per ray R = 2^(bits 2-3)
    const uint32_t shape = tile_shape % kRenderShapes;
    const uint32_t R = 1u << ((tile_shape / kRenderShapes) % 4);
    const int sx = kRenderShapeX[shape], sy = kRenderShapeY[shape];
    // R lanes per pixel: keep 128-ish threads per CTA by narrowing the pixel tile
    const int px = sx / (int)R > 0 ? sx / (int)R : 1;
    dim3 block(px * R, sy);
    dim3 grid((W + px - 1) / px, (H + sy - 1) / sy);
    const size_t smem = tf_smem_entries(tf_n, false) * sizeof(float4);
    const bool tex = filter == S3R_FILTER_TEXTURE;
    switch (fmt) {
    case S3R_BRICK_F32:
        return tex ? launch_frame_render_fmt<S3R_BRICK_F32, true>(a, grid, block, smem, R, s)
                   : launch_frame_render_fmt<S3R_BRICK_F32, false>(a, grid, block, smem, R, s);
    case S3R_BRICK_F16:
        return tex ? launch_frame_render_fmt<S3R_BRICK_F16, true>(a, grid, block, smem, R, s)
                   : launch_frame_render_fmt<S3R_BRICK_F16, false>(a, grid, block, smem, R, s);
    case S3R_BRICK_BF16:
        return tex ? launch_frame_render_fmt<S3R_BRICK_BF16, true>(a, grid, block, smem, R, s)
                   : launch_frame_render_fmt<S3R_BRICK_BF16, false>(a, grid, block, smem, R, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int Fmt, bool kTex>
cudaError_t launch_frame_segments_fmt(const FrameArgs& a, const SegArgs& sa, uint32_t fx, dim3 block, size_t smem,
                                      uint32_t sms, cudaStream_t s)
{
    auto kernel = sa.lanes ? frame_segments_kernel<Fmt, kTex, true> : frame_segments_kernel<Fmt, kTex, false>;
    if (smem > 48 * 1024) {
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return err;
    }
    int per_sm = 0;
    cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)(block.x * block.y), smem);
    if (err != cudaSuccess) return err;
    kernel<<<sms * (uint32_t)(per_sm > 0 ? per_sm : 1), block, smem, s>>>(a, sa, fx);
    return cudaGetLastError();
}

cudaError_t launch_frame_segments(const FrameArgs& a, const SegArgs& sa, uint32_t W, uint32_t H, uint32_t tf_n,
                                  uint32_t fmt, uint32_t shape, uint32_t filter, uint32_t sms, cudaStream_t s)
{
    if (sa.words > kSegMaskWords) return cudaErrorInvalidValue;
    shape %= kSegShapes;
    const uint32_t fx = (uint32_t)kSegShapeX[shape];
    const dim3 block(kSegThreads);
    const size_t smem = tf_smem_entries(tf_n, true) * sizeof(float4);
    const bool tex = filter == S3R_FILTER_TEXTURE;
    cudaError_t err;
    switch (fmt) {
    case S3R_BRICK_F32:
        err = tex ? launch_frame_segments_fmt<S3R_BRICK_F32, true>(a, sa, fx, block, smem, sms, s)
                  : launch_frame_segments_fmt<S3R_BRICK_F32, false>(a, sa, fx, block, smem, sms, s);
        break;
    case S3R_BRICK_F16:
        err = tex ? launch_frame_segments_fmt<S3R_BRICK_F16, true>(a, sa, fx, block, smem, sms, s)
                  : launch_frame_segments_fmt<S3R_BRICK_F16, false>(a, sa, fx, block, smem, sms, s);
        break;
    case S3R_BRICK_BF16:
        err = tex ? launch_frame_segments_fmt<S3R_BRICK_BF16, true>(a, sa, fx, block, smem, sms, s)
                  : launch_frame_segments_fmt<S3R_BRICK_BF16, false>(a, sa, fx, block, smem, sms, s);
        break;
    default: return cudaErrorInvalidValue;
    }
    if (err != cudaSuccess) return err;
    const uint64_t npix = (uint64_t)W * H;
    frame_composite_kernel<<<(uint32_t)((npix + 255) / 256), 256, 0, s>>>(a, sa);
    return cudaGetLastError();
}

cudaError_t launch_seg_items(const uint2* list, uint32_t nblocks, uint2* items, cudaStream_t s)
{
    if (nblocks) seg_items_kernel<<<nblocks, 128, 0, s>>>(list, items);
    return cudaGetLastError();
}

cudaError_t launch_frame_render_mode(const FrameArgs& a, const s3r_presentation& pres, const float* bricks2,
                                     uint32_t W, uint32_t H, uint32_t tf_n, uint32_t filter, cudaStream_t s)
{
    const dim3 block(8, 16); // 8 x 4 pixels a warp
    const dim3 grid((W + 7) / 8, (H + 15) / 16);
    const size_t smem = tf_smem_entries(tf_n, false) * sizeof(float4);
    auto launch = [&](auto kernel) {
        const cudaError_t err = allow_table(kernel, smem);
        if (err != cudaSuccess) return err;
        kernel<<<grid, block, smem, s>>>(a, pres, bricks2);
        return cudaGetLastError();
    };
    return with_mode(pres.mode, [&](auto mode) {
        constexpr int m = decltype(mode)::value;
        return filter == S3R_FILTER_TEXTURE ? launch(frame_render_mode_kernel<true, m>)
                                            : launch(frame_render_mode_kernel<false, m>);
    });
}

cudaError_t launch_frame_backward(const FrameArgs& a, uint32_t W, uint32_t H, uint32_t tf_n, cudaStream_t s)
{
    // 16x4-pixel CTAs, 16x2 pixels a warp.  8 blocks of depth 6 at 512x512: long transparent rays take 254 us with 8x8
    // (8x4 a warp: its rays share most of the cells they add to), 264 with this, 274 with 32x2; rays that end early in
    // opaque blocks 201, 186 and 188 us, where 32x2 with eight reductions a sample took 199 (342 for the long rays)
    dim3 block(16, 4);
    dim3 grid((W + 15) / 16, (H + 3) / 4);
    const size_t smem = tf_smem_entries(tf_n, false) * sizeof(float4);
    if (smem + sizeof(BackwardShared) > 47 * 1024) {
        cudaError_t err =
            cudaFuncSetAttribute(frame_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return err;
    }
    frame_backward_kernel<<<grid, block, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_dtf_reduce(const float* part, float* dtf, uint32_t n, cudaStream_t s)
{
    dtf_reduce_kernel<<<(n + 31) / 32, 256, 0, s>>>(part, dtf, n);
    return cudaGetLastError();
}

} // namespace s3r
