// Device code of the tile interpolation (the hierarchical midpoint fill of one tile in shared memory and
// its finest level written to HBM), kept apart from the kernels (interp.cu) so that another kernel can run
// tiles too.  See interp.cu for the algorithm and its reference.
#pragma once

#include "s3r_internal.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

namespace s3r {
namespace {

constexpr float kHalf = 0.5f;
constexpr float kQuarter = 0.25f;
constexpr float kSixth = (float)(1.0 / 6.0);

__device__ __forceinline__ float qnan() { return __int_as_float(0x7fc00000); }

// put(): v may be +inf (internal no-field) or NaN; put_nan(): v is already NaN
// wherever it is masked (see inf_to_nan), so the float store needs no test.
template <typename OutT> struct Store;
template <> struct Store<float> {
    __device__ static void put(float* out, uint64_t i, float v, float, float)
    {
        out[i] = isinf(v) ? qnan() : v;
    }
    __device__ static void put_nan(float* out, uint64_t i, float v, float, float) { out[i] = v; }
};
template <> struct Store<__half> {
    __device__ static void put(__half* out, uint64_t i, float v, float inv_scale, float offset)
    {
        out[i] = (isinf(v) || isnan(v)) ? __ushort_as_half((unsigned short)0x7e00)
                                             : __float2half_rn((v - offset) * inv_scale);
    }
    __device__ static void put_nan(__half* out, uint64_t i, float v, float inv_scale, float offset)
    {
        out[i] = isnan(v) ? __ushort_as_half((unsigned short)0x7e00) : __float2half_rn((v - offset) * inv_scale);
    }
};
template <> struct Store<__nv_bfloat16> {
    __device__ static void put(__nv_bfloat16* out, uint64_t i, float v, float inv_scale, float offset)
    {
        out[i] = (isinf(v) || isnan(v)) ? __ushort_as_bfloat16((unsigned short)0x7fc0)
                                             : __float2bfloat16_rn((v - offset) * inv_scale);
    }
    __device__ static void put_nan(__nv_bfloat16* out, uint64_t i, float v, float inv_scale, float offset)
    {
        out[i] = isnan(v) ? __ushort_as_bfloat16((unsigned short)0x7fc0)
                          : __float2bfloat16_rn((v - offset) * inv_scale);
    }
};

// Two vertices adjacent along x, already NaN where masked, in one aligned store
// (the pair starts at an even x of a row whose pitch keeps it aligned).
template <typename OutT> struct Store2;
template <> struct Store2<float> {
    __device__ static void put_nan(float* out, float v0, float v1, float, float)
    {
        *reinterpret_cast<float2*>(out) = make_float2(v0, v1);
    }
};
// 16-bit pairs: (v - offset) / scale as one FMA per value and one paired conversion;
// a NaN stays NaN through both.
template <> struct Store2<__half> {
    __device__ static void put_nan(__half* out, float v0, float v1, float inv_scale, float offset)
    {
        const float c = -offset * inv_scale;
        *reinterpret_cast<__half2*>(out) = __floats2half2_rn(__fmaf_rn(v0, inv_scale, c), __fmaf_rn(v1, inv_scale, c));
    }
};
template <> struct Store2<__nv_bfloat16> {
    __device__ static void put_nan(__nv_bfloat16* out, float v0, float v1, float inv_scale, float offset)
    {
        const float c = -offset * inv_scale;
        *reinterpret_cast<__nv_bfloat162*>(out) =
            __floats2bfloat162_rn(__fmaf_rn(v0, inv_scale, c), __fmaf_rn(v1, inv_scale, c));
    }
};

// +inf -> NaN in one FFMA, every other value (-0 included) unchanged:
// 0 * v is +-0 for finite v (the sign of v, so v + 0 * v == v exactly) and NaN
// for infinite v.
__device__ __forceinline__ float inf_to_nan(float v) { return __fmaf_rn(0.f, v, v); }

// Internally a masked value is +inf: every stencil sum that touches it is
// +inf, which reproduces the reference's rule "any no-field value in the
// stencil gives the no-field value" without tests, and finite sums round as
// before.  NaN keeps its meaning "not computed yet".
__device__ __forceinline__ float to_internal(float v) { return v == kNoField ? __int_as_float(0x7f800000) : v; }

// Coarse levels above a tile of 2^kGridTileLog2 cells.
constexpr uint32_t kMaxGridLevels = S3R_MAX_DEPTH - kGridTileLog2;

// The threads that run one tile: a CTA of kInterpThreads (kN = kInterpThreads, CTA barriers) or one warp
// (kN = 32, warp barriers; the warp-per-tile kernel for tiles of up to 8 cells).  tid is the thread's
// index among them.
template <uint32_t kN> struct Crew {
    uint32_t tid;
    __device__ __forceinline__ void sync() const
    {
        if constexpr (kN == 32) __syncwarp();
        else __syncthreads();
    }
};

// One 27-point level held in registers: lane p < 27 holds point p (x fastest)
// of a cube -- the 8 corners known, each midpoint its sparse value or NaN --
// and gets it filled: edges from their two ends, faces from their four edges,
// the centre from its six faces, the stencil sums in the reference's order.
// Neighbours come by shuffle, so no shared memory and no __syncwarp.
__device__ __forceinline__ float level27(float v, uint32_t lane)
{
    const uint32_t px = lane % 3, py = (lane / 3) % 3, pz = lane / 9;
    const uint32_t nodd = lane < 27 ? (px & 1) + (py & 1) + (pz & 1) : 3u;
    {
        const bool mine = nodd == 1;
        const uint32_t st = (px & 1) ? 1 : ((py & 1) ? 3 : 9);
        const float lo = __shfl_sync(0xffffffffu, v, mine ? lane - st : lane);
        const float hi = __shfl_sync(0xffffffffu, v, mine ? lane + st : lane);
        if (mine && isnan(v)) v = kHalf * (lo + hi);
    }
    {
        const bool mine = nodd == 2;
        const uint32_t s1 = (px & 1) ? 1 : 3; // the two odd axes, ascending
        const uint32_t s2 = (pz & 1) ? 9 : 3;
        const float a = __shfl_sync(0xffffffffu, v, mine ? lane - s1 : lane);
        const float b = __shfl_sync(0xffffffffu, v, mine ? lane + s1 : lane);
        const float c = __shfl_sync(0xffffffffu, v, mine ? lane - s2 : lane);
        const float d = __shfl_sync(0xffffffffu, v, mine ? lane + s2 : lane);
        if (mine && isnan(v)) v = kQuarter * (a + b + c + d);
    }
    {
        const float f12 = __shfl_sync(0xffffffffu, v, 12), f14 = __shfl_sync(0xffffffffu, v, 14);
        const float f10 = __shfl_sync(0xffffffffu, v, 10), f16 = __shfl_sync(0xffffffffu, v, 16);
        const float f4 = __shfl_sync(0xffffffffu, v, 4), f22 = __shfl_sync(0xffffffffu, v, 22);
        if (lane == 13 && isnan(v)) v = kSixth * (f12 + f14 + f10 + f16 + f4 + f22);
    }
    return v;
}

// One warp, all lanes: walk from the block's root corners down L levels to the
// tile's cube, each level's 27 points in registers (level27) with the sparse
// values from known(l, gx, gy, gz) (NaN where no node; at levels below the root
// the corner points come from the level above).  Lanes 0-7 return the tile's 8
// corners (lane & 1, lane >> 1 & 1, lane >> 2).
template <class Known>
__device__ __forceinline__ float descend_regs(uint32_t d, uint32_t L, uint32_t ox, uint32_t oy, uint32_t oz,
                                              uint32_t lane, Known&& known)
{
    const uint32_t px = lane % 3, py = (lane / 3) % 3, pz = lane / 9;
    const bool is_corner = lane < 27 && !((px | py | pz) & 1);
    const uint32_t from = is_corner ? (px >> 1) + 2 * (py >> 1) + 4 * (pz >> 1) : lane;
    // every level's values first: their loads are independent of one another
    float val[kMaxGridLevels];
#pragma unroll
    for (uint32_t l = 0; l < kMaxGridLevels; ++l) {
        val[l] = 0.f;
        if (l < L && lane < 27) {
            const uint32_t size = 1u << (d - l), hs = size >> 1;
            val[l] = known((ox & ~(size - 1)) + hs * px, (oy & ~(size - 1)) + hs * py, (oz & ~(size - 1)) + hs * pz);
        }
    }
    uint32_t size = 1u << d, gx0 = 0, gy0 = 0, gz0 = 0;
    float corner = 0.f;
#pragma unroll
    for (uint32_t l = 0; l < kMaxGridLevels; ++l) {
        if (l >= L) break;
        float v = val[l];
        if (l > 0) {
            const float cv = __shfl_sync(0xffffffffu, corner, from);
            if (is_corner) v = cv;
        }
        v = level27(v, lane);
        const uint32_t hs = size >> 1;
        const uint32_t qx = (ox - gx0) >= hs ? 1u : 0u;
        const uint32_t qy = (oy - gy0) >= hs ? 1u : 0u;
        const uint32_t qz = (oz - gz0) >= hs ? 1u : 0u;
        const uint32_t pick =
            lane < 8 ? (qx + (lane & 1)) + 3 * (qy + ((lane >> 1) & 1)) + 9 * (qz + (lane >> 2)) : lane;
        corner = __shfl_sync(0xffffffffu, v, pick);
        gx0 += qx * hs;
        gy0 += qy * hs;
        gz0 += qz * hs;
        size = hs;
    }
    return corner;
}

// One level of one tile: every cube of the level (2^j per axis) is handled by
// one thread, which reads its 27 points (8 corners known from the coarser
// levels, 19 midpoints holding a sparse value or NaN), fills the NaN midpoints
// in registers (edges, then faces, then the centre) and writes back the
// midpoints it owns: those with every coordinate on the cube's low side or
// middle, plus the far side where the cube is the last along that axis.
// Midpoints shared with a neighbour are computed by both from the same values,
// so a neighbour reading one while it is written reads the same number.
__device__ __forceinline__ void cube_level(float* s, uint32_t E, uint32_t T, uint32_t j)
{
    const uint32_t m = 1u << j, sz = T >> j, hs = sz >> 1;
    const uint32_t st0 = hs, st1 = E * hs, st2 = E * E * hs;
    const uint32_t ncubes = 1u << (3 * j);
#pragma unroll 1
    for (uint32_t c = threadIdx.x; c < ncubes; c += blockDim.x) {
        const uint32_t ci = c & (m - 1), cj = (c >> j) & (m - 1), ck = c >> (2 * j);
        const uint32_t base = ci * sz + E * (cj * sz + E * (ck * sz));
        float v[27];
#pragma unroll
        for (int p = 0; p < 27; ++p) v[p] = s[base + (p % 3) * st0 + ((p / 3) % 3) * st1 + (p / 9) * st2];
#pragma unroll
        for (int p = 0; p < 27; ++p) {
            const int a = p % 3, b = (p / 3) % 3, cc = p / 9;
            if ((a & 1) + (b & 1) + (cc & 1) == 1 && isnan(v[p])) {
                const int st = (a & 1) ? 1 : ((b & 1) ? 3 : 9);
                v[p] = kHalf * (v[p - st] + v[p + st]);
            }
        }
#pragma unroll
        for (int p = 0; p < 27; ++p) {
            const int a = p % 3, b = (p / 3) % 3, cc = p / 9;
            if ((a & 1) + (b & 1) + (cc & 1) == 2 && isnan(v[p])) {
                const int s1 = (a & 1) ? 1 : 3;
                const int s2 = (cc & 1) ? 9 : 3;
                v[p] = kQuarter * (v[p - s1] + v[p + s1] + v[p - s2] + v[p + s2]);
            }
        }
        if (isnan(v[13])) v[13] = kSixth * (v[12] + v[14] + v[10] + v[16] + v[4] + v[22]);
        const bool lx = ci == m - 1, ly = cj == m - 1, lz = ck == m - 1;
#pragma unroll
        for (int p = 0; p < 27; ++p) {
            const int a = p % 3, b = (p / 3) % 3, cc = p / 9;
            if ((a & 1) + (b & 1) + (cc & 1) == 0) continue;
            if ((a < 2 || lx) && (b < 2 || ly) && (cc < 2 || lz))
                s[base + a * st0 + b * st1 + cc * st2] = v[p];
        }
    }
}

// Shared tile of (2^k+1)^3 floats, rounded up to whole float4s for the vector fill.
inline size_t tile_smem_bytes(uint32_t tile_log2)
{
    const size_t E = (1u << tile_log2) + 1u;
    return ((E * E * E + 3) / 4) * 16;
}

// Parity-split layout of a tile of T cells (T even): vertex (x, y, z) lives in
// sub-array c = (x&1) | (y&1)<<1 | (z&1)<<2 at (x>>1) + nx*((y>>1) + ny*(z>>1)),
// with nx = T/2 along an odd axis and T/2+1 along an even one.  At the finest
// level every class of midpoints then sits in its own dense array, so a warp
// walking one class touches consecutive words (no bank conflicts), and the
// even sub-array is the same problem at half resolution for the coarser levels.
template <uint32_t T> struct SplitTile {
    static constexpr uint32_t H = T / 2, G = T / 2 + 1;
    __host__ __device__ static constexpr uint32_t n(uint32_t odd) { return odd ? H : G; }
    __host__ __device__ static constexpr uint32_t size(uint32_t c) { return n(c & 1) * n((c >> 1) & 1) * n((c >> 2) & 1); }
    // sum of the sizes of classes 0 .. c-1 (sizes G^3, HG^2, HG^2, H^2G, HG^2, H^2G, H^2G, H^3)
    __host__ __device__ static constexpr uint32_t base(uint32_t c)
    {
        constexpr uint32_t G3 = G * G * G, HG2 = H * G * G, H2G = H * H * G;
        return (c >= 1 ? G3 : 0) + (c >= 2 ? HG2 : 0) + (c >= 3 ? HG2 : 0) + (c >= 4 ? H2G : 0) +
               (c >= 5 ? HG2 : 0) + (c >= 6 ? H2G : 0) + (c >= 7 ? H2G : 0);
    }
    // element (i, j, k) of class c
    __host__ __device__ static constexpr uint32_t idx(uint32_t c, uint32_t i, uint32_t j, uint32_t k)
    {
        return base(c) + i + n(c & 1) * (j + n((c >> 1) & 1) * k);
    }
    __host__ __device__ static constexpr uint32_t at(uint32_t x, uint32_t y, uint32_t z)
    {
        return idx((x & 1) | ((y & 1) << 1) | ((z & 1) << 2), x >> 1, y >> 1, z >> 1);
    }
};

// The first warp of the tile's threads, T >= 4: the tile cube's 27 points (corners at 0 and T, midpoints at
// T/2) from its corners and the sparse values already in the tile -- the
// tile's first level, cube_level on its single cube, in registers.
template <uint32_t T> __device__ __forceinline__ void tile_top(float* s, uint32_t lane)
{
    using S = SplitTile<T>;
    const uint32_t px = lane % 3, py = (lane / 3) % 3, pz = lane / 9;
    constexpr uint32_t h = T / 2;
    const uint32_t off = lane < 27 ? S::at(px * h, py * h, pz * h) : 0;
    float v = lane < 27 ? s[off] : 0.f;
    v = level27(v, lane);
    if (lane < 27 && ((px | py | pz) & 1)) s[off] = v;
}

// The 19 midpoints of one 2x2x2 cube from its 8 corners (v[p], p = a + 3b + 9c,
// a, b, c in {0, 1, 2}); kSlots: v also holds sparse values (or NaN) at the
// midpoints, which are kept.  Edges, then faces, then the centre, stencil sums
// in the reference's order.  kLowZDone: the cube's z = 0 face is final already
// (the z = 2 face of the cube below it), only the points above it are filled.
template <bool kSlots, bool kLowZDone = false> __device__ __forceinline__ void fill_cube(float v[27])
{
#pragma unroll
    for (int p = 0; p < 27; ++p) {
        const int a = p % 3, b = (p / 3) % 3, cc = p / 9;
        if (kLowZDone && cc == 0) continue;
        if ((a & 1) + (b & 1) + (cc & 1) == 1 && (!kSlots || isnan(v[p]))) {
            const int st = (a & 1) ? 1 : ((b & 1) ? 3 : 9);
            v[p] = kHalf * (v[p - st] + v[p + st]);
        }
    }
#pragma unroll
    for (int p = 0; p < 27; ++p) {
        const int a = p % 3, b = (p / 3) % 3, cc = p / 9;
        if (kLowZDone && cc == 0) continue;
        if ((a & 1) + (b & 1) + (cc & 1) == 2 && (!kSlots || isnan(v[p]))) {
            const int s1 = (a & 1) ? 1 : 3;
            const int s2 = (cc & 1) ? 9 : 3;
            v[p] = kQuarter * (v[p - s1] + v[p + s1] + v[p - s2] + v[p + s2]);
        }
    }
    if (!kSlots || isnan(v[13])) v[13] = kSixth * (v[12] + v[14] + v[10] + v[16] + v[4] + v[22]);
}

// cube_level with the grid stride, tile size and level known at compile time (the coarse levels
// inside a tile): the 27 point offsets become immediates and the cube loop is unrolled.
template <uint32_t E, uint32_t T, uint32_t J, uint32_t kN>
__device__ __forceinline__ void cube_level_ct(float* s, uint32_t tid)
{
    constexpr uint32_t m = 1u << J, sz = T >> J, hs = sz >> 1;
    constexpr uint32_t st0 = hs, st1 = E * hs, st2 = E * E * hs;
    constexpr uint32_t ncubes = 1u << (3 * J);
#pragma unroll
    for (uint32_t c0 = 0; c0 < ncubes; c0 += kN) {
        const uint32_t c = c0 + tid;
        if (ncubes % kN != 0 && c >= ncubes) break;
        const uint32_t ci = c & (m - 1), cj = (c >> J) & (m - 1), ck = c >> (2 * J);
        const uint32_t base = ci * sz + E * (cj * sz + E * (ck * sz));
        float v[27];
#pragma unroll
        for (int p = 0; p < 27; ++p) v[p] = s[base + (p % 3) * st0 + ((p / 3) % 3) * st1 + (p / 9) * st2];
        fill_cube<true>(v);
        const bool lx = ci == m - 1, ly = cj == m - 1, lz = ck == m - 1;
#pragma unroll
        for (int p = 0; p < 27; ++p) {
            const int a = p % 3, b = (p / 3) % 3, cc = p / 9;
            if ((a & 1) + (b & 1) + (cc & 1) == 0) continue;
            if ((a < 2 || lx) && (b < 2 || ly) && (cc < 2 || lz)) s[base + a * st0 + b * st1 + cc * st2] = v[p];
        }
    }
}

// The coarse levels 1 .. K-2 of a tile of T = 2^K cells on its even sub-array (G^3, a tile of T/2 cells).
template <uint32_t G, uint32_t H, uint32_t J, uint32_t K, uint32_t kN>
__device__ __forceinline__ void tile_levels(float* s, Crew<kN> cw)
{
    if constexpr (J + 1 < K) {
        cube_level_ct<G, H, J, kN>(s, cw.tid);
        cw.sync();
        tile_levels<G, H, J + 1, K, kN>(s, cw);
    }
}

// Where a tile's finest level goes, masked values already NaN.  row: the cube's row (b, cc) of vertices, of which
// v0 and v1 (x = 0, 1) are its own and v2 is the next cube's first; far_x: v2 of the block's last cube along x;
// up: on to the next cube along z.
//
// A plan brick: rows padded to whole sectors, so a row's two vertices of a cube go out as one aligned store.
template <typename OutT, bool kSector> struct BrickCursor {
    OutT* p;
    uint32_t e, pitch, e2;
    float inv_scale, offset;
    __device__ __forceinline__ void row(uint32_t b, uint32_t cc, float v0, float v1, float) const
    {
        Store2<OutT>::put_nan(p + b * pitch + cc * e2, v0, v1, inv_scale, offset);
    }
    __device__ __forceinline__ void far_x(uint32_t b, uint32_t cc, float v) const
    {
        if constexpr (std::is_same<OutT, float>::value && kSector) {
            if (pitch >= e + 7) {
                // a padded brick (plan layout, d >= 3): x = 2^d starts a sector of its own
                // (rows are 32-byte aligned, 2^d is a multiple of 8, the pitch is 2^d + 8):
                // write the whole sector, the padding as NaN
                float4* q = reinterpret_cast<float4*>(p + 2 + b * pitch + cc * e2);
                q[0] = make_float4(v, qnan(), qnan(), qnan());
                q[1] = make_float4(qnan(), qnan(), qnan(), qnan());
                return;
            }
        }
        Store<OutT>::put_nan(p, 2 + b * pitch + cc * e2, v, inv_scale, offset);
    }
    __device__ __forceinline__ void up() { p += 2 * e2; }
};
// A plain (2^d+1)^3 grid: its rows are of odd length, so every other one starts in the middle of an 8-byte word.  In
// those the cube stores v1 and v2 -- which the next cube, whose own first vertex v2 is, then leaves to it -- and the
// row's first cube v0 besides, so that all rows go out in aligned pairs.
struct GridCursor {
    float* p;
    uint32_t e, e2;
    uint32_t odd;   // 1: the cube's first row starts in the middle of an 8-byte word
    bool first;     // the block's first cube along x
    __device__ __forceinline__ void row(uint32_t b, uint32_t cc, float v0, float v1, float v2) const
    {
        float* q = p + b * e + cc * e2;
        if ((b + cc + odd) & 1) {
            if (first) q[0] = v0;
            *reinterpret_cast<float2*>(q + 1) = make_float2(v1, v2);
        } else {
            *reinterpret_cast<float2*>(q) = make_float2(v0, v1);
        }
    }
    __device__ __forceinline__ void far_x(uint32_t b, uint32_t cc, float v) const
    {
        if (!((b + cc + odd) & 1)) p[2 + b * e + cc * e2] = v;
    }
    __device__ __forceinline__ void up() { p += 2 * e2; }
};
// A 3-D texture array, written in place through its surface: no linear grid and no copy into the array.
struct SurfaceCursor {
    cudaSurfaceObject_t s;
    int x, y, z;
    __device__ __forceinline__ void row(uint32_t b, uint32_t cc, float v0, float v1, float) const
    {
        surf3Dwrite(make_float2(v0, v1), s, x * 4, y + (int)b, z + (int)cc);
    }
    __device__ __forceinline__ void far_x(uint32_t b, uint32_t cc, float v) const
    {
        surf3Dwrite(v, s, (x + 2) * 4, y + (int)b, z + (int)cc);
    }
    __device__ __forceinline__ void up() { z += 2; }
};

// One finest-level cube (ci, cj, ck) of a tile: reads its corners from the even
// sub-array -- kFirst: all 8; else the upper 4, its z = 0 face being the z = 2
// face of the cube below it, already in v -- and, when flagged as holding a
// sparse midpoint, its midpoint slots (above the z = 0 face unless kFirst);
// computes its midpoints in registers and stores the vertices it owns: its low
// octant, plus the far side where it is the last cube of the block along an
// axis, with the 16-bit encoding fused into the store.  Masked corners become
// NaN as they are loaded, so unflagged cubes produce NaN directly (a NaN in a
// stencil sum gives NaN as +inf gives +inf); flagged cubes test their slots for
// NaN ("no sparse value") before any slot is overwritten, then turn masked
// sparse values to NaN.  A reused face went through the same steps in the cube
// below, so every vertex gets the value a fresh cube would give it.
template <uint32_t T, bool kFirst, class Cur>
__device__ __forceinline__ void finest_cube(const float* s, bool has, uint32_t ci, uint32_t cj, uint32_t ck, float v[27],
                                            const Cur& cur, bool lx, bool ly, bool lz)
{
    using S = SplitTile<T>;
#pragma unroll
    for (int p = 0; p < 27; ++p) {
        const uint32_t a = p % 3, b = (p / 3) % 3, cc = p / 9;
        if (!kFirst && cc < 2) continue;
        if (!((a | b | cc) & 1)) v[p] = inf_to_nan(s[S::idx(0, ci + (a >> 1), cj + (b >> 1), ck + (cc >> 1))]);
    }
    if (has) {
#pragma unroll
        for (int p = 0; p < 27; ++p) {
            const uint32_t a = p % 3, b = (p / 3) % 3, cc = p / 9;
            if (!kFirst && cc == 0) continue;
            const uint32_t cls = (a & 1) | ((b & 1) << 1) | ((cc & 1) << 2);
            if (cls) v[p] = s[S::idx(cls, ci + (a >> 1), cj + (b >> 1), ck + (cc >> 1))];
        }
        fill_cube<true, !kFirst>(v);
#pragma unroll
        for (int p = 0; p < 27; ++p) {
            if (!kFirst && p / 9 == 0) continue;
            if ((p % 3) & 1 || ((p / 3) % 3) & 1 || (p / 9) & 1) v[p] = inf_to_nan(v[p]);
        }
    } else {
        fill_cube<false, !kFirst>(v);
    }
    auto row = [&](uint32_t b, uint32_t cc) {
        const int p = 3 * (int)b + 9 * (int)cc;
        cur.row(b, cc, v[p], v[p + 1], v[p + 2]);
    };
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) row(r & 1, r >> 1);
    // the far side where this is the block's last cube along an axis: the x = 2 face (with its
    // y = 2 / z = 2 edges where those are far too), then y = 2 (x < 2), then z = 2 (x, y < 2)
    if (lx) {
#pragma unroll
        for (uint32_t b = 0; b < 3; ++b)
#pragma unroll
            for (uint32_t cc = 0; cc < 3; ++cc)
                if ((b < 2 || ly) && (cc < 2 || lz)) cur.far_x(b, cc, v[2 + 3 * b + 9 * cc]);
    }
    if (ly) {
        row(2, 0);
        row(2, 1);
        if (lz) row(2, 2);
    }
    if (lz) {
        row(0, 2);
        row(1, 2);
    }
}

// The finest level of a tile, written straight to its place: its H^3 2x2x2 cubes in
// runs of Z along z, one run per thread (runs consecutive along x within a
// warp), so that each cube after the first of a run takes its z = 0 face from
// the one below; Z makes the runs about as many as the tile's threads (kN).
// at(x, y, z): the cursor of the cube whose low corner is vertex (x, y, z) of the tile.
template <uint32_t T, uint32_t kN, class At>
__device__ __forceinline__ void finest_store(const float* s, const uint32_t* flags, bool far_x, bool far_y, bool far_z,
                                             uint32_t tid, At&& at)
{
    using S = SplitTile<T>;
    constexpr uint32_t H = S::H;
    constexpr uint32_t lh = (H >= 2) ? (31 - __builtin_clz(H)) : 0;
    constexpr uint32_t per = H * H * H / kN;
    constexpr uint32_t Z = per >= H ? H : (per >= 1 ? per : 1);
    constexpr uint32_t lzr = 31 - __builtin_clz(Z);
    constexpr uint32_t nruns = H * H * H / Z;
#pragma unroll 1
    for (uint32_t rr = tid; rr < nruns; rr += kN) {
        const uint32_t ci = rr & (H - 1), cj = (rr >> lh) & (H - 1), ck0 = (rr >> (2 * lh)) << lzr;
        const bool lx = far_x && ci == H - 1, ly = far_y && cj == H - 1;
        float v[27];
        auto cur = at(2 * ci, 2 * cj, 2 * ck0);
        {
            const uint32_t c = ci + H * (cj + H * ck0);
            const bool has = (flags[c >> 5] >> (c & 31)) & 1u;
            finest_cube<T, true>(s, has, ci, cj, ck0, v, cur, lx, ly, far_z && ck0 == H - 1);
        }
#pragma unroll 1
        for (uint32_t z = 1; z < Z; ++z) {
            const uint32_t ck = ck0 + z;
            const uint32_t c = ci + H * (cj + H * ck);
            const bool has = (flags[c >> 5] >> (c & 31)) & 1u;
#pragma unroll
            for (int p = 0; p < 9; ++p) v[p] = v[p + 18];
            cur.up();
            finest_cube<T, false>(s, has, ci, cj, ck, v, cur, lx, ly, far_z && ck == H - 1);
        }
    }
}

// Entries of the next work item, loaded into registers in three stages, each
// issued one phase of the current tile ahead of its use, so that the chain of
// dependent global loads -- item and block, then entry positions and node
// indices, then node values -- completes behind the current tile's work
// instead of stalling the tile's threads at every tile.
constexpr uint32_t kPrefetch = 2; // entries per thread held in registers
struct Prefetch {
    uint32_t item;
    uint32_t flag; // word tid of the item's cube flags
    uint32_t cidx; // threads 0-7: the coarse-grid index of tile corner tid (0xffffffff: none)
    float corner;
    uint32_t node_base, e0, e1; // a plan holds fewer than 2^32 nodes and entries
    uint32_t loc[kPrefetch];
    uint32_t node[kPrefetch];
    float val[kPrefetch];
};

// stage 1: the item's block, entry range, flag word and corner positions in the coarse grid
template <uint32_t kN>
__device__ __forceinline__ void prefetch_head(Prefetch& pf, const TileArgs& a, uint32_t item, uint32_t tid)
{
    pf.item = item;
    pf.e0 = pf.e1 = 0;
    pf.cidx = 0xffffffffu;
    if (item >= a.nitems) return;
    const uint2 it = a.items[item];
    const PlanBlock* B = &a.blocks[it.x];
    pf.node_base = (uint32_t)B->node_base;
    pf.e0 = (uint32_t)a.entry_off[item];
    pf.e1 = (uint32_t)a.entry_off[item + 1];
    if (tid < a.flag_words) pf.flag = a.flags[(uint64_t)item * a.flag_words + tid];
    if (tid < 8) {
        const uint32_t L = B->coarse_log2;
        if (L > 0) {
            const uint32_t tile = it.y & 0x7fffffffu, mL = 1u << L, E = mL + 1;
            const uint32_t cx = (tile & (mL - 1)) + (tid & 1);
            const uint32_t cy = ((tile >> L) & (mL - 1)) + ((tid >> 1) & 1);
            const uint32_t cz = (tile >> (2 * L)) + (tid >> 2);
            pf.cidx = B->coarse_off + cx + E * (cy + E * cz);
        }
    }
}

// stage 2: positions and node indices of the first kPrefetch * kN entries, and the corners
template <uint32_t kN> __device__ __forceinline__ void prefetch_index(Prefetch& pf, const TileArgs& a, uint32_t tid)
{
    if (pf.cidx != 0xffffffffu) pf.corner = a.coarse[pf.cidx];
#pragma unroll
    for (uint32_t q = 0; q < kPrefetch; ++q) {
        const uint32_t i = pf.e0 + tid + q * kN;
        if (i < pf.e1) {
            pf.loc[q] = a.entry_local[i];
            pf.node[q] = a.entry_node[i];
        }
    }
}

// stage 3: their node values
template <uint32_t kN> __device__ __forceinline__ void prefetch_values(Prefetch& pf, const TileArgs& a, uint32_t tid)
{
#pragma unroll
    for (uint32_t q = 0; q < kPrefetch; ++q)
        if (pf.e0 + tid + q * kN < pf.e1) pf.val[q] = a.sparse[pf.node_base + pf.node[q]];
}

struct TileItem {
    uint32_t d, k, L, tx, ty, tz, blk, pitch;
    uint32_t slots; // the tile has flagged cubes, which read its midpoint slots
    uint64_t node_base, dense_off;
    uint32_t item;
};

// One tile of T = 2^k cells of a plan.  Tiles of T >= 2 use the split layout; T = 1
// (depth-0 blocks) is a plain 2x2x2 copy of the root corners.
// cw: the CTA or the warp running the tile; next_item(): the next work item's number (read once the current
// item's entries are placed, so that its first prefetch stage goes out behind this tile's work).
template <uint32_t T, typename OutT, uint32_t kN, class NextFn>
__device__ __forceinline__ void run_tile(const TileArgs& a, float* s, uint32_t* flags, const TileItem& t, Prefetch& pf,
                                         Crew<kN> cw, NextFn next_item)
{
    constexpr uint32_t E = T + 1, E3 = E * E * E;
    using S = SplitTile<T < 2 ? 2 : T>;
    auto at = [](uint32_t x, uint32_t y, uint32_t z) -> uint32_t {
        if constexpr (T < 2) return x + 2 * (y + 2 * z);
        else return S::at(x, y, z);
    };
    const uint32_t d = t.d, L = t.L;
    const uint32_t ox = t.tx * T, oy = t.ty * T, oz = t.tz * T;
    const uint32_t e = (1u << d) + 1u;
    constexpr uint32_t nflags = T >= 2 ? (S::H * S::H * S::H + 31) / 32 : 0;
    if (cw.tid < nflags) flags[cw.tid] = pf.flag; // the plan's flags, prefetched
    // 1. the tile's sparse values, NaN elsewhere
    {
        const float4 nan4 = make_float4(qnan(), qnan(), qnan(), qnan());
        float4* s4 = reinterpret_cast<float4*>(s);
        // the even sub-array always (the coarse levels test it for NaN); the midpoint slots only
        // where a flagged cube will read them
        uint32_t n4 = (E3 + 3) / 4;
        if constexpr (T >= 2) {
            constexpr uint32_t G3 = S::G * S::G * S::G;
            if (!t.slots) n4 = (G3 + 3) / 4;
        }
#pragma unroll 1
        for (uint32_t p = cw.tid; p < n4; p += kN) s4[p] = nan4;
    }
    cw.sync();
    auto place = [&](uint32_t loc, float v) {
        if (loc < E3) s[loc] = v;
    };
    // the prefetched entries, then any beyond what the registers held
#pragma unroll
    for (uint32_t q = 0; q < kPrefetch; ++q)
        if (pf.e0 + cw.tid + q * kN < pf.e1) place(pf.loc[q], to_internal(pf.val[q]));
    for (uint32_t i = pf.e0 + cw.tid + kPrefetch * kN; i < pf.e1; i += kN)
        place(a.entry_local[i], to_internal(a.sparse[t.node_base + a.entry_node[i]]));
    // a tile of a block with coarse levels: its corners from the block's coarse grid
    if (pf.cidx != 0xffffffffu) s[at((cw.tid & 1) * T, ((cw.tid >> 1) & 1) * T, (cw.tid >> 2) * T)] = pf.corner;
    prefetch_head<kN>(pf, a, next_item(), cw.tid); // the current item's entries are placed
    cw.sync();
    // 2. the tile cube's own midpoints (its first level): the first warp, its 27 points in registers
    if constexpr (T >= 4) {
        if (kN == 32 || cw.tid < 32) tile_top<T>(s, cw.tid & 31);
        cw.sync();
    }
    prefetch_index<kN>(pf, a, cw.tid);
    // 3. the remaining coarser levels on the even sub-array (a tile of T/2 cells)
    if constexpr (T >= 8) tile_levels<S::G, S::H, 1, 31 - __builtin_clz(T), kN>(s, cw);
    // 4. the finest level, straight to HBM, while the next item's entries load
    prefetch_values<kN>(pf, a, cw.tid);
    float inv_scale = 1.f, offset = 0.f;
    if (a.scale_offset) {
        const float2 so = a.scale_offset[t.blk];
        inv_scale = 1.f / so.x;
        offset = so.y;
    }
    const uint32_t mL = 1u << L;
    OutT* out = reinterpret_cast<OutT*>(a.out) + t.dense_off;
    const bool far_x = t.tx == mL - 1, far_y = t.ty == mL - 1, far_z = t.tz == mL - 1;
    if constexpr (T >= 2) {
        const uint32_t pitch = t.pitch;
        const uint32_t e2 = e * pitch; // slab stride (a brick holds fewer than 2^32 elements)
        finest_store<T, kN>(s, flags, far_x, far_y, far_z, cw.tid, [&](uint32_t x, uint32_t y, uint32_t z) {
            return BrickCursor<OutT, (T >= 8)>{out + (((oz + z) * e + (oy + y)) * pitch + (ox + x)), e, pitch, e2,
                                               inv_scale, offset};
        });
    } else {
        // depth-0 block: its 8 root corners
        for (uint32_t q = cw.tid; q < 8; q += kN) {
            const uint32_t x = q & 1, y = (q >> 1) & 1, z = q >> 2;
            Store<OutT>::put(out, ((uint64_t)(oz + z) * e + (oy + y)) * t.pitch + ox + x, s[at(x, y, z)],
                             inv_scale, offset);
        }
    }
}

// ---------------------------------------------------------------- blocks from their node lists
//
// A subtree's dense grid from its nodes as the caller holds them (vertex indices and values in any order), tile by
// tile as above.  A block of one tile, or of 8 and up to kGridDirectNodes nodes, has every tile read the whole node list; else
// the nodes were scattered beforehand, each value to its vertex's place in a grid and one bit into a mask of the
// block's vertices (rows of whole words), so that a tile reads 17^2 mask rows and the values of the nodes it holds
// instead of 17^3 grid values, and the grid itself is never cleared.

// The tile's node values from the mask and grid, by kN threads: thread `tid` takes the rows tid, tid + kN, ... and
// keeps up to 8 loads in flight; row_mask gets every row's bits.
template <uint32_t T, uint32_t kN, class Put>
__device__ __forceinline__ void gather_nodes(const uint32_t* bits, const float* vals, uint32_t e, uint32_t ox,
                                             uint32_t oy, uint32_t oz, uint32_t tid, uint32_t* row_mask, Put&& put)
{
    constexpr uint32_t E = T + 1, kRows = E * E, kPer = (kRows + kN - 1) / kN;
    const uint32_t words = (e + 31) / 32, w = ox >> 5, sh = ox & 31;
    uint32_t mask[kPer];
#pragma unroll
    for (uint32_t r = 0; r < kPer; ++r) {
        const uint32_t row = tid + r * kN;
        mask[r] = 0;
        if (row < kRows) {
            const uint32_t* b = bits + ((uint64_t)(oz + row / E) * e + (oy + row % E)) * words + w;
            const uint32_t lo = b[0], hi = sh + E > 32 ? b[1] : 0u;
            mask[r] = __funnelshift_r(lo, hi, sh) & ((1u << E) - 1u);
        }
    }
#pragma unroll
    for (uint32_t r = 0; r < kPer; ++r)
        if (tid + r * kN < kRows) row_mask[tid + r * kN] = mask[r];
#pragma unroll 1
    for (uint32_t r = 0; r < kPer; ++r) {
        // (a register array indexed by a loop variable would live in local memory)
        uint32_t m = 0;
#pragma unroll
        for (uint32_t q = 0; q < kPer; ++q)
            if (q == r) m = mask[q];
        const uint32_t row = tid + r * kN, y = row % E, z = row / E;
        const float* src = vals + ((uint64_t)(oz + z) * e + (oy + y)) * e + ox;
        while (m) {
            uint32_t x[8];
            float v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                x[q] = 32;
                if (m) {
                    x[q] = (uint32_t)__ffs((int)m) - 1;
                    m &= m - 1;
                    v[q] = src[x[q]];
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (x[q] < 32) put(x[q], y, z, to_internal(v[q]));
        }
    }
}

// The flags of the finest-level cubes that hold a node at one of their midpoints, from the rows' bits: along a row of
// cubes, the rows with y or z odd count at all three positions of a cube, the four even ones at its middle.  By the
// kInterpThreads - 32 threads after the first warp, tid counted from them.
template <uint32_t T> __device__ __forceinline__ void flags_from_rows(const uint32_t* row_mask, uint32_t* flags,
                                                                      uint32_t tid)
{
    constexpr uint32_t H = T / 2, E = T + 1;
    for (uint32_t q = tid; q < H * H; q += kInterpThreads - 32) {
        const uint32_t y = 2 * (q % H), z = 2 * (q / H);
        const uint32_t* r = row_mask + y + E * z;
        const uint32_t all = r[1] | r[E] | r[E + 1] | r[E + 2] | r[2 * E + 1];
        const uint32_t mid = r[0] | r[2] | r[2 * E] | r[2 * E + 2];
        const uint32_t odd = (all | (all << 1) | (all >> 1) | mid) & 0xaaaaaaaau; // bit 2i + 1: cube i
        uint32_t f = 0;
#pragma unroll
        for (uint32_t i = 0; i < H; ++i) f |= ((odd >> (2 * i + 1)) & 1u) << i;
        if (f) atomicOr(&flags[(H * q) >> 5], f << ((H * q) & 31));
    }
}

// One tile (tx, ty, tz) of T = 2^k cells of block b, by a CTA.  cursor(x, y, z): the output cursor of the cube whose
// low corner is the block's vertex (x, y, z); put0(x, y, z, v): a vertex of a depth-0 block.
template <uint32_t T, class At, class Put0>
__device__ __forceinline__ void run_grid_tile(const GridBlock& b, const float* vals, const uint32_t* bits, float* s,
                                              float* desc, uint32_t* row_mask, uint32_t* flags, uint32_t tx,
                                              uint32_t ty, uint32_t tz, At&& cursor, Put0&& put0)
{
    constexpr uint32_t E = T + 1, E3 = E * E * E, kN = kInterpThreads;
    constexpr uint32_t lt = 31 - __builtin_clz(T);
    using S = SplitTile<T < 2 ? 2 : T>;
    const uint32_t tid = threadIdx.x, d = b.depth, L = d - lt;
    const uint32_t ox = tx * T, oy = ty * T, oz = tz * T, e = (1u << d) + 1u;
    constexpr uint32_t nflags = T >= 2 ? (S::H * S::H * S::H + 31) / 32 : 0;
    auto slot = [](uint32_t x, uint32_t y, uint32_t z) -> uint32_t {
        if constexpr (T < 2) return x + 2 * (y + 2 * z);
        else return S::at(x, y, z);
    };
    for (uint32_t q = tid; q < nflags; q += kN) flags[q] = 0u;
    const float4 nan4 = make_float4(qnan(), qnan(), qnan(), qnan());
    for (uint32_t p = tid; p < (E3 + 3) / 4; p += kN) reinterpret_cast<float4*>(s)[p] = nan4;
    if (b.direct) {
        for (uint32_t q = tid; q < E * E; q += kN) row_mask[q] = 0u;
        if (tid < 27) desc[tid] = qnan();
    }
    __syncthreads();
    float corner = 0.f; // lanes 0-7 of warp 0: the tile's corners from the coarse levels
    if (b.direct) {
        for (uint32_t i0 = tid; i0 < b.n; i0 += 4 * kN) {
            uint32_t x[4], y[4], z[4];
            float v[4];
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t i = i0 + q * kN;
                x[q] = 0xffffffffu;
                if (i < b.n) {
                    x[q] = b.n2i[3 * (size_t)i];
                    y[q] = b.n2i[3 * (size_t)i + 1];
                    z[q] = b.n2i[3 * (size_t)i + 2];
                    v[q] = b.sparse[i];
                }
            }
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                if (x[q] >= e || y[q] >= e || z[q] >= e) continue; // no node, or one outside the block: ignored
                const float w = to_internal(v[q]);
                // L <= 1: the lattice of tile corners is the root cube's 27 points
                if (L > 0 && ((x[q] | y[q] | z[q]) & (T - 1)) == 0)
                    desc[(x[q] >> lt) + 3 * (y[q] >> lt) + 9 * (z[q] >> lt)] = w;
                const uint32_t lx = x[q] - ox, ly = y[q] - oy, lz = z[q] - oz;
                if (lx < E && ly < E && lz < E) {
                    s[slot(lx, ly, lz)] = w;
                    atomicOr(&row_mask[ly + E * lz], 1u << lx);
                }
            }
        }
    } else {
        // the tile's corners by the first warp, its nodes by the others meanwhile
        const float* bv = vals + b.val_off;
        const uint32_t* bb = bits + b.bit_off;
        if (tid < 32) {
            const uint32_t words = (e + 31) / 32;
            corner = descend_regs(d, L, ox, oy, oz, tid, [&](uint32_t gx, uint32_t gy, uint32_t gz) {
                const uint64_t row = (uint64_t)gz * e + gy;
                // both at once: the value means something only where the bit is set
                const float v = bv[row * e + gx];
                const uint32_t m = bb[row * words + (gx >> 5)];
                return (m >> (gx & 31)) & 1u ? to_internal(v) : qnan();
            });
        } else {
            gather_nodes<T, kN - 32>(bb, bv, e, ox, oy, oz, tid - 32, row_mask,
                                     [&](uint32_t x, uint32_t y, uint32_t z, float v) { s[slot(x, y, z)] = v; });
        }
    }
    __syncthreads();
    if (tid < 32) {
        // the corners, then the tile cube's own midpoints in registers; the flags by the other warps
        if (L > 0) {
            if (b.direct)
                corner = descend_regs(d, L, ox, oy, oz, tid, [&](uint32_t gx, uint32_t gy, uint32_t gz) {
                    return desc[(gx >> lt) + 3 * (gy >> lt) + 9 * (gz >> lt)];
                });
            if (tid < 8) s[slot((tid & 1) * T, ((tid >> 1) & 1) * T, (tid >> 2) * T)] = corner;
            __syncwarp();
        }
        if constexpr (T >= 4) tile_top<T>(s, tid);
    } else {
        if constexpr (T >= 2) flags_from_rows<T>(row_mask, flags, tid - 32);
    }
    __syncthreads();
    if constexpr (T >= 8) tile_levels<S::G, S::H, 1, lt, kN>(s, Crew<kN>{tid});
    const uint32_t mL = 1u << L;
    if constexpr (T >= 2) {
        finest_store<T, kN>(s, flags, tx == mL - 1, ty == mL - 1, tz == mL - 1, tid,
                            [&](uint32_t x, uint32_t y, uint32_t z) { return cursor(ox + x, oy + y, oz + z); });
    } else {
        for (uint32_t q = tid; q < 8; q += kN) {
            const uint32_t x = q & 1, y = (q >> 1) & 1, z = q >> 2;
            const float v = s[slot(x, y, z)];
            put0(x, y, z, isinf(v) ? qnan() : v);
        }
    }
}

} // namespace
} // namespace s3r
