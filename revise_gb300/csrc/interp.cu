// Sparse-octree -> dense-grid interpolation for sm_103a.
//
// Restates the hierarchical midpoint fill of the reference
// (include/s3dmm/DenseFieldInterpolator.hpp:198-419; GPU form
// src/s3dmm_cuda/DenseFieldInterpolatorArr_cu_3.cu:69-188 and :197-257):
// level by level, every cube's edge midpoints take 1/2 of their two ends,
// face midpoints 1/4 of their four edge midpoints, the cell centre 1/6 of its
// six face centres, unless a sparse node already defines the vertex; any
// stencil value equal to the no-field value makes the result the no-field
// value, which becomes NaN on output.
//
// GB300 form: a cube at level L is self-contained -- every vertex inside it
// (faces and edges included) depends only on the cube's 8 corners and on the
// sparse nodes inside it -- so the grid is cut into tiles of 2^k cells, each
// computed by one CTA (one warp, for plans of tiles up to 8 cells) in shared
// memory in a single launch:
//   1. the tile's sparse nodes are placed into a NaN-filled shared tile;
//   2. one warp walks the L = d - k coarse levels down from the block's root
//      corners to the tile's 8 corners (27 points per level);
//   3. the k fine levels run over the shared tile (edges, faces, cells);
//   4. the tile's owned vertices go to HBM once, coalesced along x, with
//      no-field -> NaN and optional FP16/BF16 encoding fused into the store.
// The reference instead makes d full-grid passes through global memory.
// Sums run in the reference CPU interpolator's order, so results are
// bit-identical to it.
#include "interp_tile.cuh"
#include "s3r_internal.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

namespace s3r {
namespace {

// p: 16-byte aligned up to the last n % 4 words, or (vec false) anywhere
__global__ void fill_u32_kernel(uint32_t* p, uint64_t n, uint32_t v, bool vec)
{
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n4 = vec ? n / 4 : 0;
    for (uint64_t i = t; i < n4; i += step) reinterpret_cast<uint4*>(p)[i] = make_uint4(v, v, v, v);
    for (uint64_t i = 4 * n4 + t; i < n; i += step) p[i] = v;
}

// vals[ord(n2i[i])] = sparse[i] and the vertex's bit, for the scattered blocks of a set (block blockIdx.y)
// (scatterSparseFieldKernel, DenseFieldInterpolatorArr_cu_3.cu:38-51)
__global__ void scatter_kernel(GridArgs a)
{
    const GridBlock b = a.table ? a.table[blockIdx.y] : a.one;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (b.direct || i >= b.n) return;
    const uint32_t e = (1u << b.depth) + 1u, words = (e + 31) / 32;
    const uint32_t x = b.n2i[3 * (size_t)i], y = b.n2i[3 * (size_t)i + 1], z = b.n2i[3 * (size_t)i + 2];
    if (x >= e || y >= e || z >= e) return; // out-of-range node: ignored (the reference asserts)
    const uint64_t row = (uint64_t)z * e + y;
    a.vals[b.val_off + row * e + x] = b.sparse[i];
    atomicOr(&a.bits[b.bit_off + row * words + (x >> 5)], 1u << (x & 31));
}

// The blocks of a set from their node lists, one CTA per tile (a set of one block: its tile is the CTA index; else
// the block is found in the running tile counts).  kSurface: into 3-D arrays, else into plain grids.
// Bound by the latency of a tile's phases, 8 CTAs per SM in flight; reading the mask instead of a NaN-filled grid
// took the fill pass away and shortened the tile's first phase from 39 dependent grid loads a thread to a few.
template <bool kSurface> __global__ void __launch_bounds__(kInterpThreads, 8) interp_grid_kernel(GridArgs a)
{
    extern __shared__ float4 s_tile[]; // tile_smem_bytes(): (2^k+1)^3 floats rounded up to whole float4s
    float* s = reinterpret_cast<float*>(s_tile);
    __shared__ float desc[27];                   // direct: the lattice of tile corners of a block of 8 tiles
    __shared__ uint32_t row_mask[17 * 17];       // per row of the tile the vertices that hold a node
    __shared__ uint32_t flags[(8 * 8 * 8) / 32]; // one bit per finest cube
    uint32_t tile = blockIdx.x;
    GridBlock b = a.one;
    if (a.table) {
        uint32_t lo = 0, hi = a.nblocks;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (a.tile_off[mid] <= tile) lo = mid;
            else hi = mid;
        }
        b = a.table[lo];
        tile -= a.tile_off[lo];
    }
    const uint32_t k = b.depth < kGridTileLog2 ? b.depth : kGridTileLog2, L = b.depth - k, mL = 1u << L;
    const uint32_t tx = tile & (mL - 1), ty = (tile >> L) & (mL - 1), tz = tile >> (2 * L);
    const uint32_t e = (1u << b.depth) + 1u;
    auto run = [&](auto size) {
        constexpr uint32_t T = decltype(size)::value;
        if constexpr (kSurface) {
            run_grid_tile<T>(b, a.vals, a.bits, s, desc, row_mask, flags, tx, ty, tz,
                             [&](uint32_t x, uint32_t y, uint32_t z) {
                                 return SurfaceCursor{b.surface, (int)x, (int)y, (int)z};
                             },
                             [&](uint32_t x, uint32_t y, uint32_t z, float v) {
                                 surf3Dwrite(v, (cudaSurfaceObject_t)b.surface, (int)x * 4, (int)y, (int)z);
                             });
        } else {
            // (2^9+1)^3 elements: offsets fit 32 bits.  A cube's low corner has even coordinates, so its first row
            // starts at an even element of the grid: the parities are the grid's own.
            const uint32_t odd = (uint32_t)(reinterpret_cast<uintptr_t>(b.out) >> 2) & 1u;
            run_grid_tile<T>(b, a.vals, a.bits, s, desc, row_mask, flags, tx, ty, tz,
                             [&](uint32_t x, uint32_t y, uint32_t z) {
                                 return GridCursor{b.out + ((z * e + y) * e + x), e, e * e, odd, x == 0};
                             },
                             [&](uint32_t x, uint32_t y, uint32_t z, float v) { b.out[(z * e + y) * e + x] = v; });
        }
    };
    switch (k) {
    case 0: run(std::integral_constant<uint32_t, 1>()); break;
    case 1: run(std::integral_constant<uint32_t, 2>()); break;
    case 2: run(std::integral_constant<uint32_t, 4>()); break;
    case 3: run(std::integral_constant<uint32_t, 8>()); break;
    default: run(std::integral_constant<uint32_t, 16>()); break;
    }
}

// Work item `item` of the batched plan as the tile it names.
__device__ __forceinline__ TileItem decode_item(const TileArgs& a, uint32_t item)
{
    TileItem t;
    t.item = item;
    const uint2 it = a.items[item];
    t.blk = it.x;
    const uint32_t tile = it.y & 0x7fffffffu;
    t.slots = it.y >> 31;
    const PlanBlock b = a.blocks[t.blk];
    t.d = b.depth;
    t.k = b.tile_log2;
    t.L = b.coarse_log2;
    t.node_base = b.node_base;
    t.dense_off = b.dense_off;
    t.pitch = b.pitch;
    const uint32_t mL = 1u << t.L;
    t.tx = tile & (mL - 1);
    t.ty = (tile >> t.L) & (mL - 1);
    t.tz = tile >> (2 * t.L);
    return t;
}

template <typename OutT>
__global__ void __launch_bounds__(kInterpThreads, 8) interp_tiles_kernel(TileArgs a)
{
    extern __shared__ float4 s_tile[]; // tile_smem_bytes(): (2^k+1)^3 floats rounded up to whole float4s
    float* s = reinterpret_cast<float*>(s_tile);
    __shared__ uint32_t flags[(16 * 16 * 16) / 32]; // one bit per finest cube, tiles up to 32 cells
    __shared__ uint32_t item_s, next_s[2];
    const uint32_t nitems = a.nitems;
    const Crew<kInterpThreads> cw{threadIdx.x};
    // Work items come from the queue counter (zeroed before the launch).  The
    // next item is taken at the start of the current one so its entries can be
    // prefetched.  The slot it goes to alternates: a warp still reading slot
    // i & 1 after the loop's closing barrier must not see thread 0 refill it for
    // item i + 2 (the barriers inside the tile keep thread 0 from getting that far).
    if (threadIdx.x == 0) item_s = atomicAdd(a.queue, 1u);
    __syncthreads();
    uint32_t item = item_s;
    Prefetch pf;
    prefetch_head<kInterpThreads>(pf, a, item, threadIdx.x);
    prefetch_index<kInterpThreads>(pf, a, threadIdx.x);
    prefetch_values<kInterpThreads>(pf, a, threadIdx.x);
    for (uint32_t iter = 0;; ++iter) {
        if (item >= nitems) break;
        uint32_t* next_p = &next_s[iter & 1];
        if (threadIdx.x == 0) *next_p = atomicAdd(a.queue, 1u);
        const TileItem t = decode_item(a, item);
        auto next = [next_p] { return *next_p; };
        switch (t.k) {
        case 0: run_tile<1, OutT>(a, s, flags, t, pf, cw, next); break;
        case 1: run_tile<2, OutT>(a, s, flags, t, pf, cw, next); break;
        case 2: run_tile<4, OutT>(a, s, flags, t, pf, cw, next); break;
        case 3: run_tile<8, OutT>(a, s, flags, t, pf, cw, next); break;
        case 4: run_tile<16, OutT>(a, s, flags, t, pf, cw, next); break;
        default: run_tile<32, OutT>(a, s, flags, t, pf, cw, next); break;
        }
        __syncthreads();
        item = *next_p;
    }
}

// Plans whose tiles are all of 8 cells or fewer: one warp per tile.  Each warp holds its own split tile
// (9^3 floats) and flag words in shared memory, takes its own items from the queue and synchronizes only
// with itself, so an SM keeps 32 tiles in flight instead of 8 CTAs' worth: a tile is a chain of short
// dependent phases (fill, placement, tile cube, coarse level, finest level), and more chains per SM hide
// more of their latency.  Same tile code, same results as the CTA kernel.
constexpr uint32_t kWarpTileFloats = ((9 * 9 * 9 + 3) / 4) * 4; // tile_smem_bytes(3) / 4
template <typename OutT> __global__ void __launch_bounds__(kInterpThreads, 8) interp_warp_tiles_kernel(TileArgs a)
{
    constexpr uint32_t kWarps = kInterpThreads / 32;
    __shared__ float4 s_all[kWarps][kWarpTileFloats / 4];
    __shared__ uint32_t flags_all[kWarps][2]; // 8-cell tiles: 64 finest cubes
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* s = reinterpret_cast<float*>(s_all[w]);
    uint32_t* flags = flags_all[w];
    const Crew<32> cw{lane};
    const uint32_t nitems = a.nitems;
    uint32_t item = lane == 0 ? atomicAdd(a.queue, 1u) : 0u;
    item = __shfl_sync(0xffffffffu, item, 0);
    Prefetch pf;
    prefetch_head<32>(pf, a, item, lane);
    prefetch_index<32>(pf, a, lane);
    prefetch_values<32>(pf, a, lane);
    while (item < nitems) {
        const uint32_t nxt = lane == 0 ? atomicAdd(a.queue, 1u) : 0u; // read by the warp once placed
        const TileItem t = decode_item(a, item);
        auto next = [nxt] { return __shfl_sync(0xffffffffu, nxt, 0); };
        switch (t.k) {
        case 0: run_tile<1, OutT>(a, s, flags, t, pf, cw, next); break;
        case 1: run_tile<2, OutT>(a, s, flags, t, pf, cw, next); break;
        case 2: run_tile<4, OutT>(a, s, flags, t, pf, cw, next); break;
        default: run_tile<8, OutT>(a, s, flags, t, pf, cw, next); break;
        }
        __syncwarp();
        item = __shfl_sync(0xffffffffu, nxt, 0);
    }
}

// Per-block preparation of a plan frame, one CTA per block:
//  * 16-bit bricks: the {scale, offset} of the block's valid sparse values; all dense values are means of
//    sparse values, so they stay inside this range;
//  * a block cut into 2^L > 1 tiles per axis: its coarse grid, the (2^L+1)^3 vertices at multiples of
//    the tile edge, from the sparse nodes on it, filled level by level exactly as a tile is filled (the
//    reference's midpoint rules, sums in its order).  A midpoint of a coarse level depends only on the
//    points of that level's cube, so the full grid holds the values a descent from the block's root
//    along any one tile's path computes -- each tile then reads its 8 corners from it instead of
//    descending itself, and the plan carries the coarse nodes once per block instead of once per tile.
// What bounds it is latency: the rounds of a thread's loads of the values and the levels of the coarse grid.  So 8
// loads are in flight, grids of up to 9^3 are filled in shared memory, and few blocks of many nodes get wider CTAs
// (launch_block_prep).
constexpr uint32_t kPrepGrid = 9 * 9 * 9;
__global__ void __launch_bounds__(1024) block_prep_kernel(PrepArgs a)
{
    __shared__ float s_grid[kPrepGrid];
    __shared__ float slo[32], shi[32];
    const uint32_t b = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
    const PlanBlock B = a.blocks[b];
    const uint32_t L = B.coarse_log2, T = 1u << L, E = T + 1, E3 = E * E * E;
    if (a.scale_offset) {
        const uint64_t n0 = a.node_off[b], n1 = a.node_off[b + 1];
        float lo = INFINITY, hi = -INFINITY;
        for (uint64_t i = n0 + tid; i < n1; i += 8 * nt) {
            float v[8];
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) v[q] = i + q * nt < n1 ? a.sparse[i + q * nt] : kNoField;
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q)
                if (v[q] != kNoField) { // a NaN changes neither
                    lo = fminf(lo, v[q]);
                    hi = fmaxf(hi, v[q]);
                }
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if ((tid & 31) == 0) {
            slo[tid >> 5] = lo;
            shi[tid >> 5] = hi;
        }
        __syncthreads();
        if (tid == 0) {
            for (uint32_t i = 1; i < nt / 32; ++i) {
                lo = fminf(lo, slo[i]);
                hi = fmaxf(hi, shi[i]);
            }
            float scale = hi - lo;
            if (!(scale > 0.f) || !isfinite(scale)) scale = 1.f;
            if (!isfinite(lo)) lo = 0.f;
            a.scale_offset[b] = make_float2(scale, lo);
        }
    }
    if (L == 0) return;
    auto fill = [&](float* g) {
        for (uint32_t p = tid; p < E3; p += nt) g[p] = qnan();
        __syncthreads();
        for (uint32_t i = a.centry_off[b] + tid; i < a.centry_off[b + 1]; i += nt) {
            const uint2 ce = a.centry[i];
            if (ce.x < E3) g[ce.x] = to_internal(a.sparse[B.node_base + ce.y]);
        }
        __syncthreads();
        for (uint32_t j = 0; j < L; ++j) {
            cube_level(g, E, T, j);
            __syncthreads();
        }
    };
    float* out = a.coarse + B.coarse_off;
    if (E3 <= kPrepGrid) {
        fill(s_grid);
        for (uint32_t p = tid; p < E3; p += nt) out[p] = s_grid[p];
    } else {
        fill(out);
    }
}

inline uint32_t ctas_for(uint64_t n, uint32_t threads)
{
    uint64_t c = (n + threads - 1) / threads;
    if (c > 152ull * 64) c = 152ull * 64;
    return c ? (uint32_t)c : 1u;
}

template <typename OutT>
cudaError_t launch_tiles(const TileArgs& a, uint32_t tile_log2_max, uint32_t grid_ctas, cudaStream_t s)
{
    if (tile_log2_max <= 3) {
        interp_warp_tiles_kernel<OutT><<<grid_ctas, kInterpThreads, 0, s>>>(a);
        return cudaGetLastError();
    }
    const size_t smem = tile_smem_bytes(tile_log2_max);
    auto kern = interp_tiles_kernel<OutT>;
    if (smem > 48 * 1024) {
        cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return err;
    }
    kern<<<grid_ctas, kInterpThreads, smem, s>>>(a);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_fill_u32(uint32_t* p, uint64_t n, uint32_t v, cudaStream_t s)
{
    const bool vec = reinterpret_cast<uintptr_t>(p) % 16 == 0;
    fill_u32_kernel<<<ctas_for(vec ? (n + 3) / 4 : n, 256), 256, 0, s>>>(p, n, v, vec);
    return cudaGetLastError();
}

GridBlock grid_block(const uint16_t* n2i, const float* sparse, uint32_t n, uint32_t depth)
{
    GridBlock b{};
    b.n2i = n2i;
    b.sparse = sparse;
    b.n = n;
    b.depth = depth;
    b.direct = depth <= kGridTileLog2 || (depth == kGridTileLog2 + 1 && n <= kGridDirectNodes);
    return b;
}

cudaError_t launch_interp_grid(const GridArgs& a, bool surface, uint32_t scattered_nodes, uint64_t bit_words,
                               cudaStream_t s, uint32_t* launches)
{
    uint32_t count = 1, depth_max = a.depth_max;
    cudaError_t err;
    if (bit_words) {
        if ((err = cudaMemsetAsync(a.bits, 0, bit_words * sizeof(uint32_t), s)) != cudaSuccess) return err;
        if (scattered_nodes) {
            scatter_kernel<<<dim3((scattered_nodes + 255) / 256, a.nblocks), 256, 0, s>>>(a);
            if ((err = cudaGetLastError()) != cudaSuccess) return err;
            ++count;
        }
    }
    const size_t smem = tile_smem_bytes(depth_max < kGridTileLog2 ? depth_max : kGridTileLog2);
    if (surface) interp_grid_kernel<true><<<a.tiles, kInterpThreads, smem, s>>>(a);
    else interp_grid_kernel<false><<<a.tiles, kInterpThreads, smem, s>>>(a);
    if (launches) *launches += count;
    return cudaGetLastError();
}

uint32_t interp_plan_ctas_per_sm(uint32_t fmt, uint32_t tile_log2)
{
    const bool warp = tile_log2 <= 3; // the warp-per-tile kernel (static shared memory only)
    const size_t smem = warp ? 0 : tile_smem_bytes(tile_log2);
    int n = 0;
    cudaError_t e = cudaErrorInvalidValue;
    auto occ = [&](auto kern) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, kInterpThreads, smem);
    };
    switch (fmt) {
    case S3R_BRICK_F32: warp ? occ(interp_warp_tiles_kernel<float>) : occ(interp_tiles_kernel<float>); break;
    case S3R_BRICK_F16: warp ? occ(interp_warp_tiles_kernel<__half>) : occ(interp_tiles_kernel<__half>); break;
    case S3R_BRICK_BF16:
        warp ? occ(interp_warp_tiles_kernel<__nv_bfloat16>) : occ(interp_tiles_kernel<__nv_bfloat16>);
        break;
    default: break;
    }
    return (e == cudaSuccess && n > 0) ? (uint32_t)n : 1u;
}

cudaError_t launch_interp_plan(const TileArgs& a, uint32_t fmt, uint32_t tile_log2_max, uint32_t grid_ctas,
                               cudaStream_t s)
{
    if (a.nitems == 0) return cudaSuccess;
    switch (fmt) {
    case S3R_BRICK_F32: return launch_tiles<float>(a, tile_log2_max, grid_ctas, s);
    case S3R_BRICK_F16: return launch_tiles<__half>(a, tile_log2_max, grid_ctas, s);
    case S3R_BRICK_BF16: return launch_tiles<__nv_bfloat16>(a, tile_log2_max, grid_ctas, s);
    default: return cudaErrorInvalidValue;
    }
}

// Wider CTAs while every block's is resident at once and a thread is left two rounds of loads.
cudaError_t launch_block_prep(const PrepArgs& a, uint32_t nblocks, uint32_t max_nodes, uint32_t sms, cudaStream_t s)
{
    if (nblocks == 0) return cudaSuccess;
    uint32_t threads = kInterpThreads;
    if (a.scale_offset)
        while (threads < 1024 && 2 * threads * 16 <= max_nodes && (uint64_t)nblocks * 2 * threads <= 2048ull * sms)
            threads *= 2;
    block_prep_kernel<<<nblocks, threads, 0, s>>>(a);
    return cudaGetLastError();
}

} // namespace s3r
