// Image-part kernels for sm_103a: crop rectangle of the non-transparent
// pixels (getBoundRect, src/s3vs_worker/cuda/VsWorker_cu.cpp:51-88), the crop
// itself, and compositing of ARGB32 image parts with blendImagePart's integer
// src-over-dst arithmetic (src/s3vs_lib/BlendImagePart.hpp:61-145), one thread
// per destination pixel walking the parts in order.
#include "s3r_internal.h"

namespace s3r {
namespace {

// One CTA per row at a time, four pixels a load where rows are whole 16-byte words.  Every bound is kept as a
// maximum, so that the accumulators start from zero; the last CTA hands the rectangle and the flag beside it to the
// host and zeroes them for the next call, which saves the copies in and out (2 Mpixel: 34 us with a division per
// pixel, 5 with this).
__global__ void __launch_bounds__(256) bound_rect_kernel(const uint32_t* __restrict__ img, uint32_t W, uint32_t H,
                                                         bool vec, int32_t* acc, int32_t* host)
{
    // acc: {W - min x, H - min y, max x + 1, max y + 1, flag, CTAs done}
    __shared__ int32_t cta[4];
    if (threadIdx.x < 4) cta[threadIdx.x] = 0;
    __syncthreads();
    int32_t lo = INT32_MAX, hi = -1, top = INT32_MAX, bottom = -1;
    for (uint32_t y = blockIdx.x; y < H; y += gridDim.x) {
        const uint32_t* row = img + (size_t)y * W;
        bool any = false;
        if (vec) {
            for (uint32_t q = threadIdx.x; q < W / 4; q += 256) {
                const uint4 p = __ldg(reinterpret_cast<const uint4*>(row) + q);
                const uint32_t m = (p.x >> 24 ? 1u : 0u) | (p.y >> 24 ? 2u : 0u) | (p.z >> 24 ? 4u : 0u) |
                                   (p.w >> 24 ? 8u : 0u);
                if (m) {
                    any = true;
                    lo = min(lo, (int32_t)(4 * q) + __ffs((int)m) - 1);
                    hi = max(hi, (int32_t)(4 * q) + 31 - __clz((int)m));
                }
            }
        } else {
            for (uint32_t x = threadIdx.x; x < W; x += 256)
                if (__ldg(row + x) >> 24) {
                    any = true;
                    lo = min(lo, (int32_t)x);
                    hi = max(hi, (int32_t)x);
                }
        }
        if (any) {
            top = min(top, (int32_t)y);
            bottom = (int32_t)y;
        }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    top = __reduce_min_sync(0xffffffffu, top);
    bottom = __reduce_max_sync(0xffffffffu, bottom);
    if ((threadIdx.x & 31) == 0 && hi >= 0) {
        atomicMax(&cta[0], (int32_t)W - lo);
        atomicMax(&cta[1], (int32_t)H - top);
        atomicMax(&cta[2], hi + 1);
        atomicMax(&cta[3], bottom + 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (cta[2])
            for (int i = 0; i < 4; ++i) atomicMax(&acc[i], cta[i]);
        __threadfence();
        if (atomicAdd(&acc[5], 1) == (int32_t)gridDim.x - 1) {
            __threadfence();
            for (int i = 0; i < 5; ++i) host[i] = atomicExch(&acc[i], 0);
            acc[5] = 0;
            __threadfence_system();
        }
    }
}

__global__ void __launch_bounds__(256) crop_kernel(const uint32_t* __restrict__ img, uint32_t W, int32_t x0, int32_t y0,
                                                   int32_t w, int32_t h, uint32_t* __restrict__ dst)
{
    for (int32_t y = (int32_t)blockIdx.x; y < h; y += (int32_t)gridDim.x)
        for (int32_t x = (int32_t)threadIdx.x; x < w; x += 256)
            dst[(uint64_t)y * w + x] = img[(uint64_t)(y0 + y) * W + (x0 + x)];
}

__device__ __forceinline__ uint32_t blend_px(uint32_t d, uint32_t s)
{
    const uint32_t as = s >> 24;
    if (as == 0) return d;
    if (as == 255u) return s;
    const uint32_t ad = d >> 24;
    if (ad == 0) return s;
    const uint32_t a = as + ad * (255u - as) / 255u;
    uint32_t out = (a & 0xffu) << 24;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        const uint32_t cs = (s >> (8 * b)) & 0xffu, cd = (d >> (8 * b)) & 0xffu;
        out |= (((cs * as + cd * (a - as)) / a) & 0xffu) << (8 * b);
    }
    return out;
}

// The first kComposeInline parts travel with the launch; more come from device memory.
struct ComposeParts {
    s3r_image_part p[kComposeInline];
};
__global__ void compose_kernel(const ComposeParts few, const s3r_image_part* __restrict__ many, uint32_t nparts,
                               int32_t just_copy_first, uint32_t* __restrict__ dst, int32_t dw, int32_t dh,
                               int32_t offx, int32_t offy)
{
    const int32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= dw || y >= dh) return;
    const int32_t gx = x + offx, gy = y + offy; // image-part coordinates
    uint32_t d = dst[(uint64_t)y * dw + x];
    bool touched = false;
    for (uint32_t p = 0; p < nparts; ++p) {
        const s3r_image_part& pt = many ? many[p] : few.p[p];
        const int32_t sx = gx - pt.origin[0], sy = gy - pt.origin[1];
        if (sx < 0 || sy < 0 || sx >= pt.size[0] || sy >= pt.size[1]) continue;
        const uint32_t s = pt.pixels[(uint64_t)sy * pt.size[0] + sx];
        d = (p == 0 && just_copy_first) ? s : blend_px(d, s);
        touched = true;
    }
    if (touched) dst[(uint64_t)y * dw + x] = d;
}

} // namespace

cudaError_t launch_bound_rect(const uint32_t* img, uint32_t W, uint32_t H, int32_t* acc, int32_t* host, cudaStream_t s)
{
    uint32_t ctas = H < 152 * 4 ? H : 152 * 4;
    if (ctas == 0) ctas = 1;
    const bool vec = W % 4 == 0 && reinterpret_cast<uintptr_t>(img) % 16 == 0;
    bound_rect_kernel<<<ctas, 256, 0, s>>>(img, W, H, vec, acc, host);
    return cudaGetLastError();
}

cudaError_t launch_crop(const uint32_t* img, uint32_t W, const int32_t rect[4], uint32_t* dst, cudaStream_t s)
{
    if (rect[2] <= 0 || rect[3] <= 0) return cudaSuccess;
    const uint32_t ctas = rect[3] < 152 * 8 ? (uint32_t)rect[3] : 152 * 8;
    crop_kernel<<<ctas, 256, 0, s>>>(img, W, rect[0], rect[1], rect[2], rect[3], dst);
    return cudaGetLastError();
}

cudaError_t launch_compose(const s3r_image_part* parts, const s3r_image_part* parts_dev, uint32_t nparts,
                           int32_t just_copy_first, uint32_t* dst, int32_t dw, int32_t dh, int32_t offx, int32_t offy,
                           cudaStream_t s)
{
    if (dw <= 0 || dh <= 0 || nparts == 0) return cudaSuccess;
    ComposeParts few{};
    for (uint32_t i = 0; i < nparts && !parts_dev; ++i) few.p[i] = parts[i];
    dim3 block(32, 8);
    dim3 grid((dw + 31) / 32, (dh + 7) / 8);
    compose_kernel<<<grid, block, 0, s>>>(few, parts_dev, nparts, just_copy_first, dst, dw, dh, offx, offy);
    return cudaGetLastError();
}

} // namespace s3r
