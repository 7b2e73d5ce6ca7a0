// Host side of the s3r C ABI (include/s3r.h): contexts, argument checks,
// parameter set-up restated from the reference's host code, the batched
// plan (tile binning of the octree nodes), CUDA-graph capture of a frame and
// the tile-size / CTA-shape autotuner.  Built with -ffp-contract=off so that
// float set-up code rounds as written.
#include "s3r_internal.h"

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

using namespace s3r;

namespace {

thread_local std::string g_last_error;

} // namespace

struct s3r_ctx {
    int device = 0;
    std::string err;
    cudaError_t last_cuda = cudaSuccess; // behind the last S3R_ERR_CUDA
    float* grid = nullptr; // block interpolation scratch: scattered node values, and their mask (rows of whole words)
    size_t grid_cap = 0;   // floats
    uint32_t* grid_bits = nullptr;
    size_t grid_bits_cap = 0; // words
    int32_t* rect_dev = nullptr; // launch_bound_rect's accumulators, a part's overflow flag among them
    int32_t* rect_host = nullptr; // pinned
    s3r_image_part* parts_dev = nullptr;
    size_t parts_cap = 0;
    cudaStream_t capture = nullptr;
    float* worker_dense[2] = {nullptr, nullptr}; // s3r_render_scene_part: primary / secondary dense field
    size_t worker_cap[2] = {0, 0};
    // s3r_render_scene_part with the texture filter: per depth field textures for a chunk of blocks (primary /
    // secondary; kPartTextureBytes of them at most), the
    // transfer-function texture
    std::vector<s3r_texture*> worker_tex[2][S3R_MAX_DEPTH + 1];
    uint64_t worker_tex_bytes = 0;
    s3r_tf_texture* worker_tf = nullptr;
    // a part's blocks at once: tables staged through pinned memory, and the pixels' result lists
    char* part_host = nullptr;
    char* part_dev = nullptr;
    size_t part_cap = 0, part_used = 0;
    char* part_lists = nullptr;
    size_t part_lists_cap = 0;
    uint64_t launches = 0;
    int sms = 152;
};

// One captured frame (interpolation + render) and the arguments it was captured for.
struct FrameGraph {
    cudaGraphExec_t exec = nullptr;
    const void* key[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    uint32_t dims[5] = {0, 0, 0, 0, 0}; // W, H, tf_n, filter and block-major variant of the launches
    uint32_t kernels = 0;
};

struct s3r_plan {
    s3r_ctx* ctx = nullptr;
    s3r_frame_desc desc{};
    uint32_t nblocks = 0, level = 0, fmt = 0;
    uint32_t max_nodes = 0; // of one block
    uint32_t tile_log2 = 4;             // the largest tile edge (log2 cells) over the blocks
    uint8_t tile_by_depth[S3R_MAX_DEPTH + 1] = {}; // per block depth: its tile edge (log2), capped by the depth
    uint32_t render_tile = 0;
    std::vector<uint32_t> blocks;      // 4 per block
    std::vector<uint64_t> node_off;    // nblocks+1
    std::vector<uint16_t> n2i;         // host copy (re-binning by the autotuner)
    std::vector<uint64_t> vertex_off;  // nblocks+1
    uint64_t vertices = 0, nodes = 0, tiles = 0, entries = 0;
    uint64_t brick_elems = 0;          // elements of the brick store (rows padded to the pitch)
    std::vector<uint32_t> pitch;       // per block: brick row pitch in elements
    // device
    PlanBlock* blocks_dev = nullptr;
    uint2* items_dev = nullptr;
    uint64_t* entry_off_dev = nullptr;
    uint16_t* entry_local_dev = nullptr;
    uint32_t* entry_node_dev = nullptr;
    uint32_t* flags_dev = nullptr;
    uint32_t flag_words = 1;
    uint32_t* centry_off_dev = nullptr; // per block the sparse nodes on its coarse grid
    uint2* centry_dev = nullptr;
    float* coarse_dev[2] = {nullptr, nullptr}; // per data slot: the blocks' coarse grids of the frame
    bool any_coarse = false;
    uint32_t* queue_dev = nullptr;
    uint64_t* node_off_dev = nullptr;
    float2* scale_offset_dev = nullptr;
    // the second data slot of s3r_frame_run_host (slot 0 is the brick store above): its own bricks and
    // per-brick 16-bit scales, so that two frames can be on the GPU at once
    void* bricks_1 = nullptr;
    float2* scale_offset_1 = nullptr;
    void* bricks = nullptr;
    // what is staged with a view, one allocation and one copy: the table, the view, the cover and the block list
    void* stage_dev = nullptr;
    void* stage_pinned = nullptr;
    size_t stage_bytes = 0;
    RenderBlock* table_dev = nullptr;
    s3r_view* view_dev = nullptr;
    int32_t* cover_dev = nullptr;    // union of the present blocks' view rectangles {x0, y0, x1, y1}
    uint2* seg_list_dev = nullptr;   // the blocks' {key, first item}, deepest first, and {0, items}
    uint32_t grid_ctas = 0;
    // host render table (rects depend on the view)
    std::vector<RenderBlock> table_host;
    RenderBlock* table_pinned = nullptr;
    s3r_view* view_pinned = nullptr;
    int32_t* cover_pinned = nullptr;
    uint2* seg_list_pinned = nullptr;
    cudaEvent_t staged = nullptr;   // the staging copy
    cudaEvent_t expanded = nullptr; // the work items expanded from it
    bool have_view = false;
    s3r_view last_view{};
    // frame graphs: slot 0 for s3r_frame_run, slots 1 and 2 for the two buffers of s3r_frame_run_host
    FrameGraph graphs[3];
    float* dtf_part = nullptr; // adjoint: kDtfParts copies of the transfer-function gradient
    size_t dtf_part_floats = 0;
    // block-major render: the block cells deepest first, the work items of the staged view, per data slot the
    // per-rank block results and rank masks, and one work-queue counter per data slot
    std::vector<uint32_t> seg_order;
    int staged_tile = -1;               // the render tile the view is staged for (-1: the table alone)
    bool seg_now = false;               // the staged view renders block-major
    bool seg_lanes = false;             // some of them have several lanes to a ray
    uint32_t* seg_queue = nullptr;      // 2 counters
    float4* seg_buf[2] = {nullptr, nullptr};
    unsigned long long* seg_mask[2] = {nullptr, nullptr}; // behind seg_buf, in its allocation
    uint2* seg_items_dev = nullptr;     // SegArgs::items, expanded from the block list; behind seg_mask[0]
    uint64_t seg_items_cap = 0;
    uint64_t seg_pixels[2] = {0, 0};    // pixels the buffers hold
    uint32_t seg_words = 0;
    // a data slot's block-major frames, on whatever streams, take its results, masks and queue counter in turn
    cudaEvent_t seg_done[2] = {nullptr, nullptr};
    unsigned long long seg_user[2] = {~0ull, ~0ull}; // the stream of the last one (its id: a handle may come again)
    std::mutex seg_turn;
    // s3r_frame_run_host: per slot a device copy of the frame's sparse values and its image, and the
    // streams and events that overlap frame k's copies with frames k-1 and k+1
    float* hs_sparse[2] = {nullptr, nullptr};
    uint32_t* hs_argb[2] = {nullptr, nullptr};
    float* hs_tf[2] = {nullptr, nullptr}; // per slot: the frame's transfer function, copied on the caller's stream
    uint32_t hs_tf_n = 0;
    uint64_t hs_pixels = 0;
    uint64_t hs_frames = 0;
    cudaStream_t hs_h2d = nullptr, hs_d2h = nullptr;
    cudaStream_t hs_comp[2] = {nullptr, nullptr}; // one compute stream per slot: frames k and k+1 overlap
    cudaEvent_t hs_copied[2] = {nullptr, nullptr}, hs_rendered[2] = {nullptr, nullptr}, hs_read[2] = {nullptr, nullptr};
    cudaEvent_t hs_entry = nullptr; // work queued on the caller's stream before a frame
};

// A block's dense field as the reference holds it for rendering (DeviceField, DenseFieldRenderer_cu.cu:503-560):
// a 3-D float array with a texture object over it (unnormalized coordinates, linear filtering, clamp).
struct s3r_texture {
    s3r_ctx* ctx = nullptr;
    uint32_t depth = 0, n = 0;
    cudaArray_t array = nullptr;
    cudaTextureObject_t tex = 0;
    cudaSurfaceObject_t surf = 0; // the interpolation writes the array in place
};

// The transfer function as the reference's colour texture (makeColorTransferTexture,
// DenseFieldRenderer_cu.cu:566-586): one row of RGBA floats, normalized coordinates, linear filtering,
// clamp along x.
struct s3r_tf_texture {
    s3r_ctx* ctx = nullptr;
    uint32_t n = 0;
    cudaArray_t array = nullptr;
    cudaTextureObject_t tex = 0;
};

void s3r::set_thread_error(const char* msg) { g_last_error = msg; }
void s3r::count_launches(s3r_ctx* ctx, uint32_t n)
{
    if (ctx) ctx->launches += n;
}

namespace {

int fail(s3r_ctx* ctx, int code, const std::string& msg)
{
    g_last_error = msg;
    if (ctx) ctx->err = msg;
    return code;
}

int cuda_fail(s3r_ctx* ctx, cudaError_t e, const char* what)
{
    if (ctx) ctx->last_cuda = e;
    return fail(ctx, S3R_ERR_CUDA, std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")");
}

#define S3R_CUDA(ctx, call)                                   \
    do {                                                      \
        cudaError_t e_ = (call);                              \
        if (e_ != cudaSuccess) return cuda_fail(ctx, e_, #call); \
    } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

int set_device(s3r_ctx* ctx)
{
    int cur = -1;
    cudaError_t e = cudaGetDevice(&cur);
    if (e == cudaSuccess && cur == ctx->device) return S3R_OK;
    e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaSetDevice");
    return S3R_OK;
}

// ---------------------------------------------------------------- geometry

void block_cube_f(uint32_t level, const uint32_t idx[3], float c[3], float& h)
{
    const float top = 5.f;
    h = top / (float)(1u << level);
    for (int d = 0; d < 3; ++d)
        c[d] = -top + h * (float)(1u + (idx[d] << 1));
}

int clampi(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }

// DenseFieldRenderer_cu.cu:374-409: bounding box of the projected cube corners,
// truncated toward zero, clamped to the viewport; {x, y, w, h} with w = max - min.
// Every block of a level goes through this whenever the camera moves, so the 8
// corners are worked out side by side (arrays the compiler vectorizes) from the
// products of the 2 coordinates they have per axis; each corner's sums and
// quotients are rounded as the one-by-one form rounds them.
void view_rect(const s3r_view& v, const uint32_t idx[3], int32_t rect[4])
{
    float c[3], h;
    block_cube_f(v.level, idx, c, h);
    const float lcam = 0.01f * 2 * 5.f;
    const float pixel = v.cam.h / (float)v.H;
    const float* r = v.cam.view_r;
    const float* t = v.cam.view_t;
    float q[3][8];
    for (int a = 0; a < 3; ++a) {
        float prod[3][2];
        for (int d = 0; d < 3; ++d) {
            prod[d][0] = r[3 * a + d] * (c[d] - h);
            prod[d][1] = r[3 * a + d] * (c[d] + h);
        }
        for (int i = 0; i < 8; ++i) q[a][i] = prod[0][i & 1] + prod[1][(i >> 1) & 1] + prod[2][i >> 2] + t[a];
    }
    float fx[8], fy[8];
    bool full = false;
    if (v.cam.ortho) {
        for (int i = 0; i < 8; ++i) {
            fx[i] = q[0][i] / pixel;
            fy[i] = q[1][i] / pixel;
        }
    } else {
        for (int i = 0; i < 8; ++i) full |= q[2][i] >= 0;
        for (int i = 0; i < 8 && !full; ++i) {
            fx[i] = -q[0][i] / q[2][i] * lcam / pixel;
            fy[i] = -q[1][i] / q[2][i] * lcam / pixel;
        }
    }
    if (full) {
        // a corner behind the eye: the whole viewport (bb << {0,0} << viewportSize)
        rect[0] = rect[1] = 0;
        rect[2] = (int)v.W;
        rect[3] = (int)v.H;
        return;
    }
    int xmin = INT32_MAX, xmax = INT32_MIN, ymin = INT32_MAX, ymax = INT32_MIN;
    for (int i = 0; i < 8; ++i) {
        const int sx = clampi((int)fx[i] + (int)(v.W >> 1), 0, (int)v.W - 1);
        const int sy = clampi((int)fy[i] + (int)(v.H >> 1), 0, (int)v.H - 1);
        xmin = std::min(xmin, sx);
        xmax = std::max(xmax, sx);
        ymin = std::min(ymin, sy);
        ymax = std::max(ymax, sy);
    }
    rect[0] = xmin;
    rect[1] = ymin;
    rect[2] = xmax - xmin;
    rect[3] = ymax - ymin;
}

int check_view(s3r_ctx* ctx, const s3r_view* v)
{
    if (!v) return fail(ctx, S3R_ERR_INVALID, "view is null");
    if (v->W == 0 || v->H == 0 || v->W > 32768 || v->H > 32768)
        return fail(ctx, S3R_ERR_INVALID, "viewport size out of range");
    if (v->tf_n < 2 || v->tf_n > 4096) return fail(ctx, S3R_ERR_INVALID, "tf_n must be in [2, 4096]");
    if (v->level > 12) return fail(ctx, S3R_ERR_INVALID, "level out of range");
    if (!(v->field_max > v->field_min)) return fail(ctx, S3R_ERR_INVALID, "field range is empty");
    if (!(v->quality > 0.f)) return fail(ctx, S3R_ERR_INVALID, "quality must be positive");
    if (v->filter != S3R_FILTER_EXACT && v->filter != S3R_FILTER_TEXTURE)
        return fail(ctx, S3R_ERR_INVALID, "unknown filter");
    return S3R_OK;
}

// ---------------------------------------------------------------- ordering

// Split of one index range by one eye coordinate (UniformIndexRangeSplitter,
// include/UniformIndexRangeSplitter.hpp:27-57), in the reference's float type.
struct Split {
    uint32_t before[2];
    uint32_t at; // ~0u: none
    uint32_t after[2];
};

Split split_range(uint32_t lo, uint32_t hi, float c0, float c1, float x)
{
    Split s;
    if (x <= c0) {
        s.before[0] = s.before[1] = 0;
        s.at = ~0u;
        s.after[0] = lo;
        s.after[1] = hi;
        return s;
    }
    if (x >= c1) {
        s.before[0] = lo;
        s.before[1] = hi;
        s.at = ~0u;
        s.after[0] = s.after[1] = 0;
        return s;
    }
    const float factor = (float)(hi - lo) / (c1 - c0);
    const uint32_t at = (uint32_t)((x - c0) * factor) + lo;
    s.before[0] = lo;
    s.before[1] = at;
    s.at = at;
    s.after[0] = at + 1;
    s.after[1] = hi;
    return s;
}

// Split of the box index range [0, n) by one eye coordinate when the boxes' boundaries sit at coords[0..n]
// (NonUniformIndexRangeSplitter, include/NonUniformIndexRangeSplitter.hpp:27-56): the first boundary not below
// x decides, so an eye exactly on a boundary belongs to the box before it.
Split split_boundaries(const float* coords, uint32_t n, float x)
{
    const float* it = std::lower_bound(coords, coords + n + 1, x);
    Split s;
    if (it == coords) {
        s.before[0] = s.before[1] = 0;
        s.at = ~0u;
        s.after[0] = 0;
        s.after[1] = n;
    } else if (it == coords + n + 1) {
        s.before[0] = 0;
        s.before[1] = n;
        s.at = ~0u;
        s.after[0] = s.after[1] = 0;
    } else {
        const uint32_t at = (uint32_t)(it - coords) - 1;
        s.before[0] = 0;
        s.before[1] = at;
        s.at = at;
        s.after[0] = at + 1;
        s.after[1] = n;
    }
    return s;
}

// Macro-block visiting order: the 27 cells of the 3x3x3 split (0 = before the
// eye, 1 = at it, 2 = beyond it per axis) taken corners first, then edges,
// faces and the eye's own cell (include/BackToFrontOrder.hpp:182-209).
constexpr uint8_t kMacroOrder[27] = {0, 2, 6, 8, 18, 20, 24, 26, 1, 3, 5, 7, 9, 11,
                                     15, 17, 19, 21, 23, 25, 4, 10, 12, 14, 16, 22, 13};

// Inside one macro block: anti-diagonal sweeps of increasing coordinate sum,
// the same successor rule as include/BackToFrontOrder.hpp:246-307 (unsigned
// arithmetic kept), mirrored on axes beyond the eye.
bool next_in_box(uint32_t p[3], const uint32_t mn[3], const uint32_t mx[3])
{
    uint32_t s = p[0] + p[1] + p[2];
    if (s + 3 == mx[0] + mx[1] + mx[2]) return false;
    if (p[0] > mn[0] && p[1] + 1 < mx[1]) {
        --p[0];
        ++p[1];
    } else if (p[0] + p[1] > mn[0] + mn[1] && p[2] + 1 < mx[2]) {
        if (s - mn[1] - p[2] < mx[0] + 1) {
            p[0] = s - mn[1] - p[2] - 1;
            p[1] = mn[1];
            p[2] = p[2] + 1;
        } else {
            p[0] = mx[0] - 1;
            p[1] = s - mx[0] - p[2];
            p[2] = p[2] + 1;
        }
    } else {
        ++s;
        const uint32_t x0 = s - mn[1] - mn[2];
        if (x0 < mx[0]) {
            p[0] = x0;
            p[1] = mn[1];
            p[2] = mn[2];
        } else {
            const uint32_t x1 = s - mx[0] + 1 - mn[2];
            if (x1 < mx[1]) {
                p[0] = mx[0] - 1;
                p[1] = x1;
                p[2] = mn[2];
            } else {
                p[0] = mx[0] - 1;
                p[1] = mx[1] - 1;
                p[2] = s + 2 - mx[0] - mx[1];
            }
        }
    }
    return true;
}

// Visits a 3-D index grid in back-to-front order for the per-axis splits of
// the eye (BackToFrontOrder::iterator, include/BackToFrontOrder.hpp:79-320):
// macro blocks in kMacroOrder, inside each the anti-diagonal sweep, mirrored on
// axes beyond the eye.  f(pos) gets each index triple.
template <class F> void b2f_traverse(const Split sp[3], F&& f)
{
    for (uint8_t ord : kMacroOrder) {
        const uint32_t mp[3] = {ord % 3u, (ord / 3u) % 3u, ord / 9u};
        uint32_t mn[3], mx[3];
        bool valid = true;
        for (int a = 0; a < 3; ++a) {
            const Split& s = sp[a];
            if (mp[a] == 0) {
                mn[a] = s.before[0];
                mx[a] = s.before[1];
                valid &= s.before[0] != s.before[1];
            } else if (mp[a] == 1) {
                mn[a] = s.at;
                mx[a] = s.at + 1;
                valid &= s.at != ~0u;
            } else {
                mn[a] = s.after[0];
                mx[a] = s.after[1];
                valid &= s.after[0] != s.after[1];
            }
        }
        if (!valid) continue;
        uint32_t p[3] = {mn[0], mn[1], mn[2]};
        do {
            uint32_t q[3];
            for (int a = 0; a < 3; ++a) q[a] = mp[a] == 2 ? mx[a] - 1 + mn[a] - p[a] : p[a];
            f(q);
        } while (next_in_box(p, mn, mx));
    }
}

// IndexCubeSplitter<3> (include/IndexCubeSplitter.hpp:36-196) over the world cube [-5, 5]^3: per axis the
// number of slabs (split_count taken greedily along x, then y, then z, each at most 2^level) and their
// index boundaries i*size/slabs and world boundaries (the float formula of init_axis_split).
struct CubeSplit {
    uint32_t n[3];
    std::vector<uint32_t> idx[3];
    std::vector<float> coord[3];
};

CubeSplit cube_split(uint32_t level, uint32_t split_count)
{
    CubeSplit cs;
    const uint32_t size = 1u << level;
    const uint64_t max_split = 1ull << (3 * level);
    uint32_t count = (uint32_t)std::min<uint64_t>(max_split, split_count);
    for (int a = 0; a < 3; ++a) {
        if (count <= size) {
            cs.n[a] = count;
            count = 1;
        } else {
            cs.n[a] = size;
            count = std::max(1u, count / size);
        }
    }
    const float origin = -5.f, length = 10.f;
    for (int a = 0; a < 3; ++a) {
        const uint32_t k = cs.n[a];
        cs.idx[a].assign(k + 1, 0);
        cs.coord[a].assign(k + 1, 0.f);
        cs.idx[a][k] = size;
        cs.coord[a][0] = origin;
        cs.coord[a][k] = origin + length;
        for (uint32_t i = 1; i < k; ++i) {
            const uint32_t si = (uint32_t)((uint64_t)i * size / k);
            cs.idx[a][i] = si;
            cs.coord[a][i] = origin + length * (float)si / (float)size;
        }
    }
    return cs;
}

void put_box(const CubeSplit& cs, const uint32_t q[3], uint32_t* out)
{
    for (int a = 0; a < 3; ++a) {
        out[a] = cs.idx[a][q[a]];
        out[3 + a] = cs.idx[a][q[a] + 1];
    }
}

// ---------------------------------------------------------------- plan

void plan_free_device(s3r_plan* p)
{
    auto f = [](void* q) {
        if (q) cudaFree(q);
    };
    f(p->blocks_dev);
    f(p->items_dev);
    f(p->entry_off_dev);
    f(p->entry_local_dev);
    f(p->entry_node_dev);
    f(p->flags_dev);
    f(p->centry_off_dev);
    f(p->centry_dev);
    f(p->coarse_dev[0]);
    f(p->coarse_dev[1]);
    p->centry_off_dev = nullptr;
    p->centry_dev = nullptr;
    p->coarse_dev[0] = p->coarse_dev[1] = nullptr;
    p->blocks_dev = nullptr;
    p->items_dev = nullptr;
    p->entry_off_dev = nullptr;
    p->entry_local_dev = nullptr;
    p->entry_node_dev = nullptr;
    p->flags_dev = nullptr;
}

void plan_drop_graph(s3r_plan* p)
{
    for (auto& g : p->graphs) {
        if (g.exec) cudaGraphExecDestroy(g.exec);
        g = FrameGraph{};
    }
}

template <class T> int upload(s3r_ctx* ctx, T** dst, const std::vector<T>& src)
{
    const size_t bytes = std::max<size_t>(src.size(), 1) * sizeof(T);
    cudaError_t e = cudaMalloc(dst, bytes);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc(plan)");
    if (!src.empty()) {
        e = cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMemcpy(plan)");
    }
    return S3R_OK;
}

// Bins every block's nodes by tile of 2^tile_log2 cells (closed tiles: nodes on
// shared faces, edges and corners go to every tile containing them; in a block
// of several tiles the lattice points of the tile grid go to the block's coarse
// grid instead, whose values every frame computes once per block), lists the
// coarse-grid nodes and the work items (largest tiles first), and uploads them.
// by_depth: per block depth the tile edge (log2 cells) of that depth's blocks; NULL: tile_log2 for all.
int plan_bin(s3r_plan* p, uint32_t tile_log2, const uint8_t* by_depth = nullptr)
{
    s3r_ctx* ctx = p->ctx;
    const uint32_t nb = p->nblocks;
    std::vector<PlanBlock> pb(nb);
    std::vector<uint64_t> tiles_off(nb + 1, 0), coarse_off(nb + 1, 0);
    uint8_t tl_of[S3R_MAX_DEPTH + 1];
    for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d)
        tl_of[d] = (uint8_t)std::min<uint32_t>(by_depth ? by_depth[d] : tile_log2, d);
    tile_log2 = 0;
    for (uint32_t b = 0; b < nb; ++b) tile_log2 = std::max<uint32_t>(tile_log2, tl_of[p->blocks[4 * b + 3]]);
    for (uint32_t b = 0; b < nb; ++b) {
        const uint32_t d = p->blocks[4 * b + 3];
        const uint32_t k = tl_of[d];
        const uint32_t L = d - k;
        pb[b].depth = d;
        pb[b].tile_log2 = k;
        pb[b].coarse_log2 = L;
        pb[b].node_base = p->node_off[b];
        pb[b].dense_off = p->vertex_off[b];
        pb[b].pitch = p->pitch[b];
        const uint64_t m = 1ull << L;
        tiles_off[b + 1] = tiles_off[b] + m * m * m;
        coarse_off[b + 1] = coarse_off[b] + (m + 1) * (m + 1) * (m + 1);
    }
    if (coarse_off[nb] > 0xffffffffull) return fail(ctx, S3R_ERR_INVALID, "coarse grids too large");
    for (uint32_t b = 0; b < nb; ++b) pb[b].coarse_off = (uint32_t)coarse_off[b];
    const uint64_t ntiles = tiles_off[nb];
    std::vector<int32_t> coarse(coarse_off[nb], -1);
    std::vector<uint64_t> count(ntiles + 1, 0);

    const unsigned nthreads = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    auto parallel = [&](auto&& fn) {
        std::vector<std::thread> th;
        for (unsigned t = 0; t < nthreads; ++t)
            th.emplace_back([&, t] {
                for (uint32_t b = t; b < nb; b += nthreads) fn(b);
            });
        for (auto& x : th) x.join();
    };
    auto tile_span = [](uint32_t x, uint32_t T, uint32_t m, uint32_t& lo, uint32_t& hi) {
        lo = x == 0 ? 0 : (x - 1) / T;
        hi = std::min(x / T, m - 1);
    };
    // pass 1: counts and coarse grids
    parallel([&](uint32_t b) {
        const PlanBlock& B = pb[b];
        const uint32_t T = 1u << B.tile_log2, m = 1u << B.coarse_log2, m1 = m + 1;
        for (uint64_t i = p->node_off[b]; i < p->node_off[b + 1]; ++i) {
            const uint32_t x = p->n2i[3 * i], y = p->n2i[3 * i + 1], z = p->n2i[3 * i + 2];
            const bool lattice = (x % T == 0) && (y % T == 0) && (z % T == 0);
            if (lattice) coarse[B.coarse_off + (x / T) + m1 * ((y / T) + m1 * (z / T))] = (int32_t)(i - p->node_off[b]);
            if (lattice && B.coarse_log2 > 0) continue;
            uint32_t xl, xh, yl, yh, zl, zh;
            tile_span(x, T, m, xl, xh);
            tile_span(y, T, m, yl, yh);
            tile_span(z, T, m, zl, zh);
            for (uint32_t tz = zl; tz <= zh; ++tz)
                for (uint32_t ty = yl; ty <= yh; ++ty)
                    for (uint32_t tx = xl; tx <= xh; ++tx)
                        ++count[tiles_off[b] + tx + m * (ty + m * tz)];
        }
    });
    // items: largest tiles first, then block order
    std::vector<uint64_t> order(ntiles);
    {
        std::vector<uint32_t> bord(nb);
        for (uint32_t b = 0; b < nb; ++b) bord[b] = b;
        std::stable_sort(bord.begin(), bord.end(),
                         [&](uint32_t a, uint32_t c) { return pb[a].tile_log2 > pb[c].tile_log2; });
        uint64_t o = 0;
        for (uint32_t b : bord)
            for (uint64_t t = tiles_off[b]; t < tiles_off[b + 1]; ++t) order[o++] = t;
    }
    std::vector<uint2> items(ntiles);
    std::vector<uint64_t> entry_off(ntiles + 1, 0);
    std::vector<uint64_t> slot(ntiles); // tile (block-major) -> item position
    std::vector<uint32_t> tile_block(ntiles);
    for (uint32_t b = 0; b < nb; ++b)
        for (uint64_t t = tiles_off[b]; t < tiles_off[b + 1]; ++t) tile_block[t] = b;
    for (uint64_t it = 0; it < ntiles; ++it) {
        const uint64_t t = order[it];
        slot[t] = it;
        const uint32_t b = tile_block[t];
        items[it] = make_uint2(b, (uint32_t)(t - tiles_off[b]));
        entry_off[it + 1] = entry_off[it] + count[t];
    }
    const uint64_t nentries = entry_off[ntiles];
    if (nentries > 0xffffffffull) return fail(ctx, S3R_ERR_INVALID, "too many tile entries (2^32 or more)");
    std::vector<uint16_t> local(nentries);
    std::vector<uint32_t> node(nentries);
    // per item: one bit per finest 2x2x2 cube of the tile, set when one of the cube's midpoints holds
    // a node (the cube along each odd axis of the node, both neighbours along each even one)
    const uint32_t hmax = std::max(1u, (1u << tile_log2) / 2);
    const uint32_t fwords = std::max(1u, (hmax * hmax * hmax + 31) / 32);
    std::vector<uint32_t> flags(ntiles * fwords, 0u);
    auto flag_node = [&](uint32_t* f, uint32_t H, uint32_t x, uint32_t y, uint32_t z) {
        if (!((x | y | z) & 1)) return;
        auto span = [H](uint32_t v, uint32_t& lo, uint32_t& hi) {
            if (v & 1) {
                lo = hi = v >> 1;
            } else {
                lo = v ? (v >> 1) - 1 : 0;
                hi = std::min(v >> 1, H - 1);
            }
        };
        uint32_t x0, x1, y0, y1, z0, z1;
        span(x, x0, x1);
        span(y, y0, y1);
        span(z, z0, z1);
        for (uint32_t k = z0; k <= z1; ++k)
            for (uint32_t j = y0; j <= y1; ++j)
                for (uint32_t i = x0; i <= x1; ++i) {
                    const uint32_t c = i + H * (j + H * k);
                    f[c >> 5] |= 1u << (c & 31);
                }
    };
    std::vector<uint64_t> cursor(ntiles);
    for (uint64_t t = 0; t < ntiles; ++t) cursor[t] = entry_off[slot[t]];
    // pass 2: fill (tiles of one block are only touched by that block's thread)
    parallel([&](uint32_t b) {
        const PlanBlock& B = pb[b];
        const uint32_t T = 1u << B.tile_log2, m = 1u << B.coarse_log2, E = T + 1;
        for (uint64_t i = p->node_off[b]; i < p->node_off[b + 1]; ++i) {
            const uint32_t x = p->n2i[3 * i], y = p->n2i[3 * i + 1], z = p->n2i[3 * i + 2];
            const bool lattice = (x % T == 0) && (y % T == 0) && (z % T == 0);
            if (lattice && B.coarse_log2 > 0) continue;
            uint32_t xl, xh, yl, yh, zl, zh;
            tile_span(x, T, m, xl, xh);
            tile_span(y, T, m, yl, yh);
            tile_span(z, T, m, zl, zh);
            for (uint32_t tz = zl; tz <= zh; ++tz)
                for (uint32_t ty = yl; ty <= yh; ++ty)
                    for (uint32_t tx = xl; tx <= xh; ++tx) {
                        const uint64_t t = tiles_off[b] + tx + m * (ty + m * tz);
                        const uint64_t e = cursor[t]++;
                        local[e] = (uint16_t)tile_offset(T, x - tx * T, y - ty * T, z - tz * T);
                        node[e] = (uint32_t)(i - p->node_off[b]);
                        if (T >= 2)
                            flag_node(&flags[slot[t] * fwords], T / 2, x - tx * T, y - ty * T, z - tz * T);
                    }
        }
        (void)E;
    });
    // the nodes on every block's coarse grid (the lattice of tile corners), once per block: the frame's
    // block_prep_kernel fills the coarse grids from them
    std::vector<uint32_t> centry_off(nb + 1, 0);
    std::vector<uint2> centry;
    for (uint32_t b = 0; b < nb; ++b) {
        if (pb[b].coarse_log2 > 0) {
            const uint64_t n = coarse_off[b + 1] - coarse_off[b];
            for (uint64_t q = 0; q < n; ++q) {
                const int32_t nd = coarse[coarse_off[b] + q];
                if (nd >= 0) centry.push_back(make_uint2((uint32_t)q, (uint32_t)nd));
            }
        }
        if (centry.size() > 0xffffffffull) return fail(ctx, S3R_ERR_INVALID, "too many coarse-grid nodes");
        centry_off[b + 1] = (uint32_t)centry.size();
    }
    // items whose tile holds no node at an odd position have no flagged cube, so nothing reads their
    // midpoint slots: the top bit of the tile field says "fill the slots"
    for (uint64_t it = 0; it < ntiles; ++it)
        for (uint32_t w = 0; w < fwords; ++w)
            if (flags[it * fwords + w]) {
                items[it].y |= 0x80000000u;
                break;
            }
    plan_free_device(p);
    int rc;
    if ((rc = upload(ctx, &p->blocks_dev, pb))) return rc;
    if ((rc = upload(ctx, &p->items_dev, items))) return rc;
    if ((rc = upload(ctx, &p->entry_off_dev, entry_off))) return rc;
    if ((rc = upload(ctx, &p->entry_local_dev, local))) return rc;
    if ((rc = upload(ctx, &p->entry_node_dev, node))) return rc;
    if ((rc = upload(ctx, &p->flags_dev, flags))) return rc;
    if ((rc = upload(ctx, &p->centry_off_dev, centry_off))) return rc;
    if ((rc = upload(ctx, &p->centry_dev, centry))) return rc;
    p->any_coarse = false;
    for (uint32_t b = 0; b < nb; ++b) p->any_coarse |= pb[b].coarse_log2 > 0;
    for (int q = 0; q < 2; ++q) {
        cudaError_t e = cudaMalloc(&p->coarse_dev[q], std::max<uint64_t>(coarse_off[nb], 1) * sizeof(float));
        if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc(coarse grids)");
    }
    p->flag_words = fwords;
    p->tile_log2 = tile_log2;
    std::memcpy(p->tile_by_depth, tl_of, sizeof(tl_of));
    p->tiles = ntiles;
    p->entries = nentries;
    // persistent grid: the CTAs that fit on every SM at once, fed by the work queue
    const uint32_t per_sm = interp_plan_ctas_per_sm(p->fmt, tile_log2);
    p->grid_ctas = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(ntiles, (uint64_t)ctx->sms * per_sm));
    plan_drop_graph(p);
    return S3R_OK;
}

// Whether the caller is capturing this stream (the legacy stream cannot be captured, nor asked about while another is).
bool capturing(cudaStream_t s)
{
    if (!s || s == cudaStreamLegacy) return false;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &status) != cudaSuccess) (void)cudaGetLastError();
    return status != cudaStreamCaptureStatusNone;
}

void plan_free_segments(s3r_plan* p)
{
    for (int b = 0; b < 2; ++b) {
        if (p->seg_buf[b]) cudaFree(p->seg_buf[b]);
        p->seg_buf[b] = nullptr;
        p->seg_mask[b] = nullptr;
        p->seg_pixels[b] = 0;
    }
    p->seg_items_dev = nullptr;
    p->seg_items_cap = 0;
}

uint64_t seg_pixel_bytes(const s3r_plan* p) { return (3ull * (1u << p->level) - 2) * sizeof(float4); }

// The block-major render's per-rank results and rank masks for `npix` pixels (`roomy` where they are allocated), in the
// second data slot too once there is a host-buffer pipeline, and behind those of the first slot room for `items` work
// items.  Called before a frame is
// launched in the block-major form.  The first allocation waits for nothing; a slot that has become too small waits for
// the frames that use it and is allocated again, which drops the plan's captured frames (they hold the old buffers).
// (In stream order, by cudaMallocAsync and cudaFreeAsync, a larger view's first frame takes 290 instead of 360 us, but a
// plan's first one, which maps new memory, 730 instead of 520: 512 mixed blocks at 1920x1080.)
int plan_ensure_segments(s3r_plan* p, uint64_t npix, uint64_t roomy, uint64_t items, cudaStream_t s)
{
    s3r_ctx* ctx = p->ctx;
    const uint32_t words = (3 * (1u << p->level) - 2 + 63) / 64;
    p->seg_words = words;
    for (int b = 0; b < (p->hs_h2d ? 2 : 1); ++b) {
        if (p->seg_buf[b] && p->seg_pixels[b] >= npix && (b || p->seg_items_cap >= items)) continue;
        if (capturing(s)) return fail(ctx, S3R_ERR_UNSUPPORTED, "allocation in a stream capture");
        std::lock_guard<std::mutex> lock(p->seg_turn);
        plan_drop_graph(p);
        if (p->seg_buf[b]) {
            for (cudaEvent_t done : p->seg_done) S3R_CUDA(ctx, cudaEventSynchronize(done)); // both slots read the items
            cudaFree(p->seg_buf[b]);
        }
        p->seg_buf[b] = nullptr;
        const uint64_t pixels = p->seg_pixels[b] >= npix ? p->seg_pixels[b] : std::max(npix, roomy),
                       room = b ? 0 : (p->seg_items_cap >= items ? p->seg_items_cap : items + items / 4);
        p->seg_pixels[b] = 0;
        if (b == 0) p->seg_items_cap = 0;
        const size_t results = pixels * seg_pixel_bytes(p), masks = (size_t)words * pixels * sizeof(unsigned long long);
        const cudaError_t e = cudaMalloc(&p->seg_buf[b], results + masks + room * sizeof(uint2));
        if (e != cudaSuccess) {
            p->seg_buf[b] = nullptr;
            (void)cudaGetLastError(); // an allocation failure leaves no error behind for later launches
            return cuda_fail(ctx, e, "cudaMalloc(block-major render buffers)");
        }
        char* mask = reinterpret_cast<char*>(p->seg_buf[b]) + results;
        p->seg_mask[b] = reinterpret_cast<unsigned long long*>(mask);
        if (b == 0) p->seg_items_dev = reinterpret_cast<uint2*>(mask + masks);
        S3R_CUDA(ctx, cudaMemsetAsync(mask, 0, masks, s));
        S3R_CUDA(ctx, cudaEventRecord(p->seg_done[b], s)); // frames on other streams find it cleared
        p->seg_user[b] = ~0ull;
        p->seg_pixels[b] = pixels;
        if (b == 0) p->seg_items_cap = room;
    }
    return S3R_OK;
}

// Lanes to a ray (log2) for the block-major items of every depth.  A frame takes about its work spread over all warps
// plus the longest item's chain of samples; sharing a ray among lanes shortens the chains of deep blocks at the price
// of more items and instructions.  In units of a sample's time, measured on GB300: an item's set-up about 20, a ray of
// a block of 2^d cells 1.3 q 2^d on average, six tenths of a view rectangle's pixels hit the block, shared rays cost
// 1.35 as much, and the kernel that can share marches the others 1.2 times slower -- so sharing has to win clearly
// (level 2 of depths 3-7 at 800x600: 178 us without, 125 with; 64 blocks of depth 6 there: 157 without, 197 with).
// Returns the samples of an item's ray, averaged over the items.
double seg_lanes_by_depth(const s3r_plan* p, const RenderBlock* table, uint32_t fx, uint32_t fy, float quality,
                          uint32_t log_lanes[S3R_MAX_DEPTH + 1])
{
    constexpr double kSetup = 20, kHit = 0.6, kShared = 1.35, kSlower = 1.2, kMargin = 1.15;
    const double warps = 32.0 * p->ctx->sms;
    double items[S3R_MAX_DEPTH + 1] = {}, chain[S3R_MAX_DEPTH + 1];
    for (uint32_t cell : p->seg_order) {
        const RenderBlock& t = table[cell];
        if (t.rect[2] > 0 && t.rect[3] > 0)
            items[t.depth] += (double)(((uint32_t)t.rect[2] + fx - 1) / fx) * (((uint32_t)t.rect[3] + fy - 1) / fy);
    }
    for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d) {
        log_lanes[d] = 0;
        chain[d] = 1.3 * quality * (1u << d);
    }
    double best = 0, all = 0, samples = 0, longest = 0;
    for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d) {
        best += items[d] * (kSetup + kHit * chain[d]) / warps;
        all += items[d];
        samples += items[d] * chain[d];
    }
    for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d)
        if (items[d] > 0) longest = std::max(longest, kSetup + chain[d]);
    best += longest;
    // every chain length that some depth can have is tried as the longest one
    for (uint32_t d0 = 0; d0 <= S3R_MAX_DEPTH; ++d0)
        for (uint32_t l0 = 1; l0 <= 3 && items[d0] > 0; ++l0) {
            const double limit = chain[d0] / (1u << l0);
            uint32_t l[S3R_MAX_DEPTH + 1];
            double work = 0, top = 0;
            for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d) {
                l[d] = 0;
                if (items[d] == 0) continue;
                while (l[d] < 3 && chain[d] / (1u << l[d]) > limit * 1.001) ++l[d];
                const double own = chain[d] / (1u << l[d]);
                work += items[d] * (1u << l[d]) * (kSetup + kHit * own * (l[d] ? kShared : kSlower));
                if (items[d] > 0) top = std::max(top, kSetup + own);
            }
            const double t = (work / warps + top) * kMargin;
            if (t < best) {
                best = t;
                std::memcpy(log_lanes, l, sizeof(l));
            }
        }
    return all > 0 ? samples / all : 0;
}

// Whether a plan left to the render form's default (ids below kRenderShapes: one image from all of them) goes
// block-major for this view.  The measured line (depths 3-7 and 4 to 6, 200x150 to 1920x1080, from close up to far):
// with 64 blocks and more the walk's lanes sit in different blocks and wait for each other, and block-major is up to
// seven times faster (level 3, 200x150: 550 against 79 us); short segments in a large part of the image favour the
// walk, which writes no block results (level 4 of depth 3, close up: 711 against 878 us; level 2 of depths 3-7 with 19
// samples a ray, 783x588: 152 against 168; with 5 samples the second launch is not won back, 22 against 23); of 8
// blocks only small views of deep ones gain (66 against 42 us; of depth 3 the second launch costs more, 19 against 21),
// and a single one is the walk's.  Where rays may stop before their last block (alpha_stop below 1) it is the walk's
// too: block-major marches what lies behind opaque blocks (64 FP16 blocks of depth 6, 233x238: 74 against 157 us), and
// how opaque the data are is not known here.
// rects: the pixels of all view rectangles, each a ray and block that block-major sets up where the walk meets at most
// 3m - 2 blocks a ray.  Seen from outside they are 0.3 to 0.9 times as many; inside the level a block with a corner
// behind the eye has the whole viewport for its rectangle.  From 1.0 times on (1.3 in small views) the empty rays cost
// more than the march gains: level 3 of depths 3-5, 1280x720, 0.8 times: 670 against 668 us, 1.1: 781 against 712, 3.4:
// 1755 against 590; level 4 of depths 2-4, 320x200, 1.3: 133 against 157, 1.7: 152 against 117, 46 times: 2818 against
// 75.  Only views so small that their rays' chains set the time hide them: the walk takes about m (1.5 + 0.16 samples)
// us there, of which block-major saves half, and 1000 empty rays 0.027 us (64 blocks of depth 6, 50x50 pixels, 4.9
// times: 55 against 90 us; 240x160: 79 against 77; 64 of depths 2 and 3, 90x60: 24 against 21).
constexpr uint64_t kSegAutoBytes = 1ull << 30; // of block results and items
bool seg_pays(const s3r_plan* p, uint64_t covered, uint64_t rects, double samples, float quality,
              const uint32_t log_lanes[S3R_MAX_DEPTH + 1])
{
    if (p->level < 1 || p->level > 7 || covered == 0 || covered * seg_pixel_bytes(p) > kSegAutoBytes) return false;
    const double m = 1u << p->level;
    if ((double)rects > (covered < 100000 ? 1.3 : 1.0) * (double)covered * (3 * m - 2) &&
        (double)rects * 2.7e-5 > 0.5 * m * (1.5 + 0.16 * samples))
        return false;
    if (p->level == 1) {
        bool lanes = false; // shared rays of at least 32 samples
        for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d) lanes |= log_lanes[d] > 0 && 1.3 * quality * (1u << d) >= 32;
        return lanes && covered < 60000;
    }
    return samples >= 30 || (samples >= 8 && covered < 100000) || (samples >= 22 && covered < 1000000);
}

// frame: for s3r_frame_render and the frames of s3r_frame_run(_host), whose render may go block-major; the field modes
// and the adjoint read the table alone (with a block-major id the items are staged all the same, for a caller's graph).
int plan_stage_view(s3r_plan* p, const s3r_view* view, cudaStream_t s, bool frame)
{
    s3r_ctx* ctx = p->ctx;
    const bool asked = p->render_tile >= (uint32_t)kRenderWalkTiles; // block-major by its id
    if (asked && (3 * (1u << p->level) - 2 + 63) / 64 > kSegMaskWords)
        return fail(ctx, S3R_ERR_UNSUPPORTED, "the block-major render covers levels up to 7");
    // 8x4-pixel items unless asked: 16x2 take 293 against 306 us on 4096 mixed blocks (475 against 511 close up), and 1 to
    // 4 % more on 64 and 512 (64 of depth 6: 119 against 116); 4x8 take 0 to 18 % more than 8x4
    const int shape = asked ? (int)(p->render_tile - (uint32_t)kRenderWalkTiles) : 0;
    // a view staged for another form (the autotuner's) or, since then, for fewer data slots is staged again
    const bool same = p->have_view && std::memcmp(&p->last_view, view, sizeof(s3r_view)) == 0 &&
                      (!frame || (p->staged_tile == (int)p->render_tile &&
                                  (!p->seg_now || p->seg_buf[p->hs_h2d ? 1 : 0])));
    if (same) return S3R_OK;
    // the staging buffers may still feed an earlier copy
    S3R_CUDA(ctx, cudaEventSynchronize(p->staged));
    const uint32_t m = 1u << p->level;
    RenderBlock* tb = p->table_pinned;
    std::memcpy(tb, p->table_host.data(), sizeof(RenderBlock) * p->table_host.size());
    int32_t cover[4] = {INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN};
    uint64_t rects = 0; // pixels of all of them
    for (uint32_t b = 0; b < p->nblocks; ++b) {
        const uint32_t* bl = &p->blocks[4 * b];
        const uint32_t cell = bl[0] + m * (bl[1] + m * bl[2]);
        int32_t* r = tb[cell].rect;
        view_rect(*view, bl, r);
        if (r[2] > 0 && r[3] > 0) {
            cover[0] = std::min(cover[0], r[0]);
            cover[1] = std::min(cover[1], r[1]);
            cover[2] = std::max(cover[2], r[0] + r[2]);
            cover[3] = std::max(cover[3], r[1] + r[3]);
            rects += (uint64_t)r[2] * (uint64_t)r[3];
        }
    }
    if (cover[0] > cover[2]) cover[0] = cover[1] = cover[2] = cover[3] = 0;
    // block-major render: the warp-sized tiles of every block's view rectangle, deepest blocks first
    const uint64_t covered = (uint64_t)(cover[2] - cover[0]) * (uint64_t)(cover[3] - cover[1]);
    const uint32_t fx = (uint32_t)kSegShapeX[shape], fy = (uint32_t)kSegShapeY[shape];
    uint32_t log_lanes[S3R_MAX_DEPTH + 1];
    bool seg = false;
    if (asked || (frame && p->render_tile < (uint32_t)kRenderShapes && !capturing(s))) {
        const double samples = seg_lanes_by_depth(p, tb, fx, fy, view->quality, log_lanes);
        // a table that the walk refuses stays refused
        seg = asked || (view->tf_n <= kTfPlain && view->alpha_stop >= 1.f &&
                        seg_pays(p, covered, rects, samples, view->quality, log_lanes));
    }
    uint64_t n = 0; // work items
    if (seg) {
        p->seg_lanes = false;
        for (uint32_t i = 0; i < p->nblocks; ++i) {
            const uint32_t cell = p->seg_order[i];
            const RenderBlock& t = tb[cell];
            p->seg_list_pinned[i] = make_uint2(cell | log_lanes[t.depth] << kSegLanesShift, (uint32_t)n);
            if (t.rect[2] <= 0 || t.rect[3] <= 0) continue;
            uint32_t w, h;
            seg_footprint(fx, log_lanes[t.depth], w, h);
            n += (uint64_t)(((uint32_t)t.rect[2] + w - 1) / w) * (((uint32_t)t.rect[3] + h - 1) / h);
            p->seg_lanes |= log_lanes[t.depth] > 0;
        }
        p->seg_list_pinned[p->nblocks] = make_uint2(0, (uint32_t)n);
        if (asked && n > 0xffffffffull) return fail(ctx, S3R_ERR_INVALID, "too many block-major render items");
        if (!asked && covered * seg_pixel_bytes(p) + n * sizeof(uint2) > kSegAutoBytes) seg = false;
    }
    if (seg) {
        // some room to move closer in
        uint64_t roomy = std::min(covered + covered / 2, (uint64_t)view->W * view->H);
        if (!asked) roomy = std::min(roomy, kSegAutoBytes / seg_pixel_bytes(p));
        const int rc = plan_ensure_segments(p, std::max<uint64_t>(covered, 1), roomy, n, s);
        if (rc && asked) return rc;
        if (rc) {
            // no room: the walk gives the same image
            seg = false;
            ctx->err.clear();
            set_thread_error("");
        }
    }
    p->seg_now = seg;
    p->staged_tile = frame || asked ? (int)p->render_tile : -1;
    std::memcpy(p->cover_pinned, cover, sizeof(cover));
    *p->view_pinned = *view;
    S3R_CUDA(ctx, cudaMemcpyAsync(p->stage_dev, p->stage_pinned, p->stage_bytes, cudaMemcpyHostToDevice, s));
    S3R_CUDA(ctx, cudaEventRecord(p->staged, s)); // the pinned buffers may be filled again
    if (seg) {
        S3R_CUDA(ctx, launch_seg_items(p->seg_list_dev, p->nblocks, p->seg_items_dev, s));
        ++ctx->launches;
        S3R_CUDA(ctx, cudaEventRecord(p->expanded, s));
    }
    p->last_view = *view;
    p->have_view = true;
    return S3R_OK;
}

// slot 1: the second data slot of the host-buffer pipeline (its bricks, scales and work-queue counter)
int plan_launch_interp(s3r_plan* p, const float* sparse, cudaStream_t s, uint32_t* kernels, int slot = 0)
{
    s3r_ctx* ctx = p->ctx;
    float2* so = slot ? p->scale_offset_1 : p->scale_offset_dev;
    if (p->fmt != S3R_BRICK_F32 || p->any_coarse) {
        // 16-bit scales and coarse grids
        PrepArgs pa{};
        pa.blocks = p->blocks_dev;
        pa.node_off = p->node_off_dev;
        pa.sparse = sparse;
        pa.scale_offset = p->fmt != S3R_BRICK_F32 ? so : nullptr;
        pa.coarse = p->coarse_dev[slot ? 1 : 0];
        pa.centry_off = p->centry_off_dev;
        pa.centry = p->centry_dev;
        S3R_CUDA(ctx, launch_block_prep(pa, p->nblocks, p->max_nodes, (uint32_t)ctx->sms, s));
        ++*kernels;
    }
    TileArgs a{};
    a.blocks = p->blocks_dev;
    a.items = p->items_dev;
    a.nitems = (uint32_t)p->tiles;
    a.entry_off = p->entry_off_dev;
    a.entry_local = p->entry_local_dev;
    a.entry_node = p->entry_node_dev;
    a.flags = p->flags_dev;
    a.flag_words = p->flag_words;
    a.sparse = sparse;
    a.queue = p->queue_dev + slot;
    a.scale_offset = p->fmt == S3R_BRICK_F32 ? nullptr : so;
    a.coarse = p->coarse_dev[slot ? 1 : 0];
    a.out = slot ? p->bricks_1 : p->bricks;
    S3R_CUDA(ctx, cudaMemsetAsync(a.queue, 0, sizeof(uint32_t), s));
    S3R_CUDA(ctx, launch_interp_plan(a, p->fmt, p->tile_log2, p->grid_ctas, s));
    ++*kernels;
    return S3R_OK;
}

// Queues a frame's work on `s` by body(): a block-major one after the frames that used the data slot's results, masks
// and queue counter before it, whichever streams and threads they came from.  (A block-major render by its id in the
// caller's capture is ordered by the caller, its graph being launched where this cannot see it.)
template <class F> int plan_in_turn(s3r_plan* p, bool seg, int data, cudaStream_t s, F&& body)
{
    if (!seg || (p->render_tile >= (uint32_t)kRenderWalkTiles && capturing(s))) return body();
    unsigned long long id = 0;
    S3R_CUDA(p->ctx, cudaStreamGetId(s, &id));
    std::lock_guard<std::mutex> lock(p->seg_turn);
    if (p->seg_user[data] != id) S3R_CUDA(p->ctx, cudaStreamWaitEvent(s, p->seg_done[data], 0));
    p->seg_user[data] = ~0ull;
    const int rc = body();
    S3R_CUDA(p->ctx, cudaEventRecord(p->seg_done[data], s));
    p->seg_user[data] = id;
    return rc;
}

// Whether a frame of the staged view queued on `s` goes block-major.  What a caller captures in the default form walks:
// the graph may be replayed after other views, for which the results and items are allocated and cut anew, while the
// walk reads only memory that lives as long as the plan.
bool plan_block_major(const s3r_plan* p, cudaStream_t s)
{
    return p->seg_now && (p->render_tile >= (uint32_t)kRenderWalkTiles || !capturing(s));
}

int plan_launch_render(s3r_plan* p, const float* tf, float* rgba, uint32_t* argb, unsigned long long* samples,
                       bool seg, cudaStream_t s, uint32_t* kernels, int slot = 0)
{
    FrameArgs fa{};
    fa.view = p->view_dev;
    fa.table = p->table_dev;
    fa.bricks = slot ? p->bricks_1 : p->bricks;
    fa.tf = tf;
    fa.rgba = rgba;
    fa.argb = argb;
    fa.samples = samples;
    fa.scale_offset = p->fmt == S3R_BRICK_F32 ? nullptr : (slot ? p->scale_offset_1 : p->scale_offset_dev);
    fa.cover = p->cover_dev;
    if (p->staged_tile != (int)p->render_tile)
        return fail(p->ctx, S3R_ERR_INVALID, "view not staged for this render tile");
    if (seg) {
        const int data = slot ? 1 : 0;
        if (!p->seg_buf[data])
            return fail(p->ctx, S3R_ERR_INVALID, "block-major render buffers not allocated for this view");
        const bool asked = p->render_tile >= (uint32_t)kRenderWalkTiles;
        const uint32_t shape = asked ? p->render_tile - (uint32_t)kRenderWalkTiles : 0u;
        SegArgs sa{};
        sa.items = p->seg_items_dev;
        sa.count = &p->seg_list_dev[p->nblocks].y;
        sa.lanes = p->seg_lanes;
        sa.walk = !asked;
        sa.words = p->seg_words;
        sa.seg = p->seg_buf[data];
        sa.mask = p->seg_mask[data];
        sa.queue = p->seg_queue + data;
        S3R_CUDA(p->ctx, launch_frame_segments(fa, sa, p->last_view.W, p->last_view.H, p->last_view.tf_n, p->fmt, shape,
                                               p->last_view.filter, (uint32_t)p->ctx->sms, s));
        *kernels += 2;
        return S3R_OK;
    }
    S3R_CUDA(p->ctx, launch_frame_render(fa, p->last_view.W, p->last_view.H, p->last_view.tf_n, p->fmt,
                                         p->render_tile, p->last_view.filter, s));
    ++*kernels;
    return S3R_OK;
}

} // namespace

void s3r::block_sampling(uint32_t level, const uint32_t idx[3], uint32_t depth, RenderBlock& rb)
{
    block_cube_f(level, idx, rb.center, rb.half);
    const uint32_t n = (1u << depth) + 1u;
    rb.depth = depth;
    rb.texel = 2 * rb.half / (float)n;
    const double thalf = (double)rb.half + 0.5 * (double)rb.texel;
    for (int d = 0; d < 3; ++d) rb.origin[d] = rb.center[d] - (float)thalf;
    rb.factor = (float)((double)n / (2 * thalf));
}

int s3r::record_error(int code, const char* msg) { return fail(nullptr, code, msg); }

int s3r::record_cuda_error(cudaError_t e, const char* what) { return cuda_fail(nullptr, e, what); }

// ==================================================================== C ABI

extern "C" {

int s3r_abi_version(void) { return S3R_ABI_VERSION; }

const char* s3r_last_error(const s3r_ctx* ctx) { return ctx ? ctx->err.c_str() : g_last_error.c_str(); }

uint64_t s3r_ctx_launch_count(const s3r_ctx* ctx) { return ctx ? ctx->launches : 0; }

int s3r_ctx_create(int device, s3r_ctx** out)
{
    if (!out) return fail(nullptr, S3R_ERR_INVALID, "out is null");
    *out = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaGetDeviceCount");
    if (device < 0 || device >= n) return fail(nullptr, S3R_ERR_INVALID, "no such device");
    e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaSetDevice");
    s3r_ctx* c = new (std::nothrow) s3r_ctx;
    if (!c) return fail(nullptr, S3R_ERR_NOMEM, "out of host memory");
    c->device = device;
    cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device);
    if ((e = cudaMalloc(&c->rect_dev, 6 * sizeof(int32_t))) != cudaSuccess ||
        (e = cudaMemset(c->rect_dev, 0, 6 * sizeof(int32_t))) != cudaSuccess ||
        (e = cudaMallocHost(&c->rect_host, 5 * sizeof(int32_t))) != cudaSuccess ||
        (e = cudaStreamCreateWithFlags(&c->capture, cudaStreamNonBlocking)) != cudaSuccess) {
        s3r_ctx_destroy(c);
        return cuda_fail(nullptr, e, "context allocation");
    }
    *out = c;
    return S3R_OK;
}

int s3r_ctx_destroy(s3r_ctx* ctx)
{
    if (!ctx) return S3R_OK;
    cudaSetDevice(ctx->device);
    if (ctx->grid) cudaFree(ctx->grid);
    if (ctx->grid_bits) cudaFree(ctx->grid_bits);
    if (ctx->rect_dev) cudaFree(ctx->rect_dev);
    if (ctx->rect_host) cudaFreeHost(ctx->rect_host);
    if (ctx->parts_dev) cudaFree(ctx->parts_dev);
    if (ctx->capture) cudaStreamDestroy(ctx->capture);
    for (float* d : ctx->worker_dense)
        if (d) cudaFree(d);
    for (auto& per_field : ctx->worker_tex)
        for (auto& per_depth : per_field)
            for (s3r_texture* t : per_depth) s3r_texture_destroy(t);
    if (ctx->part_host) cudaFreeHost(ctx->part_host);
    if (ctx->part_dev) cudaFree(ctx->part_dev);
    if (ctx->part_lists) cudaFree(ctx->part_lists);
    s3r_tf_texture_destroy(ctx->worker_tf);
    delete ctx;
    return S3R_OK;
}

// The context's block interpolation scratch for this many scattered values and mask words (grown on demand).
static int ensure_grid(s3r_ctx* ctx, uint64_t values, uint64_t words)
{
    if (ctx->grid_cap < values) {
        if (ctx->grid) cudaFree(ctx->grid);
        ctx->grid = nullptr;
        ctx->grid_cap = 0;
        S3R_CUDA(ctx, cudaMalloc(&ctx->grid, values * sizeof(float)));
        ctx->grid_cap = values;
    }
    if (ctx->grid_bits_cap < words) {
        if (ctx->grid_bits) cudaFree(ctx->grid_bits);
        ctx->grid_bits = nullptr;
        ctx->grid_bits_cap = 0;
        S3R_CUDA(ctx, cudaMalloc(&ctx->grid_bits, words * sizeof(uint32_t)));
        ctx->grid_bits_cap = words;
    }
    return S3R_OK;
}

// One subtree from its nodes into a dense grid, or into the 3-D array behind `surface` when dense is NULL.
static int interp_block(s3r_ctx* ctx, const uint16_t* n2i, const float* sparse, uint32_t n, uint32_t depth, float* dense,
                        unsigned long long surface, cudaStream_t s)
{
    GridArgs a{};
    a.one = grid_block(n2i, sparse, n, depth);
    a.one.out = dense;
    a.one.surface = surface;
    a.nblocks = 1;
    a.tiles = grid_tiles(depth);
    a.depth_max = depth;
    const uint64_t words = a.one.direct ? 0 : grid_mask_words(depth);
    if (words) {
        if (int rc = ensure_grid(ctx, grid_vertices(depth), words)) return rc;
        a.vals = ctx->grid;
        a.bits = ctx->grid_bits;
    }
    uint32_t launches = 0;
    S3R_CUDA(ctx, launch_interp_grid(a, dense == nullptr, words ? n : 0, words, s, &launches));
    ctx->launches += launches;
    return S3R_OK;
}

int s3r_interp_dense(s3r_ctx* ctx, const uint16_t* n2i_xyz, const float* sparse, uint32_t n, uint32_t depth,
                     float* dense, void* stream)
{
    if (!ctx) return fail(nullptr, S3R_ERR_INVALID, "ctx is null");
    if (depth > S3R_MAX_DEPTH) return fail(ctx, S3R_ERR_INVALID, "depth exceeds S3R_MAX_DEPTH");
    if (!dense || (n > 0 && (!n2i_xyz || !sparse))) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    int rc = set_device(ctx);
    if (rc) return rc;
    return interp_block(ctx, n2i_xyz, sparse, n, depth, dense, 0, as_stream(stream));
}

int s3r_camera_look_at(const double eye[3], const double center[3], const double up[3], double fovy_deg, uint32_t W,
                       uint32_t H, int32_t ortho, double ortho_height, s3r_camera* out)
{
    if (!eye || !center || !up || !out || W == 0 || H == 0) return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    double z[3] = {eye[0] - center[0], eye[1] - center[1], eye[2] - center[2]};
    double zl = std::sqrt(z[0] * z[0] + z[1] * z[1] + z[2] * z[2]);
    if (!(zl > 0)) return fail(nullptr, S3R_ERR_INVALID, "eye equals center");
    for (double& c : z) c /= zl;
    double x[3] = {up[1] * z[2] - up[2] * z[1], up[2] * z[0] - up[0] * z[2], up[0] * z[1] - up[1] * z[0]};
    double xl = std::sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
    if (!(xl > 0)) return fail(nullptr, S3R_ERR_INVALID, "up is parallel to the view direction");
    for (double& c : x) c /= xl;
    double y[3] = {z[1] * x[2] - z[2] * x[1], z[2] * x[0] - z[0] * x[2], z[0] * x[1] - z[1] * x[0]};
    const float lcam = 0.01f * 2 * 5.f;
    std::memset(out, 0, sizeof(*out));
    for (int d = 0; d < 3; ++d) {
        out->eye[d] = (float)eye[d];
        out->e1[d] = (float)x[d];
        out->e2[d] = (float)y[d];
        out->n[d] = (float)z[d] * (-lcam);
        out->view_r[d] = (float)x[d];
        out->view_r[3 + d] = (float)y[d];
        out->view_r[6 + d] = (float)z[d];
    }
    const double* rows[3] = {x, y, z};
    for (int a = 0; a < 3; ++a)
        out->view_t[a] = (float)-(rows[a][0] * eye[0] + rows[a][1] * eye[1] + rows[a][2] * eye[2]);
    out->ortho = ortho ? 1 : 0;
    if (ortho) {
        out->h = (float)ortho_height;
    } else {
        out->h = (float)(2 * lcam * std::tan(0.5 * fovy_deg * M_PI / 180));
    }
    const float pixel = out->h / (float)H;
    out->w = pixel * (float)W;
    return S3R_OK;
}

int s3r_camera_from_view(const float m[16], float fovy_deg, uint32_t W, uint32_t H, s3r_camera* out)
{
    if (!m || !out || W == 0 || H == 0) return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    // m: the world -> eye transform, column-major (element (row r, column c) at m[4 c + r]): rotation R and
    // translation T.  Its inverse (a rigid motion) has rotation R^T and translation -R^T T; the eye set-up of
    // DenseFieldRenderer_cu.cu:353-372 reads the eye position -(R^T) T, the screen axes (columns of R^T,
    // normalized) and the view direction (third column of R^T) from it, in float.
    float R[3][3], T[3];
    for (int r = 0; r < 3; ++r) {
        for (int c = 0; c < 3; ++c) R[r][c] = m[4 * c + r];
        T[r] = m[12 + r];
    }
    auto normalized = [](float v[3]) {
        const float l = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        if (l > 0) {
            v[0] /= l;
            v[1] /= l;
            v[2] /= l;
        }
    };
    std::memset(out, 0, sizeof(*out));
    const float lcam = 0.01f * 2 * 5.f;
    for (int r = 0; r < 3; ++r) // (-R^T) T, summed over the columns of -R^T in order
        out->eye[r] = -R[0][r] * T[0] + -R[1][r] * T[1] + -R[2][r] * T[2];
    float x[3] = {R[0][0], R[0][1], R[0][2]}, y[3] = {R[1][0], R[1][1], R[1][2]}, z[3] = {R[2][0], R[2][1], R[2][2]};
    normalized(x);
    normalized(y);
    normalized(z);
    for (int d = 0; d < 3; ++d) {
        out->e1[d] = x[d];
        out->e2[d] = y[d];
        out->n[d] = z[d] * (-lcam);
        out->view_r[d] = R[0][d];
        out->view_r[3 + d] = R[1][d];
        out->view_r[6 + d] = R[2][d];
        out->view_t[d] = T[d];
    }
    out->h = (float)(2 * lcam * std::tan(0.5 * (double)fovy_deg * M_PI / 180));
    const float pixel = out->h / (float)H;
    out->w = pixel * (float)W;
    return S3R_OK;
}

int s3r_block_cube(uint32_t level, const uint32_t idx[3], float center[3], float* half_size)
{
    if (!idx || !center || !half_size || level > 12) return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    block_cube_f(level, idx, center, *half_size);
    return S3R_OK;
}

int s3r_block_view_rect(const s3r_view* view, const uint32_t idx[3], int32_t rect[4])
{
    if (!idx || !rect) return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    int rc = check_view(nullptr, view);
    if (rc) return rc;
    view_rect(*view, idx, rect);
    return S3R_OK;
}

int s3r_clear_viewport(s3r_ctx* ctx, uint32_t* viewport, uint32_t W, uint32_t H, uint32_t value, void* stream)
{
    if (!ctx || !viewport) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    int rc = set_device(ctx);
    if (rc) return rc;
    S3R_CUDA(ctx, launch_fill_u32(viewport, (uint64_t)W * H, value, as_stream(stream)));
    ++ctx->launches;
    return S3R_OK;
}

// pitch: the brick's row pitch in elements (0: a plain (2^depth+1)^3 grid)
static int render_block_argb_pitched(s3r_ctx* ctx, const s3r_view* view, const float* brick, uint32_t depth,
                                     uint32_t pitch, const uint32_t idx[3], const int32_t rect[4], const float* tf,
                                     uint32_t* viewport, void* stream)
{
    if (!ctx) return fail(nullptr, S3R_ERR_INVALID, "ctx is null");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (!brick || !idx || !rect || !tf || !viewport) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (depth > S3R_MAX_DEPTH) return fail(ctx, S3R_ERR_INVALID, "depth exceeds S3R_MAX_DEPTH");
    const uint32_t m = 1u << view->level;
    if (idx[0] >= m || idx[1] >= m || idx[2] >= m) return fail(ctx, S3R_ERR_INVALID, "block index outside level");
    if (rect[2] < 0 || rect[3] < 0) return fail(ctx, S3R_ERR_INVALID, "negative view rectangle");
    if ((rc = set_device(ctx))) return rc;
    RenderBlock rb{};
    block_sampling(view->level, idx, depth, rb);
    rb.pitch = pitch;
    for (int i = 0; i < 4; ++i) rb.rect[i] = rect[i];
    S3R_CUDA(ctx, launch_render_block_mode(view, nullptr, brick, nullptr, rb, tf, viewport, as_stream(stream)));
    if (rect[2] > 0 && rect[3] > 0) ++ctx->launches;
    return S3R_OK;
}

int s3r_render_block_argb(s3r_ctx* ctx, const s3r_view* view, const float* brick, uint32_t depth,
                          const uint32_t idx[3], const int32_t rect[4], const float* tf, uint32_t* viewport,
                          void* stream)
{
    return render_block_argb_pitched(ctx, view, brick, depth, 0, idx, rect, tf, viewport, stream);
}

int s3r_index_box_world(uint32_t level, const uint32_t bmin[3], const uint32_t bmax[3], double cmin[3], double cmax[3])
{
    if (!bmin || !bmax || !cmin || !cmax || level > 12) return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    // s3vs::boundingBoxOfIndexBox (src/s3vs_worker/BlockOrderUtil.hpp:29-52), float arithmetic
    const float top = 5.f;
    const float h = top / (float)(1u << level);
    for (int d = 0; d < 3; ++d) {
        if (bmax[d] <= bmin[d]) return fail(nullptr, S3R_ERR_INVALID, "empty index box");
        const float c0 = -top + h * (float)(1u + (bmin[d] << 1));
        const float c1 = -top + h * (float)(1u + ((bmax[d] - 1) << 1));
        cmin[d] = (double)c0 - (double)h;
        cmax[d] = (double)c1 + (double)h;
    }
    return S3R_OK;
}

int s3r_b2f_order(const uint32_t bmin[3], const uint32_t bmax[3], const double cmin[3], const double cmax[3],
                  const double eye[3], uint32_t* out, uint32_t capacity, uint32_t* count)
{
    if (!bmin || !bmax || !cmin || !cmax || !eye || !count || (capacity && !out))
        return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    Split sp[3];
    for (int a = 0; a < 3; ++a) {
        if (bmax[a] <= bmin[a] || !((float)cmax[a] > (float)cmin[a]))
            return fail(nullptr, S3R_ERR_INVALID, "index box or world box is empty");
        sp[a] = split_range(bmin[a], bmax[a], (float)cmin[a], (float)cmax[a], (float)eye[a]);
    }
    uint32_t n = 0;
    b2f_traverse(sp, [&](const uint32_t q[3]) {
        if (n < capacity)
            for (int a = 0; a < 3; ++a) out[3 * n + a] = q[a];
        ++n;
    });
    *count = n;
    return S3R_OK;
}

int s3r_split_index_cube(uint32_t level, uint32_t split_count, int32_t add_trailing_empty, uint32_t* boxes,
                         uint32_t capacity, uint32_t* count)
{
    if (!count || (capacity && !boxes) || split_count == 0 || level > 20)
        return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    const CubeSplit cs = cube_split(level, split_count);
    uint32_t n = 0;
    for (uint32_t z = 0; z < cs.n[2]; ++z)
        for (uint32_t y = 0; y < cs.n[1]; ++y)
            for (uint32_t x = 0; x < cs.n[0]; ++x) {
                const uint32_t q[3] = {x, y, z};
                if (n < capacity) put_box(cs, q, boxes + 6 * n);
                ++n;
            }
    if (add_trailing_empty)
        for (; n < split_count; ++n)
            if (n < capacity) std::fill(boxes + 6 * n, boxes + 6 * n + 6, 0u);
    *count = n;
    return S3R_OK;
}

int s3r_split_b2f(uint32_t level, uint32_t split_count, const double eye[3], uint32_t* boxes, uint32_t capacity,
                  uint32_t* count)
{
    if (!eye || !count || (capacity && !boxes) || split_count == 0 || level > 20)
        return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    const CubeSplit cs = cube_split(level, split_count);
    Split sp[3];
    for (int a = 0; a < 3; ++a) sp[a] = split_boundaries(cs.coord[a].data(), cs.n[a], (float)eye[a]);
    uint32_t n = 0;
    b2f_traverse(sp, [&](const uint32_t q[3]) {
        if (n < capacity) put_box(cs, q, boxes + 6 * n);
        ++n;
    });
    *count = n;
    return S3R_OK;
}

// overflow (optional): what a part's launches left in the flag beside the rectangle.
static int bound_rect(s3r_ctx* ctx, const uint32_t* viewport, uint32_t W, uint32_t H, int32_t rect[4], int32_t* overflow,
                      cudaStream_t s)
{
    S3R_CUDA(ctx, launch_bound_rect(viewport, W, H, ctx->rect_dev, ctx->rect_host, s));
    ++ctx->launches;
    S3R_CUDA(ctx, cudaStreamSynchronize(s));
    const int32_t* r = ctx->rect_host;
    if (r[2] == 0) {
        rect[0] = rect[1] = rect[2] = rect[3] = 0;
    } else {
        rect[0] = (int32_t)W - r[0];
        rect[1] = (int32_t)H - r[1];
        rect[2] = r[2] - rect[0];
        rect[3] = r[3] - rect[1];
    }
    if (overflow) *overflow = r[4];
    return S3R_OK;
}

int s3r_bound_rect(s3r_ctx* ctx, const uint32_t* viewport, uint32_t W, uint32_t H, int32_t rect[4], void* stream)
{
    if (!ctx || !viewport || !rect) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    int rc = set_device(ctx);
    if (rc) return rc;
    return bound_rect(ctx, viewport, W, H, rect, nullptr, as_stream(stream));
}

int s3r_crop(s3r_ctx* ctx, const uint32_t* image, uint32_t W, const int32_t rect[4], uint32_t* dst, void* stream)
{
    if (!ctx || !image || !rect || !dst) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (rect[0] < 0 || rect[1] < 0 || rect[2] < 0 || rect[3] < 0 || (uint32_t)(rect[0] + rect[2]) > W)
        return fail(ctx, S3R_ERR_INVALID, "crop rectangle outside the image");
    int rc = set_device(ctx);
    if (rc) return rc;
    S3R_CUDA(ctx, launch_crop(image, W, rect, dst, as_stream(stream)));
    if (rect[2] > 0 && rect[3] > 0) ++ctx->launches;
    return S3R_OK;
}

int s3r_default_light(const s3r_view* view, s3r_light* out)
{
    if (!view || !out) return fail(nullptr, S3R_ERR_INVALID, "null pointer");
    const s3r_camera& c = view->cam;
    for (int d = 0; d < 3; ++d) {
        out->pos[d] = (c.eye[d] + c.n[d]) + c.e2[d] * c.h; // DenseFieldRenderer_cu.cu:442
        out->ambient[d] = 0.f;
        out->diffuse[d] = 1.f;
        out->specular[d] = 0.1f;
    }
    return S3R_OK;
}

static int check_presentation(s3r_ctx* ctx, const s3r_presentation& pr)
{
    if (pr.mode > S3R_MODE_VALUE_ON_ISOSURFACES) return fail(ctx, S3R_ERR_INVALID, "unknown field mode");
    if (pr.level_count > S3R_MAX_LEVELS) return fail(ctx, S3R_ERR_INVALID, "more than S3R_MAX_LEVELS levels");
    if (pr.light_count > S3R_MAX_LIGHTS) return fail(ctx, S3R_ERR_INVALID, "more than S3R_MAX_LIGHTS lights");
    for (uint32_t i = 1; i < pr.level_count; ++i)
        if (!(pr.levels[i] > pr.levels[i - 1])) return fail(ctx, S3R_ERR_INVALID, "levels must ascend strictly");
    return S3R_OK;
}

static int render_block_pitched(s3r_ctx* ctx, const s3r_view* view, const s3r_presentation* pres,
                                const float* brick, const float* brick2, uint32_t depth, uint32_t pitch,
                                const uint32_t idx[3], const int32_t rect[4], const float* tf, uint32_t* viewport,
                                void* stream)
{
    if (!ctx) return fail(nullptr, S3R_ERR_INVALID, "ctx is null");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (!pres || !brick || !idx || !rect || !tf || !viewport) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if ((rc = check_presentation(ctx, *pres))) return rc;
    const bool secondary = pres->mode == S3R_MODE_VALUE_ON_ISOSURFACE || pres->mode == S3R_MODE_VALUE_ON_ISOSURFACES;
    if (secondary && !brick2) return fail(ctx, S3R_ERR_INVALID, "this mode needs the secondary field's brick");
    if (secondary && !(pres->secondary_max > pres->secondary_min))
        return fail(ctx, S3R_ERR_INVALID, "secondary field range is empty");
    if (depth > S3R_MAX_DEPTH) return fail(ctx, S3R_ERR_INVALID, "depth exceeds S3R_MAX_DEPTH");
    const uint32_t m = 1u << view->level;
    if (idx[0] >= m || idx[1] >= m || idx[2] >= m) return fail(ctx, S3R_ERR_INVALID, "block index outside level");
    if (rect[2] < 0 || rect[3] < 0) return fail(ctx, S3R_ERR_INVALID, "negative view rectangle");
    if ((rc = set_device(ctx))) return rc;
    RenderBlock rb{};
    block_sampling(view->level, idx, depth, rb);
    rb.pitch = pitch;
    for (int i = 0; i < 4; ++i) rb.rect[i] = rect[i];
    S3R_CUDA(ctx, launch_render_block_mode(view, pres, brick, brick2, rb, tf, viewport, as_stream(stream)));
    if (rect[2] > 0 && rect[3] > 0) ++ctx->launches;
    return S3R_OK;
}

int s3r_render_block(s3r_ctx* ctx, const s3r_view* view, const s3r_presentation* pres, const float* brick,
                     const float* brick2, uint32_t depth, const uint32_t idx[3], const int32_t rect[4],
                     const float* tf, uint32_t* viewport, void* stream)
{
    return render_block_pitched(ctx, view, pres, brick, brick2, depth, 0, idx, rect, tf, viewport, stream);
}

// ------------------------------------------------------------------ texture-unit path

int s3r_texture_create(s3r_ctx* ctx, uint32_t depth, s3r_texture** out)
{
    if (!ctx || !out) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (depth > S3R_MAX_DEPTH) return fail(ctx, S3R_ERR_INVALID, "depth exceeds S3R_MAX_DEPTH");
    int rc = set_device(ctx);
    if (rc) return rc;
    auto* t = new (std::nothrow) s3r_texture;
    if (!t) return fail(ctx, S3R_ERR_NOMEM, "out of host memory");
    t->ctx = ctx;
    t->depth = depth;
    t->n = (1u << depth) + 1u;
    const cudaChannelFormatDesc desc = cudaCreateChannelDesc(32, 0, 0, 0, cudaChannelFormatKindFloat);
    cudaError_t e = cudaMalloc3DArray(&t->array, &desc, make_cudaExtent(t->n, t->n, t->n), cudaArraySurfaceLoadStore);
    if (e == cudaSuccess) {
        cudaResourceDesc res;
        std::memset(&res, 0, sizeof(res));
        res.resType = cudaResourceTypeArray;
        res.res.array.array = t->array;
        cudaTextureDesc td;
        std::memset(&td, 0, sizeof(td));
        td.normalizedCoords = 0;
        td.filterMode = cudaFilterModeLinear;
        td.addressMode[0] = td.addressMode[1] = td.addressMode[2] = cudaAddressModeClamp;
        td.readMode = cudaReadModeElementType;
        e = cudaCreateTextureObject(&t->tex, &res, &td, nullptr);
        if (e == cudaSuccess) e = cudaCreateSurfaceObject(&t->surf, &res);
    }
    if (e != cudaSuccess) {
        s3r_texture_destroy(t);
        return cuda_fail(ctx, e, "field texture");
    }
    *out = t;
    return S3R_OK;
}

int s3r_texture_destroy(s3r_texture* t)
{
    if (!t) return S3R_OK;
    if (t->ctx) cudaSetDevice(t->ctx->device);
    if (t->tex) cudaDestroyTextureObject(t->tex);
    if (t->surf) cudaDestroySurfaceObject(t->surf);
    if (t->array) cudaFreeArray(t->array);
    delete t;
    return S3R_OK;
}

int s3r_texture_fill(s3r_ctx* ctx, s3r_texture* t, const float* dense, void* stream)
{
    if (!ctx || !t || !dense) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (t->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "texture belongs to another context");
    int rc = set_device(ctx);
    if (rc) return rc;
    cudaMemcpy3DParms p;
    std::memset(&p, 0, sizeof(p));
    p.srcPtr = make_cudaPitchedPtr(const_cast<float*>(dense), t->n * sizeof(float), t->n, t->n);
    p.dstArray = t->array;
    p.extent = make_cudaExtent(t->n, t->n, t->n);
    p.kind = cudaMemcpyDeviceToDevice;
    S3R_CUDA(ctx, cudaMemcpy3DAsync(&p, as_stream(stream)));
    return S3R_OK;
}

int s3r_interp_dense_texture(s3r_ctx* ctx, const uint16_t* n2i_xyz, const float* sparse, uint32_t n, s3r_texture* t,
                             void* stream)
{
    if (!ctx || !t) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (t->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "texture belongs to another context");
    int rc = set_device(ctx);
    if (rc) return rc;
    if (n > 0 && (!n2i_xyz || !sparse)) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    return interp_block(ctx, n2i_xyz, sparse, n, t->depth, nullptr, t->surf, as_stream(stream));
}

int s3r_tf_texture_create(s3r_ctx* ctx, uint32_t tf_n, s3r_tf_texture** out)
{
    if (!ctx || !out) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (tf_n < 2 || tf_n > 4096) return fail(ctx, S3R_ERR_INVALID, "tf_n must be in [2, 4096]");
    int rc = set_device(ctx);
    if (rc) return rc;
    auto* t = new (std::nothrow) s3r_tf_texture;
    if (!t) return fail(ctx, S3R_ERR_NOMEM, "out of host memory");
    t->ctx = ctx;
    t->n = tf_n;
    const cudaChannelFormatDesc desc = cudaCreateChannelDesc(32, 32, 32, 32, cudaChannelFormatKindFloat);
    cudaError_t e = cudaMallocArray(&t->array, &desc, tf_n, 1, cudaArrayTextureGather);
    if (e == cudaSuccess) {
        cudaResourceDesc res;
        std::memset(&res, 0, sizeof(res));
        res.resType = cudaResourceTypeArray;
        res.res.array.array = t->array;
        cudaTextureDesc td;
        std::memset(&td, 0, sizeof(td));
        td.normalizedCoords = 1;
        td.filterMode = cudaFilterModeLinear;
        td.addressMode[0] = cudaAddressModeClamp;
        td.readMode = cudaReadModeElementType;
        e = cudaCreateTextureObject(&t->tex, &res, &td, nullptr);
    }
    if (e != cudaSuccess) {
        s3r_tf_texture_destroy(t);
        return cuda_fail(ctx, e, "transfer-function texture");
    }
    *out = t;
    return S3R_OK;
}

int s3r_tf_texture_set(s3r_ctx* ctx, s3r_tf_texture* t, const float* tf, void* stream)
{
    if (!ctx || !t || !tf) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (t->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "texture belongs to another context");
    int rc = set_device(ctx);
    if (rc) return rc;
    const size_t row = (size_t)t->n * 4 * sizeof(float);
    S3R_CUDA(ctx, cudaMemcpy2DToArrayAsync(t->array, 0, 0, tf, row, row, 1, cudaMemcpyDeviceToDevice,
                                           as_stream(stream)));
    return S3R_OK;
}

int s3r_tf_texture_destroy(s3r_tf_texture* t)
{
    if (!t) return S3R_OK;
    if (t->ctx) cudaSetDevice(t->ctx->device);
    if (t->tex) cudaDestroyTextureObject(t->tex);
    if (t->array) cudaFreeArray(t->array);
    delete t;
    return S3R_OK;
}

int s3r_render_block_texture(s3r_ctx* ctx, const s3r_view* view, const s3r_presentation* pres,
                             const s3r_texture* field, const s3r_texture* field2, const uint32_t idx[3],
                             const int32_t rect[4], const s3r_tf_texture* tf, uint32_t* viewport, void* stream)
{
    if (!ctx) return fail(nullptr, S3R_ERR_INVALID, "ctx is null");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (!field || !idx || !rect || !tf || !viewport) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (field->ctx != ctx || tf->ctx != ctx || (field2 && field2->ctx != ctx))
        return fail(ctx, S3R_ERR_INVALID, "texture belongs to another context");
    if (tf->n != view->tf_n) return fail(ctx, S3R_ERR_INVALID, "transfer-function texture size differs from tf_n");
    s3r_presentation argb{};
    argb.mode = S3R_MODE_ARGB;
    const s3r_presentation* pr = pres ? pres : &argb;
    if ((rc = check_presentation(ctx, *pr))) return rc;
    const bool secondary = pr->mode == S3R_MODE_VALUE_ON_ISOSURFACE || pr->mode == S3R_MODE_VALUE_ON_ISOSURFACES;
    if (secondary && (!field2 || field2->depth != field->depth))
        return fail(ctx, S3R_ERR_INVALID, "this mode needs the secondary field's texture, of the same depth");
    if (secondary && !(pr->secondary_max > pr->secondary_min))
        return fail(ctx, S3R_ERR_INVALID, "secondary field range is empty");
    const uint32_t m = 1u << view->level;
    if (idx[0] >= m || idx[1] >= m || idx[2] >= m) return fail(ctx, S3R_ERR_INVALID, "block index outside level");
    if (rect[2] < 0 || rect[3] < 0) return fail(ctx, S3R_ERR_INVALID, "negative view rectangle");
    if ((rc = set_device(ctx))) return rc;
    RenderBlock rb{};
    block_sampling(view->level, idx, field->depth, rb);
    for (int i = 0; i < 4; ++i) rb.rect[i] = rect[i];
    S3R_CUDA(ctx, launch_render_block_texture(view, pr, (uint64_t)field->tex, field2 ? (uint64_t)field2->tex : 0,
                                              (uint64_t)tf->tex, rb, viewport, as_stream(stream)));
    if (rect[2] > 0 && rect[3] > 0) ++ctx->launches;
    return S3R_OK;
}

int s3r_blend_image_part_mip_host(float* dst, int32_t dw, int32_t dh, const float* src, int32_t sw, int32_t sh,
                                  int32_t ox, int32_t oy, int32_t just_copy, int32_t offx, int32_t offy)
{
    if (!dst || (!src && sw * sh > 0)) return fail(nullptr, S3R_ERR_INVALID, "null pointer");
    const int32_t dx = ox - offx, dy = oy - offy;
    if (dx < 0 || dy < 0 || dx + sw > dw || dy + sh > dh)
        return fail(nullptr, S3R_ERR_INVALID, "image part does not fit the destination");
    for (int32_t y = 0; y < sh; ++y) {
        const float* srow = src + (size_t)y * sw;
        float* drow = dst + (size_t)dw * (dy + y) + dx;
        if (just_copy) {
            std::memcpy(drow, srow, sizeof(float) * sw);
            continue;
        }
        for (int32_t i = 0; i < sw; ++i) {
            const float sv = srow[i];
            if (std::isnan(sv)) continue;
            if (std::isnan(drow[i]) || drow[i] < sv) drow[i] = sv;
        }
    }
    return S3R_OK;
}

int s3r_blend_image_part_host(uint32_t* dst, int32_t dw, int32_t dh, const uint32_t* src, int32_t sw, int32_t sh,
                              int32_t ox, int32_t oy, int32_t just_copy, int32_t offx, int32_t offy)
{
    if (!dst || (!src && sw * sh > 0)) return fail(nullptr, S3R_ERR_INVALID, "null pointer");
    const int32_t dx = ox - offx, dy = oy - offy;
    if (dx < 0 || dy < 0 || dx + sw > dw || dy + sh > dh)
        return fail(nullptr, S3R_ERR_INVALID, "image part does not fit the destination");
    for (int32_t y = 0; y < sh; ++y) {
        const uint32_t* srow = src + (size_t)y * sw;
        uint32_t* drow = dst + (size_t)dw * (dy + y) + dx;
        if (just_copy) {
            std::memcpy(drow, srow, sizeof(uint32_t) * sw);
            continue;
        }
        for (int32_t i = 0; i < sw; ++i) {
            const uint32_t s = srow[i], as = s >> 24;
            if (as == 0) continue;
            const uint32_t d = drow[i], ad = d >> 24;
            if (as == 255u || ad == 0) {
                drow[i] = s;
                continue;
            }
            const uint32_t a = as + ad * (255u - as) / 255u;
            uint32_t o = (a & 0xffu) << 24;
            for (int b = 0; b < 3; ++b) {
                const uint32_t cs = (s >> (8 * b)) & 0xffu, cd = (d >> (8 * b)) & 0xffu;
                o |= (((cs * as + cd * (a - as)) / a) & 0xffu) << (8 * b);
            }
            drow[i] = o;
        }
    }
    return S3R_OK;
}

int s3r_compose_parts(s3r_ctx* ctx, const s3r_image_part* parts, uint32_t nparts, int32_t just_copy_first,
                      uint32_t* dst, int32_t dw, int32_t dh, int32_t offx, int32_t offy, void* stream)
{
    if (!ctx || !dst || (nparts && !parts)) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    int rc = set_device(ctx);
    if (rc) return rc;
    if (nparts == 0) return S3R_OK;
    cudaStream_t s = as_stream(stream);
    if (nparts > kComposeInline) {
        if (ctx->parts_cap < nparts) {
            if (ctx->parts_dev) cudaFree(ctx->parts_dev);
            ctx->parts_dev = nullptr;
            ctx->parts_cap = 0;
            S3R_CUDA(ctx, cudaMalloc(&ctx->parts_dev, sizeof(s3r_image_part) * nparts));
            ctx->parts_cap = nparts;
        }
        S3R_CUDA(ctx, cudaMemcpyAsync(ctx->parts_dev, parts, sizeof(s3r_image_part) * nparts, cudaMemcpyHostToDevice, s));
    }
    S3R_CUDA(ctx, launch_compose(parts, nparts > kComposeInline ? ctx->parts_dev : nullptr, nparts, just_copy_first, dst,
                                 dw, dh, offx, offy, s));
    // callers may release the parts' pixels on return (and a longer list is pageable host memory copied
    // asynchronously): finish first
    S3R_CUDA(ctx, cudaStreamSynchronize(s));
    ++ctx->launches;
    return S3R_OK;
}

int s3r_make_color_transfer(const double* xs, const double* rgba, uint32_t npoints, uint32_t color_count, float* out)
{
    if (!out || color_count == 0 || (npoints && (!xs || !rgba))) return fail(nullptr, S3R_ERR_INVALID, "bad argument");
    // makeColorTransferVector (include/s3vs/ColorTransferFunction.hpp:27-69); real_type is float
    if (npoints == 0) {
        for (uint32_t i = 0; i < 4 * color_count; ++i) out[i] = 1.f;
        return S3R_OK;
    }
    if (npoints == 1) {
        for (uint32_t i = 0; i < color_count; ++i)
            for (int c = 0; c < 4; ++c) out[4 * i + c] = (float)rgba[c];
        return S3R_OK;
    }
    for (uint32_t i = 1; i < npoints; ++i)
        if (!((float)xs[i] > (float)xs[i - 1])) return fail(nullptr, S3R_ERR_INVALID, "control points not increasing");
    std::fill(out, out + 4 * color_count, 0.f);
    const float xmin = (float)xs[0], xmax = (float)xs[npoints - 1];
    float c1[4];
    for (int c = 0; c < 4; ++c) out[c] = c1[c] = (float)rgba[c];
    uint32_t i1 = 0;
    for (uint32_t ip = 1; ip < npoints; ++ip) {
        float c2[4];
        for (int c = 0; c < 4; ++c) c2[c] = (float)rgba[4 * ip + c];
        const uint32_t i2 = ip + 1 == npoints ? color_count - 1u
                                              : (uint32_t)(((float)xs[ip] - xmin) / (xmax - xmin) * (float)color_count);
        for (uint32_t i = i1 + 1; i2 > i1 && i <= i2 && i < color_count; ++i) {
            const float t = (float)(i - i1) / (float)(i2 - i1);
            for (int c = 0; c < 4; ++c) out[4 * i + c] = c1[c] * (1 - t) + c2[c] * t;
        }
        for (int c = 0; c < 4; ++c) c1[c] = c2[c];
        i1 = i2;
    }
    return S3R_OK;
}

// ------------------------------------------------------------------ plans

int s3r_frame_plan(s3r_ctx* ctx, const s3r_frame_desc* desc, s3r_plan** out)
{
    if (!ctx || !desc || !out) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    *out = nullptr;
    if (desc->level > 8) return fail(ctx, S3R_ERR_INVALID, "level out of range (max 8)");
    if (desc->nblocks == 0 || !desc->blocks || !desc->node_off || (!desc->n2i && desc->node_off[desc->nblocks]))
        return fail(ctx, S3R_ERR_INVALID, "empty or null block description");
    if (desc->brick_format > S3R_BRICK_BF16) return fail(ctx, S3R_ERR_INVALID, "unknown brick format");
    uint32_t tl = 4;
    if (desc->tile_cells) {
        if (desc->tile_cells == 8) tl = 3;
        else if (desc->tile_cells == 16) tl = 4;
        else if (desc->tile_cells == 32) tl = 5;
        else return fail(ctx, S3R_ERR_INVALID, "tile_cells must be 0, 8, 16 or 32");
    }
    int rc = set_device(ctx);
    if (rc) return rc;
    const uint32_t m = 1u << desc->level;
    auto p = new (std::nothrow) s3r_plan;
    if (!p) return fail(ctx, S3R_ERR_NOMEM, "out of host memory");
    p->ctx = ctx;
    p->desc = *desc;
    p->nblocks = desc->nblocks;
    p->level = desc->level;
    p->fmt = desc->brick_format;
    p->render_tile = desc->render_tile % kRenderTiles;
    p->blocks.assign(desc->blocks, desc->blocks + 4 * (size_t)desc->nblocks);
    p->node_off.assign(desc->node_off, desc->node_off + desc->nblocks + 1);
    p->nodes = p->node_off[desc->nblocks];
    if (p->nodes > 0xffffffffull) {
        s3r_plan_destroy(p);
        return fail(ctx, S3R_ERR_INVALID, "a plan holds fewer than 2^32 nodes");
    }
    p->n2i.assign(desc->n2i, desc->n2i + 3 * p->nodes);
    p->vertex_off.assign(desc->nblocks + 1, 0);
    p->pitch.assign(desc->nblocks, 0);
    p->vertices = 0;
    const uint32_t elem_bytes = p->fmt == S3R_BRICK_F32 ? 4u : 2u;
    p->table_host.assign((size_t)m * m * m, RenderBlock{});
    for (auto& t : p->table_host) {
        t.depth = 0xffffffffu;
        t.fmt = p->fmt;
    }
    auto bail = [&](int code) {
        s3r_plan_destroy(p);
        return code;
    };
    for (uint32_t b = 0; b < desc->nblocks; ++b) {
        const uint32_t* bl = &p->blocks[4 * b];
        if (bl[0] >= m || bl[1] >= m || bl[2] >= m)
            return bail(fail(ctx, S3R_ERR_INVALID, "block index outside the level"));
        if (bl[3] > S3R_MAX_DEPTH) return bail(fail(ctx, S3R_ERR_INVALID, "block depth exceeds S3R_MAX_DEPTH"));
        if (p->node_off[b + 1] < p->node_off[b]) return bail(fail(ctx, S3R_ERR_INVALID, "node offsets decrease"));
        if (p->node_off[b + 1] - p->node_off[b] > 0xffffffffull)
            return bail(fail(ctx, S3R_ERR_INVALID, "too many nodes in one block"));
        p->max_nodes = std::max(p->max_nodes, (uint32_t)(p->node_off[b + 1] - p->node_off[b]));
        const uint64_t e = (1ull << bl[3]) + 1;
        const uint32_t pitch = plan_brick_pitch(bl[3], elem_bytes);
        p->pitch[b] = pitch;
        p->vertex_off[b + 1] = p->vertex_off[b] + e * e * pitch;
        p->vertices += e * e * e;
        RenderBlock& t = p->table_host[bl[0] + m * (bl[1] + m * bl[2])];
        if (t.depth != 0xffffffffu) return bail(fail(ctx, S3R_ERR_INVALID, "duplicate block index"));
        block_sampling(p->level, bl, bl[3], t);
        t.brick_off = p->vertex_off[b];
        t.pitch = pitch;
        t.block = b;
        const uint32_t lim = (uint32_t)(e - 1);
        for (uint64_t i = p->node_off[b]; i < p->node_off[b + 1]; ++i)
            if (p->n2i[3 * i] > lim || p->n2i[3 * i + 1] > lim || p->n2i[3 * i + 2] > lim)
                return bail(fail(ctx, S3R_ERR_INVALID, "node index outside its block"));
    }
    p->brick_elems = p->vertex_off[desc->nblocks];
    const size_t esz = elem_bytes;
    cudaError_t e;
    if ((e = cudaMalloc(&p->bricks, std::max<uint64_t>(p->brick_elems, 1) * esz)) != cudaSuccess)
        return bail(cuda_fail(ctx, e, "cudaMalloc(bricks)"));
    if ((rc = upload(ctx, &p->node_off_dev, p->node_off))) return bail(rc);
    if ((e = cudaMalloc(&p->queue_dev, 2 * sizeof(uint32_t))) != cudaSuccess)
        return bail(cuda_fail(ctx, e, "cudaMalloc(queue)"));
    if ((e = cudaMalloc(&p->scale_offset_dev, sizeof(float2) * p->nblocks)) != cudaSuccess)
        return bail(cuda_fail(ctx, e, "cudaMalloc(scales)"));
    {
        auto round = [](size_t n) { return (n + 255) & ~(size_t)255; };
        const size_t view_off = round(sizeof(RenderBlock) * p->table_host.size()),
                     cover_off = view_off + round(sizeof(s3r_view)), list_off = cover_off + 256;
        p->stage_bytes = list_off + sizeof(uint2) * ((size_t)p->nblocks + 1);
        if ((e = cudaMalloc(&p->stage_dev, p->stage_bytes)) != cudaSuccess ||
            (e = cudaMallocHost(&p->stage_pinned, p->stage_bytes)) != cudaSuccess)
            return bail(cuda_fail(ctx, e, "cudaMalloc(view and table)"));
        auto place = [&](void* base, RenderBlock*& table, s3r_view*& view, int32_t*& cover, uint2*& list) {
            char* c = static_cast<char*>(base);
            table = reinterpret_cast<RenderBlock*>(c);
            view = reinterpret_cast<s3r_view*>(c + view_off);
            cover = reinterpret_cast<int32_t*>(c + cover_off);
            list = reinterpret_cast<uint2*>(c + list_off);
        };
        place(p->stage_dev, p->table_dev, p->view_dev, p->cover_dev, p->seg_list_dev);
        place(p->stage_pinned, p->table_pinned, p->view_pinned, p->cover_pinned, p->seg_list_pinned);
    }
    for (cudaEvent_t* ev : {&p->staged, &p->expanded, &p->seg_done[0], &p->seg_done[1]})
        if ((e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming)) != cudaSuccess)
            return bail(cuda_fail(ctx, e, "cudaEventCreate"));
    // block-major render: blocks deepest first (most samples per ray), so that the longest work items start first
    {
        std::vector<uint32_t> idx(desc->nblocks);
        for (uint32_t b = 0; b < desc->nblocks; ++b) idx[b] = b;
        std::stable_sort(idx.begin(), idx.end(),
                         [&](uint32_t a, uint32_t b) { return p->blocks[4 * a + 3] > p->blocks[4 * b + 3]; });
        p->seg_order.resize(desc->nblocks);
        for (uint32_t i = 0; i < desc->nblocks; ++i) {
            const uint32_t* bl = &p->blocks[4 * idx[i]];
            p->seg_order[i] = bl[0] + m * (bl[1] + m * bl[2]);
        }
        if ((e = cudaMalloc(&p->seg_queue, 2 * sizeof(uint32_t))) != cudaSuccess ||
            (e = cudaMemset(p->seg_queue, 0, 2 * sizeof(uint32_t))) != cudaSuccess)
            return bail(cuda_fail(ctx, e, "cudaMalloc(block-major render)"));
    }
    if ((rc = plan_bin(p, tl))) return bail(rc);
    *out = p;
    return S3R_OK;
}

static void plan_destroy_host_pipeline(s3r_plan* p);

int s3r_plan_destroy(s3r_plan* p)
{
    if (!p) return S3R_OK;
    if (p->ctx) cudaSetDevice(p->ctx->device);
    plan_destroy_host_pipeline(p);
    plan_drop_graph(p);
    plan_free_device(p);
    auto f = [](void* q) {
        if (q) cudaFree(q);
    };
    f(p->bricks);
    f(p->node_off_dev);
    f(p->queue_dev);
    f(p->scale_offset_dev);
    f(p->stage_dev);
    if (p->stage_pinned) cudaFreeHost(p->stage_pinned);
    f(p->dtf_part);
    f(p->seg_queue);
    plan_free_segments(p);
    for (cudaEvent_t ev : {p->staged, p->expanded, p->seg_done[0], p->seg_done[1]})
        if (ev) cudaEventDestroy(ev);
    delete p;
    return S3R_OK;
}

int s3r_plan_info_get(const s3r_plan* p, s3r_plan_info* out)
{
    if (!p || !out) return fail(nullptr, S3R_ERR_INVALID, "null pointer");
    out->nodes = p->nodes;
    out->vertices = p->vertices;
    out->brick_bytes = p->brick_elems * (p->fmt == S3R_BRICK_F32 ? 4 : 2);
    out->tiles = p->tiles;
    out->tile_entries = p->entries;
    out->tile_cells = 1u << p->tile_log2;
    out->render_tile = p->render_tile;
    out->brick_format = p->fmt;
    out->nblocks = p->nblocks;
    return S3R_OK;
}

int s3r_plan_tile_cells(const s3r_plan* p, uint32_t depth, uint32_t* cells)
{
    if (!p || !cells) return fail(nullptr, S3R_ERR_INVALID, "null pointer");
    if (depth > S3R_MAX_DEPTH) return fail(nullptr, S3R_ERR_INVALID, "depth exceeds S3R_MAX_DEPTH");
    *cells = 1u << p->tile_by_depth[depth];
    return S3R_OK;
}

int s3r_plan_bricks(const s3r_plan* p, void** bricks, const uint64_t** vertex_off)
{
    if (!p || !bricks || !vertex_off) return fail(nullptr, S3R_ERR_INVALID, "null pointer");
    *bricks = p->bricks;
    *vertex_off = p->vertex_off.data();
    return S3R_OK;
}

int s3r_plan_brick_pitches(const s3r_plan* p, const uint32_t** pitch)
{
    if (!p || !pitch) return fail(nullptr, S3R_ERR_INVALID, "null pointer");
    *pitch = p->pitch.data();
    return S3R_OK;
}

int s3r_plan_brick_scales(const s3r_plan* p, const float** scale_offset)
{
    if (!p || !scale_offset) return fail(nullptr, S3R_ERR_INVALID, "null pointer");
    *scale_offset = p->fmt == S3R_BRICK_F32 ? nullptr : reinterpret_cast<const float*>(p->scale_offset_dev);
    return S3R_OK;
}

int s3r_frame_interp(s3r_ctx* ctx, s3r_plan* plan, const float* sparse, void* stream)
{
    if (!ctx || !plan || (!sparse && plan->nodes)) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "plan belongs to another context");
    int rc = set_device(ctx);
    if (rc) return rc;
    uint32_t k = 0;
    rc = plan_launch_interp(plan, sparse, as_stream(stream), &k);
    ctx->launches += k;
    return rc;
}

int s3r_frame_render(s3r_ctx* ctx, s3r_plan* plan, const s3r_view* view, const float* tf, float* rgba, uint32_t* argb,
                     unsigned long long* samples, void* stream)
{
    if (!ctx || !plan || !tf) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "plan belongs to another context");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (view->level != plan->level) return fail(ctx, S3R_ERR_INVALID, "view level differs from the plan level");
    if ((rc = set_device(ctx))) return rc;
    cudaStream_t s = as_stream(stream);
    if ((rc = plan_stage_view(plan, view, s, true))) return rc;
    uint32_t k = 0;
    const bool seg = plan_block_major(plan, s);
    rc = plan_in_turn(plan, seg, 0, s, [&] { return plan_launch_render(plan, tf, rgba, argb, samples, seg, s, &k); });
    ctx->launches += k;
    return rc;
}

int s3r_frame_render_mode(s3r_ctx* ctx, s3r_plan* plan, const s3r_view* view, const s3r_presentation* pres,
                          const float* tf, const void* bricks2, float* rgba, uint32_t* argb, void* stream)
{
    if (!ctx || !plan || !tf || !pres) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "plan belongs to another context");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (view->level != plan->level) return fail(ctx, S3R_ERR_INVALID, "view level differs from the plan level");
    if (pres->mode > S3R_MODE_VALUE_ON_ISOSURFACES) return fail(ctx, S3R_ERR_INVALID, "unknown field mode");
    if (pres->level_count > S3R_MAX_LEVELS || pres->light_count > S3R_MAX_LIGHTS)
        return fail(ctx, S3R_ERR_INVALID, "too many levels or lights");
    if ((pres->mode == S3R_MODE_VALUE_ON_ISOSURFACE || pres->mode == S3R_MODE_VALUE_ON_ISOSURFACES) && !bricks2)
        return fail(ctx, S3R_ERR_INVALID, "the value-on-isosurface modes need the secondary bricks");
    if (plan->fmt != S3R_BRICK_F32) return fail(ctx, S3R_ERR_UNSUPPORTED, "field modes need F32 bricks");
    if ((rc = set_device(ctx))) return rc;
    cudaStream_t s = as_stream(stream);
    if ((rc = plan_stage_view(plan, view, s, false))) return rc;
    FrameArgs fa{};
    fa.view = plan->view_dev;
    fa.table = plan->table_dev;
    fa.bricks = plan->bricks;
    fa.tf = tf;
    fa.rgba = rgba;
    fa.argb = argb;
    fa.cover = plan->cover_dev;
    S3R_CUDA(ctx, launch_frame_render_mode(fa, *pres, static_cast<const float*>(bricks2), view->W, view->H, view->tf_n,
                                           view->filter, s));
    ++ctx->launches;
    return S3R_OK;
}

static int plan_launch_frame(s3r_plan* plan, int slot, const s3r_view* view, const float* sparse, const float* tf,
                             float* rgba, uint32_t* argb, unsigned long long* samples, cudaStream_t s);

int s3r_frame_run(s3r_ctx* ctx, s3r_plan* plan, const s3r_view* view, const float* sparse, const float* tf,
                  float* rgba, uint32_t* argb, unsigned long long* samples, void* stream)
{
    if (!ctx || !plan || !tf || (!sparse && plan->nodes)) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "plan belongs to another context");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (view->level != plan->level) return fail(ctx, S3R_ERR_INVALID, "view level differs from the plan level");
    if ((rc = set_device(ctx))) return rc;
    cudaStream_t s = as_stream(stream);
    if ((rc = plan_stage_view(plan, view, s, true))) return rc;
    return plan_launch_frame(plan, 0, view, sparse, tf, rgba, argb, samples, s);
}

// The frame as a CUDA graph in cache slot `slot`, captured again when its arguments change; into a caller's capture its
// kernels go one by one (a graph cannot be instantiated there).
static int plan_launch_frame(s3r_plan* plan, int slot, const s3r_view* view, const float* sparse, const float* tf,
                      float* rgba, uint32_t* argb, unsigned long long* samples, cudaStream_t s)
{
    s3r_ctx* ctx = plan->ctx;
    FrameGraph& G = plan->graphs[slot];
    const void* key[5] = {sparse, tf, rgba, argb, samples};
    const bool seg = plan_block_major(plan, s);
    const uint32_t dims[5] = {view->W, view->H, view->tf_n, view->filter, seg ? (plan->seg_lanes ? 2u : 1u) : 0u};
    const int data = slot == 2 ? 1 : 0; // the host pipeline's second slot has its own bricks
    if (capturing(s)) {
        uint32_t k = 0;
        int rc = plan_launch_interp(plan, sparse, s, &k, data);
        if (!rc) rc = plan_launch_render(plan, tf, rgba, argb, samples, seg, s, &k, data);
        ctx->launches += k;
        return rc;
    }
    const bool same = G.exec && std::memcmp(key, G.key, sizeof(key)) == 0 && std::memcmp(dims, G.dims, sizeof(dims)) == 0;
    if (!same) {
        if (G.exec) cudaGraphExecDestroy(G.exec);
        G = FrameGraph{};
        cudaStream_t cs = ctx->capture;
        S3R_CUDA(ctx, cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
        uint32_t k = 0;
        int r1 = plan_launch_interp(plan, sparse, cs, &k, data);
        int r3 = r1 ? r1 : plan_launch_render(plan, tf, rgba, argb, samples, seg, cs, &k, data);
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamEndCapture(cs, &graph);
        if (r3) {
            if (graph) cudaGraphDestroy(graph);
            return r3;
        }
        if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaStreamEndCapture");
        e = cudaGraphInstantiate(&G.exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            G.exec = nullptr;
            return cuda_fail(ctx, e, "cudaGraphInstantiate");
        }
        std::memcpy(G.key, key, sizeof(key));
        std::memcpy(G.dims, dims, sizeof(dims));
        G.kernels = k;
    }
    if (int rc = plan_in_turn(plan, seg, data, s, [&]() -> int {
            S3R_CUDA(ctx, cudaGraphLaunch(G.exec, s));
            return S3R_OK;
        }))
        return rc;
    ctx->launches += G.kernels;
    return S3R_OK;
}

// Releases the host-buffer pipeline's device buffers (after its copies have finished).
static void plan_free_host_slots(s3r_plan* p)
{
    if (p->hs_h2d) cudaStreamSynchronize(p->hs_h2d);
    if (p->hs_d2h) cudaStreamSynchronize(p->hs_d2h);
    for (int b = 0; b < 2; ++b)
        if (p->hs_comp[b]) cudaStreamSynchronize(p->hs_comp[b]);
    for (int b = 0; b < 2; ++b) {
        if (p->hs_sparse[b]) cudaFree(p->hs_sparse[b]);
        if (p->hs_argb[b]) cudaFree(p->hs_argb[b]);
        if (p->hs_tf[b]) cudaFree(p->hs_tf[b]);
        p->hs_sparse[b] = nullptr;
        p->hs_argb[b] = nullptr;
        p->hs_tf[b] = nullptr;
    }
    p->hs_pixels = 0;
    p->hs_tf_n = 0;
}

static void plan_destroy_host_pipeline(s3r_plan* p)
{
    plan_free_host_slots(p);
    for (int b = 0; b < 2; ++b) {
        for (cudaEvent_t* ev : {&p->hs_copied[b], &p->hs_rendered[b], &p->hs_read[b]}) {
            if (*ev) cudaEventDestroy(*ev);
            *ev = nullptr;
        }
    }
    if (p->hs_entry) cudaEventDestroy(p->hs_entry);
    p->hs_entry = nullptr;
    for (int b = 0; b < 2; ++b) {
        if (p->hs_comp[b]) cudaStreamDestroy(p->hs_comp[b]);
        p->hs_comp[b] = nullptr;
    }
    if (p->hs_h2d) cudaStreamDestroy(p->hs_h2d);
    if (p->hs_d2h) cudaStreamDestroy(p->hs_d2h);
    p->hs_h2d = p->hs_d2h = nullptr;
    if (p->bricks_1) cudaFree(p->bricks_1);
    if (p->scale_offset_1) cudaFree(p->scale_offset_1);
    p->bricks_1 = nullptr;
    p->scale_offset_1 = nullptr;
}

// The GPU work of one s3r_frame_run_host call on slot b: the copies and the frame, with the events that
// order them against the neighbouring frames.
static int frame_host_submit(s3r_ctx* ctx, s3r_plan* plan, const s3r_view* view, const float* sparse_host,
                             const float* tf, uint32_t* argb_host, cudaStream_t s, int b)
{
    int rc;
    cudaStream_t cb = plan->hs_comp[b];
    const uint64_t pixels = (uint64_t)view->W * view->H;
    // the caller's transfer function is copied on the caller's own stream into slot b's table, once the frame
    // two back (the table's last reader) has finished: work the caller queues on `stream` after this call may
    // then change or free tf
    S3R_CUDA(ctx, cudaStreamWaitEvent(s, plan->hs_rendered[b], 0));
    S3R_CUDA(ctx, cudaMemcpyAsync(plan->hs_tf[b], tf, (size_t)view->tf_n * 4 * sizeof(float), cudaMemcpyDeviceToDevice,
                                  s));
    S3R_CUDA(ctx, cudaEventRecord(plan->hs_entry, s)); // what the caller queued before comes first
    // H2D into slot b once the frame two back no longer reads it
    S3R_CUDA(ctx, cudaStreamWaitEvent(plan->hs_h2d, plan->hs_rendered[b], 0));
    if (plan->nodes)
        S3R_CUDA(ctx, cudaMemcpyAsync(plan->hs_sparse[b], sparse_host, plan->nodes * sizeof(float),
                                      cudaMemcpyHostToDevice, plan->hs_h2d));
    S3R_CUDA(ctx, cudaEventRecord(plan->hs_copied[b], plan->hs_h2d));
    // the frame on slot b's stream -- so that it overlaps the other slot's frame on the GPU -- once its
    // input has landed and the image two frames back has been read out
    S3R_CUDA(ctx, cudaStreamWaitEvent(cb, plan->hs_entry, 0));
    S3R_CUDA(ctx, cudaStreamWaitEvent(cb, plan->hs_copied[b], 0));
    S3R_CUDA(ctx, cudaStreamWaitEvent(cb, plan->hs_read[b], 0));
    if (!plan->have_view || plan->staged_tile != (int)plan->render_tile ||
        std::memcmp(&plan->last_view, view, sizeof(s3r_view)) != 0) {
        // the render table both slots read changes: let the frames in flight finish first
        for (int q = 0; q < 2; ++q) S3R_CUDA(ctx, cudaStreamSynchronize(plan->hs_comp[q]));
    }
    if ((rc = plan_stage_view(plan, view, cb, true))) return rc;
    // the table upload, and the expansion of the work items after it, may have been queued on the other slot's stream
    S3R_CUDA(ctx, cudaStreamWaitEvent(cb, plan->seg_now ? plan->expanded : plan->staged, 0));
    if ((rc = plan_launch_frame(plan, 1 + b, view, plan->hs_sparse[b], plan->hs_tf[b], nullptr, plan->hs_argb[b],
                                nullptr, cb)))
        return rc;
    S3R_CUDA(ctx, cudaEventRecord(plan->hs_rendered[b], cb));
    // D2H of the image while the next frame runs
    S3R_CUDA(ctx, cudaStreamWaitEvent(plan->hs_d2h, plan->hs_rendered[b], 0));
    S3R_CUDA(ctx, cudaMemcpyAsync(argb_host, plan->hs_argb[b], pixels * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                  plan->hs_d2h));
    S3R_CUDA(ctx, cudaEventRecord(plan->hs_read[b], plan->hs_d2h));
    return S3R_OK;
}

int s3r_frame_run_host(s3r_ctx* ctx, s3r_plan* plan, const s3r_view* view, const float* sparse_host, const float* tf,
                       uint32_t* argb_host, void* stream)
{
    if (!ctx || !plan || !tf || !argb_host || (!sparse_host && plan->nodes))
        return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "plan belongs to another context");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (view->level != plan->level) return fail(ctx, S3R_ERR_INVALID, "view level differs from the plan level");
    if ((rc = set_device(ctx))) return rc;
    cudaError_t e;
    if (!plan->hs_h2d) {
        if ((e = cudaStreamCreateWithFlags(&plan->hs_h2d, cudaStreamNonBlocking)) != cudaSuccess ||
            (e = cudaStreamCreateWithFlags(&plan->hs_d2h, cudaStreamNonBlocking)) != cudaSuccess)
            return cuda_fail(ctx, e, "cudaStreamCreate(host frames)");
        for (int b = 0; b < 2; ++b) {
            if ((e = cudaStreamCreateWithFlags(&plan->hs_comp[b], cudaStreamNonBlocking)) != cudaSuccess)
                return cuda_fail(ctx, e, "cudaStreamCreate(host frames)");
            for (cudaEvent_t* ev : {&plan->hs_copied[b], &plan->hs_rendered[b], &plan->hs_read[b]})
                if ((e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming)) != cudaSuccess)
                    return cuda_fail(ctx, e, "cudaEventCreate(host frames)");
        }
        if ((e = cudaEventCreateWithFlags(&plan->hs_entry, cudaEventDisableTiming)) != cudaSuccess)
            return cuda_fail(ctx, e, "cudaEventCreate(host frames)");
    }
    if (!plan->bricks_1) {
        const size_t esz = plan->fmt == S3R_BRICK_F32 ? 4 : 2;
        if ((e = cudaMalloc(&plan->bricks_1, std::max<uint64_t>(plan->brick_elems, 1) * esz)) != cudaSuccess ||
            (e = cudaMalloc(&plan->scale_offset_1, sizeof(float2) * std::max<uint32_t>(plan->nblocks, 1))) != cudaSuccess)
            return cuda_fail(ctx, e, "cudaMalloc(second frame slot)");
    }
    const uint64_t pixels = (uint64_t)view->W * view->H;
    if (pixels != plan->hs_pixels || view->tf_n != plan->hs_tf_n || !plan->hs_sparse[0]) {
        plan_free_host_slots(plan);
        for (int b = 0; b < 2; ++b) {
            if ((e = cudaMalloc(&plan->hs_sparse[b], std::max<uint64_t>(plan->nodes, 1) * sizeof(float))) != cudaSuccess ||
                (e = cudaMalloc(&plan->hs_argb[b], pixels * sizeof(uint32_t))) != cudaSuccess ||
                (e = cudaMalloc(&plan->hs_tf[b], (size_t)view->tf_n * 4 * sizeof(float))) != cudaSuccess) {
                plan_free_host_slots(plan);
                return cuda_fail(ctx, e, "cudaMalloc(host frames)");
            }
        }
        plan->hs_pixels = pixels;
        plan->hs_tf_n = view->tf_n;
    }
    const int b = (int)(plan->hs_frames & 1);
    if ((rc = frame_host_submit(ctx, plan, view, sparse_host, tf, argb_host, as_stream(stream), b))) {
        // a step failed part way: let everything already queued finish, so that the next call starts from
        // a pipeline whose events all stand for completed work
        cudaStreamSynchronize(plan->hs_h2d);
        for (int q = 0; q < 2; ++q) cudaStreamSynchronize(plan->hs_comp[q]);
        cudaStreamSynchronize(plan->hs_d2h);
        return rc;
    }
    ++plan->hs_frames;
    // on return this frame's input buffer is free and the previous frame's image is in host memory; the GPU
    // meanwhile renders the previous frame and then this one
    S3R_CUDA(ctx, cudaEventSynchronize(plan->hs_copied[b]));
    if (plan->hs_frames > 1) S3R_CUDA(ctx, cudaEventSynchronize(plan->hs_read[b ^ 1]));
    return S3R_OK;
}

int s3r_frame_host_sync(s3r_ctx* ctx, s3r_plan* plan)
{
    if (!ctx || !plan) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (!plan->hs_d2h) return S3R_OK;
    int rc = set_device(ctx);
    if (rc) return rc;
    S3R_CUDA(ctx, cudaStreamSynchronize(plan->hs_h2d));
    for (int b = 0; b < 2; ++b) S3R_CUDA(ctx, cudaStreamSynchronize(plan->hs_comp[b]));
    S3R_CUDA(ctx, cudaStreamSynchronize(plan->hs_d2h));
    return S3R_OK;
}

int s3r_plan_autotune(s3r_ctx* ctx, s3r_plan* plan, const s3r_view* view, const float* sparse, const float* tf,
                      uint32_t reps, void* stream)
{
    if (!ctx || !plan || !tf || (!sparse && plan->nodes)) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "plan belongs to another context");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (view->level != plan->level) return fail(ctx, S3R_ERR_INVALID, "view level differs from the plan level");
    if ((rc = set_device(ctx))) return rc;
    if (reps == 0) reps = 3;
    cudaStream_t s = as_stream(stream);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    float* img = nullptr;
    auto cleanup = [&](int code) {
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (img) cudaFree(img);
        return code;
    };
    cudaError_t e;
    if ((e = cudaEventCreate(&e0)) != cudaSuccess || (e = cudaEventCreate(&e1)) != cudaSuccess ||
        (e = cudaMalloc(&img, sizeof(float) * 4 * (size_t)view->W * view->H)) != cudaSuccess)
        return cleanup(cuda_fail(ctx, e, "autotune set-up"));
    auto timed = [&](auto&& body, float& ms) -> int {
        uint32_t k = 0;
        int r = body(&k); // warm-up
        if (r) return r;
        if ((e = cudaEventRecord(e0, s)) != cudaSuccess) return cuda_fail(ctx, e, "cudaEventRecord");
        for (uint32_t i = 0; i < reps; ++i)
            if ((r = body(&k))) return r;
        if ((e = cudaEventRecord(e1, s)) != cudaSuccess) return cuda_fail(ctx, e, "cudaEventRecord");
        if ((e = cudaEventSynchronize(e1)) != cudaSuccess) return cuda_fail(ctx, e, "cudaEventSynchronize");
        cudaEventElapsedTime(&ms, e0, e1);
        ctx->launches += k;
        return S3R_OK;
    };
    uint32_t best_tl = plan->tile_log2;
    float best = 3.4e38f;
    for (uint32_t tl = 3; tl <= 5; ++tl) {
        if ((rc = plan_bin(plan, tl))) return cleanup(rc);
        float ms = 0;
        rc = timed([&](uint32_t* k) { return plan_launch_interp(plan, sparse, s, k); }, ms);
        if (rc) return cleanup(rc);
        if (ms < best) {
            best = ms;
            best_tl = tl;
        }
    }
    // then per block depth (deepest first): a smaller tile for that depth's blocks alone, kept when faster
    // (never a larger one: the largest tile sets every CTA's shared memory)
    uint8_t by_depth[S3R_MAX_DEPTH + 1];
    for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d) by_depth[d] = (uint8_t)std::min(best_tl, d);
    bool present[S3R_MAX_DEPTH + 1] = {};
    for (uint32_t b = 0; b < plan->nblocks; ++b) present[plan->blocks[4 * b + 3]] = true;
    for (int d = S3R_MAX_DEPTH; d >= 4; --d) {
        if (!present[d] || by_depth[d] <= 3) continue;
        const uint8_t keep = by_depth[d];
        by_depth[d] = (uint8_t)(keep - 1);
        if ((rc = plan_bin(plan, best_tl, by_depth))) return cleanup(rc);
        float ms = 0;
        rc = timed([&](uint32_t* k) { return plan_launch_interp(plan, sparse, s, k); }, ms);
        if (rc) return cleanup(rc);
        if (ms < best) best = ms;
        else by_depth[d] = keep;
    }
    if ((rc = plan_bin(plan, best_tl, by_depth))) return cleanup(rc);
    uint32_t k = 0;
    if ((rc = plan_launch_interp(plan, sparse, s, &k))) return cleanup(rc);
    ctx->launches += k;
    uint32_t best_shape = plan->render_tile;
    best = 3.4e38f;
    for (uint32_t shape = 0; shape < (uint32_t)kRenderTiles; ++shape) {
        // several lanes per ray only where rays composite every block (alpha_stop >= 1)
        if (shape >= (uint32_t)kRenderShapes && shape < (uint32_t)kRenderWalkTiles && view->alpha_stop < 1.f) continue;
        plan->render_tile = shape;
        if ((rc = plan_stage_view(plan, view, s, true)) != S3R_OK) {
            if (shape < (uint32_t)kRenderWalkTiles) return cleanup(rc);
            // no room for the block-major buffers, or a level they do not cover: keep to the others
            ctx->err.clear();
            set_thread_error("");
            continue;
        }
        float ms = 0;
        const bool seg = plan_block_major(plan, s);
        rc = plan_in_turn(plan, seg, 0, s, [&] {
            return timed([&](uint32_t* kk) { return plan_launch_render(plan, tf, img, nullptr, nullptr, seg, s, kk); }, ms);
        });
        if (rc) return cleanup(rc);
        if (ms < best) {
            best = ms;
            best_shape = shape;
        }
    }
    plan->render_tile = best_shape;
    plan_drop_graph(plan);
    if (best_shape >= (uint32_t)kRenderShapes && best_shape < (uint32_t)kRenderWalkTiles) {
        // several lanes per ray won: release the block-major buffers
        cudaStreamSynchronize(s);
        plan_free_segments(plan);
    }
    return cleanup(S3R_OK);
}

int s3r_render_argb_backward(s3r_ctx* ctx, s3r_plan* plan, const s3r_view* view, const float* tf, const float* rgba,
                             const float* dl_drgba, float* dtf, float* ddense, void* stream)
{
    if (!ctx || !plan || !tf || !rgba || !dl_drgba || !dtf || !ddense)
        return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->fmt != S3R_BRICK_F32) return fail(ctx, S3R_ERR_UNSUPPORTED, "the adjoint needs FP32 bricks");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (view->filter != S3R_FILTER_EXACT)
        return fail(ctx, S3R_ERR_UNSUPPORTED, "the adjoint needs S3R_FILTER_EXACT (texture weights are piecewise constant)");
    if (view->level != plan->level) return fail(ctx, S3R_ERR_INVALID, "view level differs from the plan level");
    if ((rc = set_device(ctx))) return rc;
    cudaStream_t s = as_stream(stream);
    if ((rc = plan_stage_view(plan, view, s, false))) return rc;
    FrameArgs fa{};
    fa.view = plan->view_dev;
    fa.table = plan->table_dev;
    fa.bricks = plan->bricks;
    fa.tf = tf;
    fa.fwd_rgba = rgba;
    fa.dl_drgba = dl_drgba;
    fa.dtf = dtf;
    fa.ddense = ddense;
    const size_t nparts = (size_t)kDtfParts * 4 * view->tf_n;
    if (plan->dtf_part_floats < nparts) {
        // allocation: synchronizes the device once, on the first adjoint call (or a larger table)
        if (plan->dtf_part) cudaFree(plan->dtf_part);
        plan->dtf_part = nullptr;
        plan->dtf_part_floats = 0;
        cudaError_t e = cudaMalloc(&plan->dtf_part, nparts * sizeof(float));
        if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaMalloc(transfer-function gradient copies)");
        plan->dtf_part_floats = nparts;
    }
    fa.dtf_part = plan->dtf_part;
    S3R_CUDA(ctx, cudaMemsetAsync(plan->dtf_part, 0, nparts * sizeof(float), s));
    S3R_CUDA(ctx, launch_frame_backward(fa, view->W, view->H, view->tf_n, s));
    S3R_CUDA(ctx, launch_dtf_reduce(plan->dtf_part, dtf, 4 * view->tf_n, s));
    ctx->launches += 2;
    return S3R_OK;
}

} // extern "C"

// ------------------------------------------------------------------ worker loop

namespace {

// A part's blocks are marched by one launch per chunk (part_blocks_kernel) where a pixel's list of results stays
// short: index boxes of up to kPartSpan blocks along their three axes together (a level of 16^3 blocks: 48), since a
// ray passes at most that many.  Larger boxes, single blocks, and a part in which some pixel's list overflowed (rays
// along the faces of blocks meet more) go block by block.
constexpr uint32_t kPartSpan = 64;
// Blocks interpolated for one launch and the bytes of their dense fields: enough to fill the GPU several times.
constexpr uint32_t kPartChunkBlocks = 256;
constexpr uint64_t kPartChunkBytes = 512ull << 20;
constexpr uint64_t kPartTextureBytes = 1ull << 30;
// The lists of a strip of the part's pixels.
constexpr uint64_t kPartListBytes = 256ull << 20;

bool part_secondary(const s3r_presentation* pres)
{
    return pres && (pres->mode == S3R_MODE_VALUE_ON_ISOSURFACE || pres->mode == S3R_MODE_VALUE_ON_ISOSURFACES);
}

bool part_at_once(const uint32_t bmin[3], const uint32_t bmax[3], size_t blocks)
{
    uint64_t span = 0;
    for (int a = 0; a < 3; ++a) span += bmax[a] > bmin[a] ? bmax[a] - bmin[a] : 0;
    return blocks > 1 && span <= kPartSpan;
}

// `bytes` of the context's table buffer: where to write on the host, and where part_upload puts it on the device.
int part_table(s3r_ctx* ctx, size_t bytes, cudaStream_t s, char** host, char** dev)
{
    bytes = (bytes + 255) & ~(size_t)255;
    if (ctx->part_used + bytes > ctx->part_cap) {
        // what was staged before has to be on the device, and used, before its memory is used again
        S3R_CUDA(ctx, cudaStreamSynchronize(s));
        ctx->part_used = 0;
        if (bytes > ctx->part_cap) {
            if (ctx->part_host) cudaFreeHost(ctx->part_host);
            if (ctx->part_dev) cudaFree(ctx->part_dev);
            ctx->part_host = ctx->part_dev = nullptr;
            ctx->part_cap = 0;
            const size_t cap = std::max<size_t>(2 * bytes, 1 << 20);
            S3R_CUDA(ctx, cudaMallocHost(&ctx->part_host, cap));
            S3R_CUDA(ctx, cudaMalloc(&ctx->part_dev, cap));
            ctx->part_cap = cap;
        }
    }
    *host = ctx->part_host + ctx->part_used;
    *dev = ctx->part_dev + ctx->part_used;
    ctx->part_used += bytes;
    return S3R_OK;
}

// One chunk of a part: the blocks `refs` (back to front, rectangles not empty) blended onto the viewport.
int part_blend(s3r_ctx* ctx, const s3r_view* view, const s3r_presentation* pres, std::vector<PartRef>& refs,
               uint32_t span, const float* tf, unsigned long long tf_tex, bool texture, uint32_t* viewport, cudaStream_t s)
{
    if (refs.empty()) return S3R_OK;
    const uint32_t n = (uint32_t)refs.size();
    int32_t x0 = INT32_MAX, y0 = INT32_MAX, x1 = INT32_MIN, y1 = INT32_MIN;
    for (uint32_t i = 0; i < n; ++i) {
        const int32_t* r = refs[i].rb.rect;
        x0 = std::min(x0, r[0]);
        y0 = std::min(y0, r[1]);
        x1 = std::max(x1, r[0] + r[2]);
        y1 = std::max(y1, r[1] + r[3]);
        refs[i].order = i;
    }
    PartArgs a{};
    a.nblocks = n;
    a.cap = std::min(n, span + 1);
    a.tf = tf;
    a.tf_tex = tf_tex;
    a.x0 = x0;
    a.w = x1 - x0;
    a.overflow = ctx->rect_dev + 4;
    const uint64_t per_pixel = sizeof(uint32_t) + a.cap * (sizeof(float4) + sizeof(uint16_t));
    const int32_t rows = (int32_t)std::max<uint64_t>(
        1, std::min<uint64_t>((uint64_t)(y1 - y0), kPartListBytes / (per_pixel * (uint64_t)a.w)));
    const size_t lists = (size_t)rows * a.w * per_pixel;
    if (ctx->part_lists_cap < lists) {
        if (ctx->part_lists) cudaFree(ctx->part_lists);
        ctx->part_lists = nullptr;
        ctx->part_lists_cap = 0;
        S3R_CUDA(ctx, cudaMalloc(&ctx->part_lists, lists));
        ctx->part_lists_cap = lists;
    }
    const size_t npix = (size_t)rows * a.w;
    a.result = reinterpret_cast<float4*>(ctx->part_lists);
    a.count = reinterpret_cast<uint32_t*>(a.result + a.cap * npix);
    a.order = reinterpret_cast<uint16_t*>(a.count + npix);
    const uint32_t strips = (uint32_t)((y1 - y0 + rows - 1) / rows);
    char *host, *dev;
    const size_t refs_bytes = n * sizeof(PartRef), first_bytes = (n + 1) * sizeof(uint32_t);
    if (int rc = part_table(ctx, refs_bytes + strips * first_bytes, s, &host, &dev)) return rc;
    // the deepest blocks' rays take the most samples: their CTAs start first
    PartRef* sorted = reinterpret_cast<PartRef*>(host);
    uint32_t put = 0;
    for (int d = S3R_MAX_DEPTH; d >= 0; --d)
        for (uint32_t i = 0; i < n; ++i)
            if (refs[i].rb.depth == (uint32_t)d) sorted[put++] = refs[i];
    uint32_t tw, th;
    part_tile(pres ? pres->mode : S3R_MODE_ARGB, texture, tw, th);
    for (uint32_t k = 0; k < strips; ++k) {
        uint32_t* first = reinterpret_cast<uint32_t*>(host + refs_bytes + k * first_bytes);
        const int32_t s0 = y0 + (int32_t)k * rows, s1 = std::min(s0 + rows, y1);
        uint64_t at = 0;
        for (uint32_t i = 0; i < n; ++i) {
            const int32_t* r = sorted[i].rb.rect;
            const int32_t h = std::min(r[1] + r[3], s1) - std::max(r[1], s0);
            first[i] = (uint32_t)at;
            if (h > 0) at += (uint64_t)(((uint32_t)r[2] + tw - 1) / tw) * (((uint32_t)h + th - 1) / th);
        }
        if (at > 0x7fffffffull) return fail(ctx, S3R_ERR_INVALID, "the part's rectangles are too large");
        first[n] = (uint32_t)at;
    }
    S3R_CUDA(ctx, cudaMemcpyAsync(dev, host, refs_bytes + strips * first_bytes, cudaMemcpyHostToDevice, s));
    a.refs = reinterpret_cast<const PartRef*>(dev);
    for (uint32_t k = 0; k < strips; ++k) {
        a.first = reinterpret_cast<const uint32_t*>(dev + refs_bytes + k * first_bytes);
        a.y0 = y0 + (int32_t)k * rows;
        a.h = std::min(rows, y1 - a.y0);
        const uint32_t ctas = reinterpret_cast<const uint32_t*>(host + refs_bytes + k * first_bytes)[n];
        S3R_CUDA(ctx, launch_part(view, pres, a, ctas, texture, viewport, s));
        ctx->launches += 2;
    }
    return S3R_OK;
}

// Field textures for `need[d]` blocks of each depth (per field), kept by the context for the next chunk and call.
int part_textures(s3r_ctx* ctx, const uint32_t need[S3R_MAX_DEPTH + 1], int fields, cudaStream_t s)
{
    auto bytes_of = [](uint32_t d) { return grid_vertices(d) * sizeof(float); };
    uint64_t more = 0;
    for (int f = 0; f < fields; ++f)
        for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d)
            if (need[d] > ctx->worker_tex[f][d].size()) more += (need[d] - ctx->worker_tex[f][d].size()) * bytes_of(d);
    if (more && ctx->worker_tex_bytes + more > kPartTextureBytes) {
        S3R_CUDA(ctx, cudaStreamSynchronize(s));
        for (auto& per_field : ctx->worker_tex)
            for (auto& per_depth : per_field) {
                for (s3r_texture* t : per_depth) s3r_texture_destroy(t);
                per_depth.clear();
            }
        ctx->worker_tex_bytes = 0;
    }
    for (int f = 0; f < fields; ++f)
        for (uint32_t d = 0; d <= S3R_MAX_DEPTH; ++d)
            while (ctx->worker_tex[f][d].size() < need[d]) {
                s3r_texture* t = nullptr;
                if (int rc = s3r_texture_create(ctx, d, &t)) return rc;
                ctx->worker_tex[f][d].push_back(t);
                ctx->worker_tex_bytes += bytes_of(d);
            }
    return S3R_OK;
}

// After a part's launches failed with `rc`: whether there was no room for what they need at once.  The part's memory is
// given back then, for the block-by-block loop, which needs one block's.
bool part_no_room(s3r_ctx* ctx, int rc, cudaStream_t s)
{
    cudaStreamSynchronize(s); // the staged tables may still be read
    if (rc != S3R_ERR_CUDA || ctx->last_cuda != cudaErrorMemoryAllocation) return false;
    for (auto& per_field : ctx->worker_tex)
        for (auto& per_depth : per_field) {
            for (s3r_texture* t : per_depth) s3r_texture_destroy(t);
            per_depth.clear();
        }
    ctx->worker_tex_bytes = 0;
    auto give = [](auto*& p, size_t& cap) {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    };
    for (int f = 0; f < 2; ++f) give(ctx->worker_dense[f], ctx->worker_cap[f]);
    give(ctx->part_lists, ctx->part_lists_cap);
    give(ctx->grid, ctx->grid_cap);
    give(ctx->grid_bits, ctx->grid_bits_cap);
    (void)cudaGetLastError(); // the failure leaves no error behind for later launches
    ctx->err.clear();
    set_thread_error("");
    return true;
}

// A block of the part: its index in the caller's list and its view rectangle.
struct PartBlock {
    uint32_t b;
    int32_t rect[4];
};

// s3r_render_scene_part's blocks, back to front, in chunks: each chunk's blocks interpolated by one set of launches
// (into the context's field textures, or into dense grids), then blended.
int part_from_nodes(s3r_ctx* ctx, const s3r_view* view, const s3r_presentation* pres, const s3r_worker_blocks* wb,
                    const std::vector<PartBlock>& blocks, uint32_t span, const float* tf, uint32_t* viewport,
                    cudaStream_t s)
{
    const bool tex = view->filter == S3R_FILTER_TEXTURE, secondary = part_secondary(pres);
    const int fields = secondary ? 2 : 1;
    size_t at = 0;
    while (at < blocks.size()) {
        uint64_t vertices = 0;
        size_t end = at;
        while (end < blocks.size() && end - at < kPartChunkBlocks) {
            const uint64_t more = grid_vertices(wb->blocks[4 * blocks[end].b + 3]);
            if (end > at && (vertices + more) * sizeof(float) > kPartChunkBytes) break;
            vertices += more;
            ++end;
        }
        const uint32_t n = (uint32_t)(end - at);
        uint32_t need[S3R_MAX_DEPTH + 1] = {};
        for (size_t i = at; i < end; ++i) ++need[wb->blocks[4 * blocks[i].b + 3]];
        if (tex) {
            if (int rc = part_textures(ctx, need, fields, s)) return rc;
        } else {
            for (int f = 0; f < fields; ++f)
                if (ctx->worker_cap[f] < vertices) {
                    if (ctx->worker_dense[f]) cudaFree(ctx->worker_dense[f]);
                    ctx->worker_dense[f] = nullptr;
                    ctx->worker_cap[f] = 0;
                    S3R_CUDA(ctx, cudaMalloc(&ctx->worker_dense[f], vertices * sizeof(float)));
                    ctx->worker_cap[f] = vertices;
                }
        }
        char *host, *dev;
        const uint32_t ng = n * (uint32_t)fields;
        if (int rc = part_table(ctx, ng * sizeof(GridBlock) + (ng + 1) * sizeof(uint32_t), s, &host, &dev)) return rc;
        GridBlock* gb = reinterpret_cast<GridBlock*>(host);
        uint32_t* tile_off = reinterpret_cast<uint32_t*>(host + ng * sizeof(GridBlock));
        std::vector<PartRef> refs(n);
        uint64_t vals = 0, words = 0;
        uint32_t tiles = 0, scattered = 0, depth_max = 0, g = 0;
        for (int f = 0; f < fields; ++f) {
            uint32_t used[S3R_MAX_DEPTH + 1] = {};
            uint64_t dense = 0;
            for (uint32_t i = 0; i < n; ++i, ++g) {
                const PartBlock& pb = blocks[at + i];
                const uint32_t* bl = wb->blocks + 4 * pb.b;
                const uint64_t o = wb->node_off[pb.b], nn = wb->node_off[pb.b + 1] - o;
                GridBlock q = grid_block(wb->n2i + 3 * o, (f ? wb->sparse2 : wb->sparse) + o, (uint32_t)nn, bl[3]);
                if (!q.direct) {
                    q.val_off = vals;
                    q.bit_off = words;
                    vals += grid_vertices(bl[3]);
                    words += grid_mask_words(bl[3]);
                    scattered = std::max(scattered, (uint32_t)nn);
                }
                unsigned long long src;
                if (tex) {
                    s3r_texture* t = ctx->worker_tex[f][bl[3]][used[bl[3]]++];
                    q.surface = t->surf;
                    src = t->tex;
                } else {
                    q.out = ctx->worker_dense[f] + dense;
                    src = (unsigned long long)(uintptr_t)q.out;
                    dense += grid_vertices(bl[3]);
                }
                gb[g] = q;
                tile_off[g] = tiles;
                tiles += grid_tiles(bl[3]);
                depth_max = std::max(depth_max, bl[3]);
                PartRef& r = refs[i];
                if (f == 0) {
                    r = PartRef{};
                    block_sampling(view->level, bl, bl[3], r.rb);
                    std::memcpy(r.rb.rect, pb.rect, sizeof(pb.rect));
                    r.src1 = src;
                } else {
                    r.src2 = src;
                }
            }
        }
        tile_off[ng] = tiles;
        if (words)
            if (int rc = ensure_grid(ctx, vals, words)) return rc;
        S3R_CUDA(ctx, cudaMemcpyAsync(dev, host, ng * sizeof(GridBlock) + (ng + 1) * sizeof(uint32_t),
                                      cudaMemcpyHostToDevice, s));
        GridArgs a{};
        a.table = reinterpret_cast<const GridBlock*>(dev);
        a.tile_off = reinterpret_cast<const uint32_t*>(dev + ng * sizeof(GridBlock));
        a.nblocks = ng;
        a.tiles = tiles;
        a.depth_max = depth_max;
        a.vals = ctx->grid;
        a.bits = ctx->grid_bits;
        uint32_t launches = 0;
        S3R_CUDA(ctx, launch_interp_grid(a, tex, scattered, words, s, &launches));
        ctx->launches += launches;
        if (int rc = part_blend(ctx, view, pres, refs, span, tf, tex ? ctx->worker_tf->tex : 0, tex, viewport, s))
            return rc;
        at = end;
    }
    return S3R_OK;
}

// The checks that the per-block calls make before they launch.
int check_part(s3r_ctx* ctx, const s3r_view* view, const s3r_presentation* pres, const uint32_t* blocks,
               const std::vector<PartBlock>& list)
{
    if (pres) {
        if (int rc = check_presentation(ctx, *pres)) return rc;
        if (part_secondary(pres) && !(pres->secondary_max > pres->secondary_min))
            return fail(ctx, S3R_ERR_INVALID, "secondary field range is empty");
    }
    const uint32_t m = 1u << view->level;
    for (const PartBlock& p : list) {
        const uint32_t* bl = blocks + 4 * p.b;
        if (bl[0] >= m || bl[1] >= m || bl[2] >= m) return fail(ctx, S3R_ERR_INVALID, "block index outside level");
    }
    return S3R_OK;
}

} // namespace

extern "C" {

int s3r_render_scene_part(s3r_ctx* ctx, const s3r_view* view, const s3r_presentation* pres,
                          const s3r_worker_blocks* wb, const uint32_t box_min[3], const uint32_t box_max[3],
                          const float* tf, uint32_t* viewport, int32_t rect[4], void* stream)
{
    if (!ctx) return fail(nullptr, S3R_ERR_INVALID, "ctx is null");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (!wb || !box_min || !box_max || !tf || !viewport || !rect) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (wb->nblocks && (!wb->blocks || !wb->node_off || !wb->n2i || !wb->sparse))
        return fail(ctx, S3R_ERR_INVALID, "null block data");
    const bool secondary = part_secondary(pres);
    if (secondary && !wb->sparse2) return fail(ctx, S3R_ERR_INVALID, "this mode needs the secondary field");
    if ((rc = set_device(ctx))) return rc;
    const cudaStream_t s = as_stream(stream);
    const uint32_t clear = pres && pres->mode == S3R_MODE_MAX_INTENSITY ? 0x7fc00000u : 0u;
    if ((rc = s3r_clear_viewport(ctx, viewport, view->W, view->H, clear, stream))) return rc;
    // the box's blocks back to front (MacroBlock over the box, the view's eye)
    double cmin[3], cmax[3];
    if ((rc = s3r_index_box_world(view->level, box_min, box_max, cmin, cmax))) return rc;
    Split sp[3];
    for (int a = 0; a < 3; ++a)
        sp[a] = split_range(box_min[a], box_max[a], (float)cmin[a], (float)cmax[a], view->cam.eye[a]);
    // the texture filter samples through the texture unit, as the reference's renderer does: the transfer
    // function goes into the context's colour texture first
    const bool tex = view->filter == S3R_FILTER_TEXTURE;
    if (tex) {
        if (ctx->worker_tf && ctx->worker_tf->n != view->tf_n) {
            s3r_tf_texture_destroy(ctx->worker_tf);
            ctx->worker_tf = nullptr;
        }
        if (!ctx->worker_tf && (rc = s3r_tf_texture_create(ctx, view->tf_n, &ctx->worker_tf))) return rc;
        if ((rc = s3r_tf_texture_set(ctx, ctx->worker_tf, tf, stream))) return rc;
    }
    // the set's blocks by their place in the box
    const uint64_t ex = box_max[0] > box_min[0] ? box_max[0] - box_min[0] : 0,
                   ey = box_max[1] > box_min[1] ? box_max[1] - box_min[1] : 0,
                   ez = box_max[2] > box_min[2] ? box_max[2] - box_min[2] : 0;
    const bool flat = ex * ey * ez <= (1u << 18);
    std::vector<int32_t> place(flat ? ex * ey * ez : 0, -1);
    std::unordered_map<uint64_t, uint32_t> where;
    if (!flat) where.reserve(wb->nblocks * 2 + 1);
    for (uint32_t b = 0; b < wb->nblocks; ++b) {
        const uint32_t* bl = wb->blocks + 4 * b;
        if (!flat) {
            where[(uint64_t)bl[0] | ((uint64_t)bl[1] << 21) | ((uint64_t)bl[2] << 42)] = b;
        } else {
            const uint64_t x = (uint64_t)bl[0] - box_min[0], y = (uint64_t)bl[1] - box_min[1],
                           z = (uint64_t)bl[2] - box_min[2];
            if (x < ex && y < ey && z < ez) place[x + ex * (y + ey * z)] = (int32_t)b;
        }
    }
    // the blocks that can show, back to front
    std::vector<PartBlock> list;
    b2f_traverse(sp, [&](const uint32_t q[3]) {
        if (rc) return;
        PartBlock p;
        if (flat) {
            const int32_t b = place[(q[0] - box_min[0]) + ex * ((q[1] - box_min[1]) + ey * (uint64_t)(q[2] - box_min[2]))];
            if (b < 0) return; // not a block of this set
            p.b = (uint32_t)b;
        } else {
            auto it = where.find((uint64_t)q[0] | ((uint64_t)q[1] << 21) | ((uint64_t)q[2] << 42));
            if (it == where.end()) return;
            p.b = it->second;
        }
        if (wb->blocks[4 * p.b + 3] > S3R_MAX_DEPTH) {
            rc = fail(ctx, S3R_ERR_INVALID, "depth exceeds S3R_MAX_DEPTH");
            return;
        }
        view_rect(*view, wb->blocks + 4 * p.b, p.rect);
        if (p.rect[2] > 0 && p.rect[3] > 0) list.push_back(p);
    });
    if (rc) return rc;
    if (!list.empty() && (rc = check_part(ctx, view, pres, wb->blocks, list))) return rc;
    if (part_at_once(box_min, box_max, list.size())) {
        uint32_t span = 0;
        for (int a = 0; a < 3; ++a) span += box_max[a] - box_min[a];
        ctx->part_used = 0; // every call ends with its stream drained
        rc = part_from_nodes(ctx, view, pres, wb, list, span, tf, viewport, s);
        if (rc && !part_no_room(ctx, rc, s)) return rc;
        int32_t overflow = 0;
        if (!rc && ((rc = bound_rect(ctx, viewport, view->W, view->H, rect, &overflow, s)) || !overflow)) return rc;
        if ((rc = s3r_clear_viewport(ctx, viewport, view->W, view->H, clear, stream))) return rc;
    }
    for (const PartBlock& p : list) {
        const uint32_t* bl = wb->blocks + 4 * p.b;
        const uint32_t depth = bl[3];
        const uint64_t o = wb->node_off[p.b], n = wb->node_off[p.b + 1] - o;
        if (tex) {
            // DeviceField::makeField: the block's dense field interpolated into the depth's field texture
            uint32_t need[S3R_MAX_DEPTH + 1] = {};
            need[depth] = 1;
            if ((rc = part_textures(ctx, need, secondary ? 2 : 1, s))) return rc;
            for (int f = 0; f < (secondary ? 2 : 1); ++f)
                if ((rc = s3r_interp_dense_texture(ctx, wb->n2i + 3 * o, (f ? wb->sparse2 : wb->sparse) + o,
                                                   (uint32_t)n, ctx->worker_tex[f][depth][0], stream)))
                    return rc;
            if ((rc = s3r_render_block_texture(ctx, view, pres, ctx->worker_tex[0][depth][0],
                                               secondary ? ctx->worker_tex[1][depth][0] : nullptr, bl, p.rect,
                                               ctx->worker_tf, viewport, stream)))
                return rc;
            continue;
        }
        const uint64_t count = grid_vertices(depth);
        for (int f = 0; f < (secondary ? 2 : 1); ++f)
            if (ctx->worker_cap[f] < count) {
                if (ctx->worker_dense[f]) cudaFree(ctx->worker_dense[f]);
                ctx->worker_dense[f] = nullptr;
                ctx->worker_cap[f] = 0;
                S3R_CUDA(ctx, cudaMalloc(&ctx->worker_dense[f], count * sizeof(float)));
                ctx->worker_cap[f] = count;
            }
        // DeviceField::makeField: the block's dense field from its nodes
        for (int f = 0; f < (secondary ? 2 : 1); ++f)
            if ((rc = s3r_interp_dense(ctx, wb->n2i + 3 * o, (f ? wb->sparse2 : wb->sparse) + o, (uint32_t)n, depth,
                                       ctx->worker_dense[f], stream)))
                return rc;
        rc = pres ? s3r_render_block(ctx, view, pres, ctx->worker_dense[0], secondary ? ctx->worker_dense[1] : nullptr,
                                     depth, bl, p.rect, tf, viewport, stream)
                  : s3r_render_block_argb(ctx, view, ctx->worker_dense[0], depth, bl, p.rect, tf, viewport, stream);
        if (rc) return rc;
    }
    return s3r_bound_rect(ctx, viewport, view->W, view->H, rect, stream);
}

int s3r_render_scene_part_bricks(s3r_ctx* ctx, s3r_plan* plan, const s3r_view* view, const s3r_presentation* pres,
                                 const void* bricks2, const uint32_t box_min[3], const uint32_t box_max[3],
                                 const float* tf, uint32_t* viewport, int32_t rect[4], void* stream)
{
    if (!ctx || !plan) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->ctx != ctx) return fail(ctx, S3R_ERR_INVALID, "plan belongs to another context");
    int rc = check_view(ctx, view);
    if (rc) return rc;
    if (view->level != plan->level) return fail(ctx, S3R_ERR_INVALID, "view level differs from the plan level");
    if (!box_min || !box_max || !tf || !viewport || !rect) return fail(ctx, S3R_ERR_INVALID, "null pointer");
    if (plan->fmt != S3R_BRICK_F32) return fail(ctx, S3R_ERR_UNSUPPORTED, "the per-block renderer reads F32 bricks");
    const bool secondary = part_secondary(pres);
    if (secondary && !bricks2) return fail(ctx, S3R_ERR_INVALID, "this mode needs the secondary bricks");
    if ((rc = set_device(ctx))) return rc;
    const cudaStream_t s = as_stream(stream);
    const uint32_t clear = pres && pres->mode == S3R_MODE_MAX_INTENSITY ? 0x7fc00000u : 0u;
    if ((rc = s3r_clear_viewport(ctx, viewport, view->W, view->H, clear, stream))) return rc;
    double cmin[3], cmax[3];
    if ((rc = s3r_index_box_world(view->level, box_min, box_max, cmin, cmax))) return rc;
    Split sp[3];
    for (int a = 0; a < 3; ++a)
        sp[a] = split_range(box_min[a], box_max[a], (float)cmin[a], (float)cmax[a], view->cam.eye[a]);
    const uint32_t m = 1u << plan->level;
    std::vector<PartBlock> list;
    b2f_traverse(sp, [&](const uint32_t q[3]) {
        if (q[0] >= m || q[1] >= m || q[2] >= m) return;
        const RenderBlock& t = plan->table_host[q[0] + m * (q[1] + (size_t)m * q[2])];
        if (t.depth == 0xffffffffu) return;
        PartBlock p;
        p.b = t.block;
        view_rect(*view, &plan->blocks[4 * p.b], p.rect);
        if (p.rect[2] > 0 && p.rect[3] > 0) list.push_back(p);
    });
    if (!list.empty() && (rc = check_part(ctx, view, pres, plan->blocks.data(), list))) return rc;
    const float* bricks = static_cast<const float*>(plan->bricks);
    const float* b2 = static_cast<const float*>(bricks2);
    if (part_at_once(box_min, box_max, list.size())) {
        uint32_t span = 0;
        for (int a = 0; a < 3; ++a) span += box_max[a] - box_min[a];
        std::vector<PartRef> refs(list.size());
        for (size_t i = 0; i < list.size(); ++i) {
            const uint32_t* bl = &plan->blocks[4 * list[i].b];
            PartRef& r = refs[i];
            r.rb = plan->table_host[bl[0] + m * (bl[1] + (size_t)m * bl[2])];
            std::memcpy(r.rb.rect, list[i].rect, sizeof(r.rb.rect));
            const uint64_t o = plan->vertex_off[list[i].b];
            r.src1 = (unsigned long long)(uintptr_t)(bricks + o);
            r.src2 = secondary ? (unsigned long long)(uintptr_t)(b2 + o) : 0;
        }
        ctx->part_used = 0; // every call ends with its stream drained
        rc = part_blend(ctx, view, pres, refs, span, tf, 0, false, viewport, s);
        if (rc && !part_no_room(ctx, rc, s)) return rc;
        int32_t overflow = 0;
        if (!rc && ((rc = bound_rect(ctx, viewport, view->W, view->H, rect, &overflow, s)) || !overflow)) return rc;
        if ((rc = s3r_clear_viewport(ctx, viewport, view->W, view->H, clear, stream))) return rc;
    }
    for (const PartBlock& p : list) {
        const uint32_t* bl = &plan->blocks[4 * p.b];
        const uint64_t o = plan->vertex_off[p.b];
        const uint32_t pitch = plan->pitch[p.b];
        rc = pres ? render_block_pitched(ctx, view, pres, bricks + o, secondary ? b2 + o : nullptr, bl[3], pitch, bl,
                                         p.rect, tf, viewport, stream)
                  : render_block_argb_pitched(ctx, view, bricks + o, bl[3], pitch, bl, p.rect, tf, viewport, stream);
        if (rc) return rc;
    }
    return s3r_bound_rect(ctx, viewport, view->W, view->H, rect, stream);
}

} // extern "C"
