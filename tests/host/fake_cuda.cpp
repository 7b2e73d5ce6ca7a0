// A stand-in for the CUDA runtime and the kernels, linked with revise_gb300/csrc/host.cpp alone, so that what the host
// side queues -- streams, events, graphs, allocations -- is checked on a machine without a GPU.  Device memory is host
// memory; copies, fills and the expansion of work items are carried out when they are queued (or their graph is
// launched), other kernels only state what they read and write.  Every access is checked against the accesses before
// it: touching memory that was given back, running over an allocation's end, or meeting a write that nothing orders
// before it (vector clocks of the streams, joined by events and host waits) adds a line to fake_trouble().
#include "s3r_internal.h"

#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <sstream>
#include <string>
#include <vector>

using namespace s3r;

namespace {

using Clock = std::map<const void*, uint64_t>; // stream -> operations of it that are known to be over

struct Access {
    const void* p;
    uint64_t bytes;
    bool write;
};
struct Op {
    std::string name;
    std::function<std::vector<Access>()> accesses; // worked out when the operation runs
    std::function<void()> body;
};
struct Past {
    const void* stream;
    uint64_t time;
    std::string name;
    uint64_t lo, hi;
    bool write;
};
struct Memory {
    uint64_t bytes = 0;
    bool host = false, freed = false;
    std::vector<Past> past;
};
struct Graph {
    std::vector<Op> ops;
};
struct Stream {
    Clock clock;
    bool capturing = false;
    Graph graph;
};

std::map<const char*, Memory> g_memory; // by start address
std::map<const void*, Stream> g_streams;
std::map<const void*, Clock> g_events;
std::map<std::string, int> g_calls;
std::set<std::string> g_trouble;
Clock g_host;
uint64_t g_limit = ~0ull, g_used = 0, g_peak = 0, g_handle = 0x1000;
cudaError_t g_last = cudaSuccess;

void trouble(const std::string& what) { g_trouble.insert(what); }
cudaError_t result(cudaError_t e)
{
    if (e != cudaSuccess) g_last = e;
    return e;
}
void join(Clock& a, const Clock& b)
{
    for (auto& [k, v] : b) a[k] = std::max(a[k], v);
}
void join_all(Clock& a)
{
    for (auto& [h, s] : g_streams) join(a, s.clock);
}
Memory* memory_of(const void* p, uint64_t& offset)
{
    auto it = g_memory.upper_bound(static_cast<const char*>(p));
    if (it == g_memory.begin()) return nullptr;
    --it;
    offset = (uint64_t)(static_cast<const char*>(p) - it->first);
    return offset < std::max<uint64_t>(it->second.bytes, 1) ? &it->second : nullptr;
}

// One access of an operation on `stream` at `time`, everything in `before` being over.
bool check(const Access& a, const std::string& name, const void* stream, uint64_t time, const Clock& before)
{
    if (!a.p || a.bytes == 0) return true;
    uint64_t off = 0;
    Memory* m = memory_of(a.p, off);
    if (!m) return true; // the caller's own memory
    if (m->freed) {
        trouble(name + " uses freed memory");
        return false;
    }
    if (off + a.bytes > m->bytes) {
        trouble(name + " runs over the end of an allocation");
        return false;
    }
    for (const Past& b : m->past) {
        if (!(a.write || b.write) || b.hi <= off || off + a.bytes <= b.lo) continue;
        auto it = before.find(b.stream);
        if ((it == before.end() ? 0 : it->second) < b.time && b.stream != stream) trouble(name + " races with " + b.name);
    }
    if (a.write) // later accesses are ordered against this write, what it covers is ordered before it
        for (size_t i = 0; i < m->past.size();) {
            if (m->past[i].lo >= off && m->past[i].hi <= off + a.bytes) m->past.erase(m->past.begin() + (long)i);
            else ++i;
        }
    m->past.push_back({stream, time, name, off, off + a.bytes, a.write});
    return true;
}

void run(const Op& op, const void* stream)
{
    Stream& s = g_streams[stream];
    join(s.clock, g_host);
    const uint64_t time = ++s.clock[stream];
    bool ok = true;
    for (const Access& a : op.accesses()) ok &= check(a, op.name, stream, time, s.clock);
    ++g_calls[op.name];
    if (ok && op.body) op.body();
}

cudaError_t submit(cudaStream_t stream, Op op)
{
    Stream& s = g_streams[stream];
    if (s.capturing) s.graph.ops.push_back(std::move(op));
    else run(op, stream);
    return cudaSuccess;
}
cudaError_t kernel(cudaStream_t s, const char* name, std::vector<Access> a, std::function<void()> body = nullptr)
{
    // a failed call before it shows up here, as cudaGetLastError after a launch returns it
    const cudaError_t last = g_last;
    g_last = cudaSuccess;
    submit(s, Op{name, [a] { return a; }, std::move(body)});
    return last;
}

cudaError_t allocate(void** p, uint64_t bytes, bool host)
{
    if (!host && g_used + bytes > g_limit) return result(cudaErrorMemoryAllocation);
    Memory m;
    m.bytes = bytes;
    m.host = host;
    char* q = static_cast<char*>(std::calloc(std::max<uint64_t>(bytes, 256), 1));
    g_memory[q] = m;
    *p = q;
    if (!host) g_peak = std::max(g_peak, g_used += bytes);
    return cudaSuccess;
}
cudaError_t release(void* p)
{
    auto it = g_memory.find(static_cast<const char*>(p));
    if (!p || it == g_memory.end()) return cudaSuccess;
    if (it->second.freed) trouble("memory freed twice");
    it->second.freed = true; // the address is never handed out again
    if (!it->second.host) g_used -= it->second.bytes;
    return cudaSuccess;
}
template <class H> H handle() { return reinterpret_cast<H>(g_handle += 16); }

} // namespace

// ------------------------------------------------------------------ for the tests
extern "C" {
const char* fake_trouble()
{
    static std::string all;
    all.clear();
    for (auto& t : g_trouble) all += t + "\n";
    return all.c_str();
}
int fake_calls(const char* name) { return g_calls.count(name) ? g_calls[name] : 0; }
void fake_reset()
{
    g_calls.clear();
    g_trouble.clear();
    g_peak = g_used;
    g_limit = ~0ull;
    g_last = cudaSuccess;
}
void fake_limit(uint64_t more) { g_limit = more == ~0ull ? more : g_used + more; }
uint64_t fake_used() { return g_used; }
uint64_t fake_peak() { return g_peak; }

// ------------------------------------------------------------------ the runtime
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaGetLastError()
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorName(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "cudaErrorMemoryAllocation" : "error"; }
const char* cudaGetErrorString(cudaError_t e) { return cudaGetErrorName(e); }

cudaError_t cudaMalloc(void** p, size_t n)
{
    ++g_calls["cudaMalloc"];
    return allocate(p, n, false);
}
cudaError_t cudaMallocHost(void** p, size_t n) { return allocate(p, n, true); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return allocate(p, n, true); }
cudaError_t cudaFree(void* p)
{
    ++g_calls["cudaFree"];
    // (waits for the device, but a caller that leaves it to that is told)
    auto it = g_memory.find(static_cast<const char*>(p));
    if (p && it != g_memory.end())
        for (const Past& b : it->second.past) {
            auto over = g_host.find(b.stream);
            if (over == g_host.end() || over->second < b.time) trouble("memory freed that " + b.name + " may still use");
        }
    join_all(g_host);
    return release(p);
}
cudaError_t cudaFreeHost(void* p) { return release(p); }
cudaError_t cudaDeviceSynchronize()
{
    ++g_calls["cudaDeviceSynchronize"];
    join_all(g_host);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
    *s = handle<cudaStream_t>();
    g_streams[*s];
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id)
{
    *id = reinterpret_cast<unsigned long long>(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    ++g_calls["cudaStreamSynchronize"];
    if (g_streams[s].capturing) {
        trouble("cudaStreamSynchronize in a capture");
        return result(cudaErrorStreamCaptureUnsupported);
    }
    join(g_host, g_streams[s].clock);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    *e = handle<cudaEvent_t>();
    g_events[*e];
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    if (g_streams[s].capturing) return cudaSuccess;
    join(g_streams[s].clock, g_host);
    g_events[e] = g_streams[s].clock;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
    if (g_streams[s].capturing) {
        trouble("a captured stream waits for an event from outside the capture");
        return result(cudaErrorStreamCaptureIsolation);
    }
    join(g_streams[s].clock, g_events[e]);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    ++g_calls["cudaEventSynchronize"];
    join(g_host, g_events[e]);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
    static float t = 1.f;
    *ms = t += 1.f;
    return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode)
{
    g_streams[s].capturing = true;
    g_streams[s].graph = Graph{};
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g)
{
    g_streams[s].capturing = false;
    *g = reinterpret_cast<cudaGraph_t>(new Graph(g_streams[s].graph));
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st)
{
    *st = g_streams[s].capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long)
{
    *x = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph*>(g)));
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g)
{
    delete reinterpret_cast<Graph*>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x)
{
    delete reinterpret_cast<Graph*>(x);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s)
{
    for (const Op& op : reinterpret_cast<Graph*>(x)->ops) submit(s, op);
    return cudaSuccess;
}

cudaError_t cudaMemcpyAsync(void* d, const void* q, size_t n, cudaMemcpyKind, cudaStream_t s)
{
    return submit(s, Op{"copy", [=] { return std::vector<Access>{{q, n, false}, {d, n, true}}; },
                        [=] { std::memcpy(d, q, n); }});
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s)
{
    return submit(s, Op{"fill", [=] { return std::vector<Access>{{d, n, true}}; }, [=] { std::memset(d, v, n); }});
}
cudaError_t cudaMemcpy(void* d, const void* q, size_t n, cudaMemcpyKind k)
{
    cudaMemcpyAsync(d, q, n, k, nullptr);
    join(g_host, g_streams[nullptr].clock);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n)
{
    cudaMemsetAsync(d, v, n, nullptr);
    join(g_host, g_streams[nullptr].clock);
    return cudaSuccess;
}

cudaChannelFormatDesc cudaCreateChannelDesc(int x, int y, int z, int w, cudaChannelFormatKind f) { return {x, y, z, w, f}; }
cudaError_t cudaMalloc3DArray(cudaArray_t* a, const cudaChannelFormatDesc*, cudaExtent e, unsigned)
{
    return allocate(reinterpret_cast<void**>(a), e.width * std::max<size_t>(e.height, 1) * std::max<size_t>(e.depth, 1) * 4, false);
}
cudaError_t cudaMallocArray(cudaArray_t* a, const cudaChannelFormatDesc*, size_t w, size_t h, unsigned)
{
    return allocate(reinterpret_cast<void**>(a), w * std::max<size_t>(h, 1) * 16, false);
}
cudaError_t cudaFreeArray(cudaArray_t a)
{
    join_all(g_host);
    return release(a);
}
cudaError_t cudaCreateTextureObject(cudaTextureObject_t* t, const cudaResourceDesc* r, const cudaTextureDesc*,
                                    const cudaResourceViewDesc*)
{
    *t = reinterpret_cast<cudaTextureObject_t>(r->res.array.array);
    return cudaSuccess;
}
cudaError_t cudaDestroyTextureObject(cudaTextureObject_t) { return cudaSuccess; }
cudaError_t cudaCreateSurfaceObject(cudaSurfaceObject_t* t, const cudaResourceDesc* r)
{
    *t = reinterpret_cast<cudaSurfaceObject_t>(r->res.array.array);
    return cudaSuccess;
}
cudaError_t cudaDestroySurfaceObject(cudaSurfaceObject_t) { return cudaSuccess; }
cudaError_t cudaMemcpy2DToArrayAsync(cudaArray_t a, size_t, size_t, const void*, size_t, size_t w, size_t h, cudaMemcpyKind,
                                     cudaStream_t s)
{
    return submit(s, Op{"copy", [=] { return std::vector<Access>{{a, w * h, true}}; }, nullptr});
}
cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms* q, cudaStream_t s)
{
    const Access a{q->dstArray, 4, true};
    return submit(s, Op{"copy", [=] { return std::vector<Access>{a}; }, nullptr});
}
} // extern "C"

// ------------------------------------------------------------------ the kernels
namespace s3r {

uint32_t interp_plan_ctas_per_sm(uint32_t, uint32_t) { return 8; }
cudaError_t launch_fill_u32(uint32_t* p, uint64_t n, uint32_t v, cudaStream_t s)
{
    return kernel(s, "clear", {{p, 4 * n, true}}, [=] { std::fill(p, p + n, v); });
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
cudaError_t launch_interp_grid(const GridArgs& a, bool surface, uint32_t, uint64_t words, cudaStream_t s, uint32_t* launches)
{
    if (launches) ++*launches;
    std::vector<Access> acc{{a.bits, 4 * words, true}};
    for (uint32_t i = 0; i < a.nblocks; ++i) {
        const GridBlock& b = a.table ? a.table[i] : a.one; // (staged already: copies are carried out as they are queued)
        if (a.table) acc.push_back({a.table + i, sizeof(GridBlock), false});
        acc.push_back({surface ? reinterpret_cast<void*>(b.surface) : b.out, 4 * grid_vertices(b.depth), true});
        if (!b.direct) acc.push_back({a.vals + b.val_off, 4 * grid_vertices(b.depth), true});
    }
    return kernel(s, "interp_grid", acc);
}
cudaError_t launch_interp_plan(const TileArgs& a, uint32_t, uint32_t, uint32_t, cudaStream_t s)
{
    return kernel(s, "interp", {{a.sparse, 4, false}, {a.out, 4, true}, {a.queue, 4, true}});
}
cudaError_t launch_block_prep(const PrepArgs& a, uint32_t, uint32_t, uint32_t, cudaStream_t s)
{
    return kernel(s, "prep", {{a.sparse, 4, false}});
}
cudaError_t launch_render_block_texture(const s3r_view*, const s3r_presentation*, uint64_t field, uint64_t, uint64_t tf,
                                        const RenderBlock&, uint32_t* viewport, cudaStream_t s)
{
    return kernel(s, "render_block",
                  {{reinterpret_cast<void*>(field), 4, false}, {reinterpret_cast<void*>(tf), 4, false}, {viewport, 4, true}});
}
cudaError_t launch_render_block_mode(const s3r_view*, const s3r_presentation*, const float* brick, const float*,
                                     const RenderBlock&, const float*, uint32_t* viewport, cudaStream_t s)
{
    return kernel(s, "render_block", {{brick, 4, false}, {viewport, 4, true}});
}
void part_tile(uint32_t, bool, uint32_t& w, uint32_t& h)
{
    w = 8;
    h = 16;
}
cudaError_t launch_part(const s3r_view*, const s3r_presentation*, const PartArgs& a, uint32_t, bool, uint32_t* viewport,
                        cudaStream_t s)
{
    const uint64_t n = (uint64_t)a.w * a.h;
    return kernel(s, "part", {{a.refs, a.nblocks * sizeof(PartRef), false},
                              {a.first, (a.nblocks + 1) * 4, false},
                              {a.count, 4 * n, true},
                              {a.result, 16 * n * a.cap, true},
                              {a.order, 2 * n * a.cap, true},
                              {viewport, 4, true}});
}
// What the frame kernels read of the staged view when they run.
static std::vector<Access> frame_reads(const FrameArgs& a)
{
    const s3r_view& v = *a.view;
    const uint64_t n = (uint64_t)v.W * v.H;
    return {{a.view, sizeof(s3r_view), false},
            {a.table, sizeof(RenderBlock) << (3 * v.level), false},
            {a.cover, 16, false},
            {a.bricks, 4, false},
            {a.rgba, 16 * n, true},
            {a.argb, 4 * n, true}};
}
cudaError_t launch_frame_render(const FrameArgs& a, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t,
                                cudaStream_t s)
{
    submit(s, Op{"walk", [=] { return frame_reads(a); }, nullptr});
    return cudaGetLastError();
}
cudaError_t launch_frame_segments(const FrameArgs& a, const SegArgs& sa, uint32_t, uint32_t, uint32_t, uint32_t,
                                  uint32_t shape, uint32_t, uint32_t, cudaStream_t s)
{
    auto accesses = [=] {
        std::vector<Access> r = frame_reads(a);
        const s3r_view& v = *a.view;
        const uint64_t npix = (uint64_t)(a.cover[2] - a.cover[0]) * (uint64_t)(a.cover[3] - a.cover[1]);
        const uint32_t ranks = 3 * (1u << v.level) - 2;
        r.push_back({sa.count, 4, false});
        r.push_back({sa.items, *sa.count * sizeof(uint2), false});
        r.push_back({sa.seg, ranks * npix * 16, true});
        r.push_back({sa.mask, sa.words * npix * 8, true});
        r.push_back({sa.queue, 4, true});
        return r;
    };
    // the items have to cover every block's rectangle of the table that is there now
    auto body = [=] {
        std::map<uint32_t, uint32_t> lanes, tiles;
        for (uint32_t i = 0; i < *sa.count; ++i) {
            const uint32_t cell = sa.items[i].x & kSegCellMask;
            lanes[cell] = sa.lanes ? sa.items[i].x >> kSegLanesShift : 0;
            if (sa.items[i].y != tiles[cell]++) trouble("segments: items out of order");
        }
        for (uint32_t c = 0; c < 1u << (3 * a.view->level); ++c) {
            const RenderBlock& t = a.table[c];
            if (t.depth == 0xffffffffu || t.rect[2] <= 0 || t.rect[3] <= 0) continue;
            uint32_t w, h;
            seg_footprint((uint32_t)kSegShapeX[shape], lanes[c], w, h);
            if (tiles[c] < (((uint32_t)t.rect[2] + w - 1) / w) * (((uint32_t)t.rect[3] + h - 1) / h))
                trouble("segments: items of another view");
        }
    };
    submit(s, Op{"segments", accesses, body});
    return cudaGetLastError();
}
cudaError_t launch_seg_items(const uint2* list, uint32_t n, uint2* items, cudaStream_t s)
{
    auto accesses = [=] {
        return std::vector<Access>{{list, (n + 1) * sizeof(uint2), false}, {items, list[n].y * sizeof(uint2), true}};
    };
    submit(s, Op{"seg_items", accesses, [=] {
                     for (uint32_t b = 0; b < n; ++b)
                         for (uint32_t t = 0; list[b].y + t < list[b + 1].y; ++t)
                             items[list[b].y + t] = make_uint2(list[b].x, t);
                 }});
    return cudaGetLastError();
}
cudaError_t launch_frame_render_mode(const FrameArgs& a, const s3r_presentation&, const float*, uint32_t, uint32_t,
                                     uint32_t, uint32_t, cudaStream_t s)
{
    submit(s, Op{"mode", [=] { return frame_reads(a); }, nullptr});
    return cudaGetLastError();
}
cudaError_t launch_frame_backward(const FrameArgs& a, uint32_t, uint32_t, uint32_t, cudaStream_t s)
{
    return kernel(s, "backward", {{a.table, 4, false}});
}
cudaError_t launch_dtf_reduce(const float* part, float*, uint32_t, cudaStream_t s)
{
    return kernel(s, "dtf_reduce", {{part, 4, false}});
}
cudaError_t launch_bound_rect(const uint32_t* img, uint32_t W, uint32_t H, int32_t* acc, int32_t* host, cudaStream_t s)
{
    return kernel(s, "bound_rect", {{img, 4ull * W * H, false}, {acc, 24, true}, {host, 20, true}}, [=] {
        host[0] = host[2] = (int32_t)W; // all of the image
        host[1] = host[3] = (int32_t)H;
        host[4] = 0;
    });
}
cudaError_t launch_crop(const uint32_t*, uint32_t, const int32_t*, uint32_t*, cudaStream_t s) { return kernel(s, "crop", {}); }
cudaError_t launch_compose(const s3r_image_part*, const s3r_image_part*, uint32_t, int32_t, uint32_t*, int32_t, int32_t,
                           int32_t, int32_t, cudaStream_t s)
{
    return kernel(s, "compose", {});
}

} // namespace s3r
