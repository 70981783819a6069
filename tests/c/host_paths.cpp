// The library's host paths over a made-up CUDA runtime: vx_api.cpp linked with
// the calls below instead of the runtime's and with launchers that do their
// work at once on the host.  The runtime keeps, for every stream and event,
// which enqueued work it follows, and compares every access to a buffer with
// the earlier ones to the same bytes; it counts what is allocated; and it fails
// any one call on request.  Each scenario prints what it finds wrong.
#include <cuda_runtime.h>

#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "vx_internal.h"

namespace {
std::recursive_mutex g_mu;
int g_wrong = 0;
void wrong(const std::string &what) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (++g_wrong <= 20) std::printf("  wrong: %s\n", what.c_str());
}

using Clock = std::vector<long>;   // per stream: its last operation known to be over
void join(Clock &a, const Clock &b) {
    if (a.size() < b.size()) a.resize(b.size(), 0);
    for (size_t i = 0; i < b.size(); ++i) a[i] = std::max(a[i], b[i]);
}
struct Stream {
    size_t id;
    Clock clock;
};
struct Event {
    Clock clock;
    size_t stream = ~(size_t)0;    // recorded on
};
struct Access {
    const uint8_t *lo, *hi;
    bool write;
    size_t stream;
    long at;
};
std::set<Stream *> g_streams;
std::set<Event *> g_events;
std::map<uint8_t *, size_t> g_dev, g_pinned;
std::vector<Access> g_log;
Clock g_host;                      // what the host has waited for
size_t g_next_stream = 0, g_allocs = 0;
long g_calls = 0, g_fail_at = 0;   // fails the g_fail_at-th call from here
bool g_failed = false, g_making = false;   // g_making: only calls that make something fail

// while set, waits for streams that trace pick batches do not end
bool g_hold = false;
size_t g_held = 0;
std::condition_variable_any g_cv;
std::set<size_t> g_batch_streams;
std::vector<size_t> g_batch_sizes;  // whole-batch sizes that launch_raycast was given

bool fails(bool makes = false) {
    ++g_calls;
    if (g_making && !makes) return false;
    if (g_fail_at > 0 && --g_fail_at == 0) {
        g_failed = true;
        return true;
    }
    return false;
}
void hold(std::unique_lock<std::recursive_mutex> &lk, size_t stream) {
    if (!g_hold || !g_batch_streams.count(stream)) return;
    ++g_held;
    g_cv.notify_all();
    g_cv.wait(lk, [] { return !g_hold; });
}
Stream *live(cudaStream_t s, const char *call) {
    Stream *p = reinterpret_cast<Stream *>(s);
    if (!g_streams.count(p)) {
        wrong(std::string(call) + " on a stream that does not exist");
        return nullptr;
    }
    return p;
}
Event *live(cudaEvent_t e, const char *call) {
    Event *p = reinterpret_cast<Event *>(e);
    if (!g_events.count(p)) {
        wrong(std::string(call) + " on an event that does not exist");
        return nullptr;
    }
    return p;
}
size_t bytes_of(const std::map<uint8_t *, size_t> &m) {
    size_t n = 0;
    for (auto &a : m) n += a.second;
    return n;
}
// work enqueued on s that touches these ranges
struct Range {
    const void *p;
    size_t n;
    bool write;
};
void enqueue(cudaStream_t st, const char *call, std::initializer_list<Range> ranges) {
    Stream *s = live(st, call);
    if (!s) return;
    join(s->clock, g_host);
    if (s->clock.size() <= s->id) s->clock.resize(s->id + 1, 0);
    const long at = ++s->clock[s->id];
    for (const Range &r : ranges) {
        if (!r.p || !r.n) continue;
        const uint8_t *lo = static_cast<const uint8_t *>(r.p), *hi = lo + r.n;
        for (const Access &a : g_log) {
            if (a.hi <= lo || hi <= a.lo || !(a.write || r.write) || a.stream == s->id) continue;
            if (a.stream >= s->clock.size() || s->clock[a.stream] < a.at)
                wrong(std::string(call) + " does not follow earlier work on the same bytes");
        }
        g_log.push_back({lo, hi, r.write, s->id, at});
    }
}
void forget(uint8_t *p, size_t n) {
    std::vector<Access> keep;
    for (const Access &a : g_log)
        if (a.hi <= p || p + n <= a.lo) keep.push_back(a);
        else if (a.stream >= g_host.size() || g_host[a.stream] < a.at)
            wrong("memory freed while work on it is under way");
    g_log.swap(keep);
}
cudaError_t give(void **p, size_t n, std::map<uint8_t *, size_t> &m) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (fails(true)) return cudaErrorMemoryAllocation;
    ++g_allocs;
    uint8_t *q = static_cast<uint8_t *>(std::malloc(n ? n : 1));
    std::memset(q, 0xA5, n);
    m[q] = n;
    *p = q;
    return cudaSuccess;
}
cudaError_t take(void *p, std::map<uint8_t *, size_t> &m) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (!p) return cudaSuccess;
    auto it = m.find(static_cast<uint8_t *>(p));
    if (it == m.end()) {
        wrong("memory freed that is not allocated");
        return cudaErrorInvalidValue;
    }
    // cudaFree waits for the device
    for (Stream *s : g_streams) join(g_host, s->clock);
    forget(it->first, it->second);
    std::free(it->first);
    m.erase(it);
    return cudaSuccess;
}
}  // namespace

extern "C" {
const char *cudaGetErrorString(cudaError_t) { return "made up"; }
cudaError_t cudaSetDevice(int) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    return fails() ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return give(p, n, g_dev); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return give(p, n, g_dev); }
cudaError_t cudaFree(void *p) { return take(p, g_dev); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return take(p, g_dev); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return give(p, n, g_pinned); }
cudaError_t cudaFreeHost(void *p) { return take(p, g_pinned); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) {
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (fails(true)) return cudaErrorUnknown;
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (fails()) return cudaErrorUnknown;
    enqueue(st, "cudaMemcpyAsync", {{s, n, false}, {d, n, true}});
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (fails()) return cudaErrorUnknown;
    enqueue(st, "cudaMemsetAsync", {{d, n, true}});
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (fails(true)) return cudaErrorUnknown;
    Stream *p = new Stream{g_next_stream++, {}};
    g_streams.insert(p);
    *s = reinterpret_cast<cudaStream_t>(p);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (Stream *p = live(s, "cudaStreamDestroy")) {
        join(g_host, p->clock);
        g_streams.erase(p);
        delete p;
    }
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::unique_lock<std::recursive_mutex> lk(g_mu);
    if (fails()) return cudaErrorUnknown;
    Stream *p = live(s, "cudaStreamSynchronize");
    if (!p) return cudaErrorUnknown;
    hold(lk, p->id);
    join(g_host, p->clock);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    for (Stream *s : g_streams) join(g_host, s->clock);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (fails(true)) return cudaErrorUnknown;
    Event *p = new Event;
    g_events.insert(p);
    *e = reinterpret_cast<cudaEvent_t>(p);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (Event *p = live(e, "cudaEventDestroy")) {
        g_events.erase(p);
        delete p;
    }
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (fails()) return cudaErrorUnknown;
    Event *p = live(e, "cudaEventRecord");
    Stream *q = live(s, "cudaEventRecord");
    if (p && q) {
        join(q->clock, g_host);
        p->clock = q->clock;
        p->stream = q->id;
    }
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::unique_lock<std::recursive_mutex> lk(g_mu);
    if (fails()) return cudaErrorUnknown;
    if (Event *p = live(e, "cudaEventSynchronize")) {
        hold(lk, p->stream);
        join(g_host, p->clock);
    }
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (fails()) return cudaErrorUnknown;
    Stream *q = live(s, "cudaStreamWaitEvent");
    Event *p = live(e, "cudaStreamWaitEvent");
    if (p && q) join(q->clock, p->clock);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.0f;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) {
    return cudaErrorUnknown;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorUnknown; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorUnknown; }
}  // extern "C"

namespace vx {
#define OVER std::lock_guard<std::recursive_mutex> lk(g_mu); if (fails()) return cudaErrorUnknown
cudaError_t QueueScratch::reserve(size_t) { return cudaErrorUnknown; }
void QueueScratch::release() {}
cudaError_t launch_beam(const FrameArgs &fa, float *beam, cudaStream_t s) {
    OVER;
    enqueue(s, "launch_beam", {{beam, sizeof(float) * fa.bw * fa.bh, true}});
    return cudaSuccess;
}
// every record names its row and the frame's jitter, so a test sees whose it is
cudaError_t launch_primary(const FrameArgs &fa, cudaStream_t s) {
    OVER;
    const size_t a = (size_t)fa.y0 * fa.W, n = (size_t)(fa.y1 - fa.y0) * fa.W;
    enqueue(s, "launch_primary",
            {{fa.beam, sizeof(float) * fa.bw * fa.bh, false},
             {fa.rec + a, n * sizeof(VxHitRecord), true},
             {fa.shadow ? fa.shadow + a : nullptr, fa.shadow ? n * sizeof(VxShadowRecord) : 0, true}});
    for (size_t i = a; i < a + n; ++i) {
        std::memset(fa.rec + i, 0, sizeof(VxHitRecord));
        fa.rec[i].voxel[0] = (int32_t)i;
        fa.rec[i].steps = (uint32_t)fa.cam.jitter_x;
    }
    return cudaSuccess;
}
cudaError_t launch_pack_compact(const VxHitRecord *rec, const VxShadowRecord *sh, size_t first,
                                size_t n, const int32_t *, uint32_t, uint32_t, VxCompactRecord *out,
                                uint32_t *, cudaStream_t s) {
    OVER;
    enqueue(s, "launch_pack_compact", {{rec + first, n * sizeof(VxHitRecord), false},
                                       {sh + first, n * sizeof(VxShadowRecord), false},
                                       {out + first, n * sizeof(VxCompactRecord), true}});
    for (size_t i = first; i < first + n; ++i) out[i].w[0] = (uint32_t)rec[i].voxel[0];
    return cudaSuccess;
}
cudaError_t launch_pack(const VxHitRecord *rec, const VxShadowRecord *sh, size_t first, size_t n,
                        const int32_t *, uint32_t, uint32_t, VxPackedRecord *out, cudaStream_t s) {
    OVER;
    enqueue(s, "launch_pack", {{rec + first, n * sizeof(VxHitRecord), false},
                               {sh + first, n * sizeof(VxShadowRecord), false},
                               {out + first, n * sizeof(VxPackedRecord), true}});
    return cudaSuccess;
}
cudaError_t launch_raycast_one(const DevWorld &, const int32_t *, const float cam[3], const float *,
                               VxPickHit *out, int32_t *hit, cudaStream_t s) {
    OVER;
    enqueue(s, "launch_raycast_one", {{out, sizeof *out, true}});
    out->voxel[0] = (int32_t)cam[0];
    *hit = 1;
    return cudaSuccess;
}
cudaError_t launch_raycast(const DevWorld &, const int32_t *, const float *cams, const float *dirs,
                           size_t n, size_t batch, VxPickHit *out, int32_t *hit, bool,
                           const uint32_t *, cudaStream_t s) {
    OVER;
    g_batch_sizes.push_back(batch);
    enqueue(s, "launch_raycast", {{cams, n * 12, false}, {dirs, n * 12, false},
                                  {out, n * sizeof *out, true}, {hit, n * 4, true}});
    if (Stream *p = live(s, "launch_raycast")) g_batch_streams.insert(p->id);
    for (size_t i = 0; i < n; ++i) {
        out[i].voxel[0] = (int32_t)cams[3 * i];
        out[i].normal[2] = (int32_t)dirs[3 * i + 2];
        hit[i] = (int32_t)cams[3 * i + 1];
    }
    return cudaSuccess;
}
cudaError_t launch_masks_hold(const DevWorld &, uint32_t *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_tile_meta(const DevWorld &, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ao(const DevWorld &, const VxCamera &, const VxHitRecord *, float *,
                      cudaStream_t) { return cudaSuccess; }
cudaError_t launch_project_dirty(const DevWorld &, const VxCamera &, const uint32_t *, size_t,
                                 uint32_t *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_refresh_tiles(uint32_t, uint32_t, uint32_t, uint32_t, uint32_t *,
                                 cudaStream_t) { return cudaSuccess; }
cudaError_t launch_bricks_from_aos(const DevWorld &, const VxBrick *, int64_t, int64_t,
                                   cudaStream_t) { return cudaSuccess; }
cudaError_t launch_bricks_to_aos(const DevWorld &, VxBrick *, int64_t, int64_t,
                                 cudaStream_t) { return cudaSuccess; }
size_t gen_prim_bytes_per_src() { return 1; }
cudaError_t launch_gen_math(const uint32_t *, uint32_t, const float *, size_t, float *,
                            cudaStream_t) { return cudaSuccess; }
cudaError_t launch_gen_slots(const DevWorld &, uint64_t, const GenPlan &, bool,
                             cudaStream_t) { return cudaSuccess; }
cudaError_t launch_generate(const DevWorld &, const VxTerrainParams &, int16_t *,
                            cudaStream_t) { return cudaSuccess; }
cudaError_t launch_dist_fields(const DevWorld &, uint8_t *, uint8_t *, uint8_t *,
                               cudaStream_t) { return cudaSuccess; }
cudaError_t launch_edits(const DevWorld &, const uint2 *, size_t, const uint32_t *, size_t,
                         cudaStream_t) { return cudaSuccess; }
cudaError_t launch_apply_dirty_last_wins(const DevWorld &w, uint32_t *win, const uint32_t *idx,
                                         const VxBrick *bricks, size_t n, cudaStream_t s) {
    OVER;
    enqueue(s, "launch_apply_dirty", {{idx, n * 4, false}, {bricks, n * sizeof(VxBrick), false},
                                      {win, (size_t)w.d.n_bricks * 4, true}});
    for (size_t i = 0; i < n; ++i)
        if (win[idx[i]] != 0u) wrong("claims of an update that are not zero");
    return cudaSuccess;
}
cudaError_t launch_queue(const TraceArgs &, const VxRay *, size_t, VxHitRecord *, VxShadowRecord *,
                         const VxQueueTuning &, QueueScratch &, cudaStream_t) { return cudaSuccess; }
cudaError_t queue_fingerprint(const VxHitRecord *, size_t, const VxShadowRecord *, QueueScratch &,
                              cudaStream_t, unsigned long long *) { return cudaSuccess; }
cudaError_t launch_trace_rays(const TraceArgs &, const VxRay *, size_t, VxHitRecord *,
                              cudaStream_t) { return cudaSuccess; }
}  // namespace vx

namespace {
VxWorld *make_world() {
    VxWorldDesc d{};
    d.bricks_x = d.bricks_z = 64;
    d.bricks_y = 16;
    VxWorld *w = nullptr;
    if (vx_world_create(&d, &w) != VX_OK) wrong("no world");
    return w;
}
void end_world(VxWorld *w) {
    g_fail_at = 0;
    vx_world_destroy(w);
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (!g_dev.empty() || !g_pinned.empty() || !g_streams.empty() || !g_events.empty())
        wrong("a destroyed world leaves " + std::to_string(g_dev.size() + g_pinned.size()) +
              " buffers, " + std::to_string(g_streams.size()) + " streams and " +
              std::to_string(g_events.size()) + " events");
    g_log.clear();
    g_batch_streams.clear();
}

struct Batch {
    std::vector<float> cams, dirs;
    std::vector<VxPickHit> out;
    std::vector<int32_t> hit;
    explicit Batch(size_t n) : cams(3 * n), dirs(3 * n), out(n), hit(n) {
        for (size_t i = 0; i < n; ++i) {
            cams[3 * i] = (float)(i % 9973);
            cams[3 * i + 1] = (float)(i % 9967);
            dirs[3 * i + 2] = (float)(i % 9949);
        }
    }
    int run(VxWorld *w) {
        const int32_t o[3] = {0, 0, 0};
        return vx_raycast_batch_host(w, o, cams.data(), dirs.data(), hit.size(), out.data(),
                                     hit.data());
    }
    void check(const char *what) {
        for (size_t i = 0; i < hit.size(); ++i)
            if (out[i].voxel[0] != (int32_t)(i % 9973) || hit[i] != (int32_t)(i % 9967) ||
                out[i].normal[2] != (int32_t)(i % 9949)) {
                wrong(std::string(what) + ": result " + std::to_string(i));
                return;
            }
    }
};

// results right; later calls allocate nothing, whether earlier results are kept
// or not; what the world keeps does not grow with the batch
void batch_memory() {
    VxWorld *w = make_world();
    const size_t dev0 = bytes_of(g_dev), pinned0 = bytes_of(g_pinned);
    std::vector<Batch> kept;
    for (size_t n : {(size_t)1, (size_t)12288, (size_t)12289, (size_t)200000, (size_t)3000001}) {
        kept.emplace_back(n);
        if (kept.back().run(w) != VX_OK) wrong("batch");
        kept.back().check("batch");
    }
    for (size_t n : {(size_t)3000001, (size_t)200000, (size_t)7}) {
        const size_t before = g_allocs;
        kept.emplace_back(n);
        if (kept.back().run(w) != VX_OK) wrong("batch");
        kept.back().check("batch");
        if (g_allocs != before) wrong("a batch no larger than an earlier one allocates");
    }
    // every launch of a batch knows the whole batch's size, which picks the kernel
    g_batch_sizes.clear();
    if (kept[3].run(w) != VX_OK || g_batch_sizes.size() < 2) wrong("batch");
    for (size_t n : g_batch_sizes)
        if (n != 200000) wrong("a chunk is launched as a batch of " + std::to_string(n));
    if (bytes_of(g_dev) - dev0 > (size_t)28 << 20) wrong("device memory kept grows with the batch");
    if (bytes_of(g_pinned) - pinned0 > (size_t)15 << 20)
        wrong("page-locked memory kept grows with the batch");
    // a new world's first batch finds them: page-locking takes a millisecond per MB
    VxWorld *v = make_world();
    const size_t before = g_allocs;
    if (kept[3].run(v) != VX_OK) wrong("batch");
    if (g_allocs != before) wrong("a new world's first batch allocates");
    vx_world_destroy(v);
    // the last world takes them along
    end_world(w);
}

// while a batch runs, the world's other calls and other batches do too
void batch_beside_others() {
    VxWorld *w = make_world();
    Batch a(30000), b(100);
    {
        std::lock_guard<std::recursive_mutex> lk(g_mu);
        g_hold = true;
        g_held = 0;
    }
    std::thread t([&] {
        if (a.run(w) != VX_OK) wrong("batch");
    });
    {
        std::unique_lock<std::recursive_mutex> lk(g_mu);
        if (!g_cv.wait_for(lk, std::chrono::seconds(20), [] { return g_held > 0; }))
            wrong("the batch does not get to the device");
    }
    bool one = false;
    std::thread u([&] {
        const float cam[3] = {5.f, 0.f, 0.f}, dir[3] = {0.f, 1.f, 0.f};
        const int32_t o[3] = {0, 0, 0};
        VxPickHit h;
        const int rc = vx_raycast(w, cam, dir, o, &h);
        std::lock_guard<std::recursive_mutex> lk(g_mu);
        one = rc == 1 && h.voxel[0] == 5;
        g_cv.notify_all();
    });
    std::thread v([&] {
        if (b.run(w) != VX_OK) wrong("second batch");
    });
    {
        std::unique_lock<std::recursive_mutex> lk(g_mu);
        if (!g_cv.wait_for(lk, std::chrono::seconds(5), [&] { return one; }))
            wrong("a single pick waits for another thread's batch");
        const size_t first = g_held;
        (void)first;
        if (!g_cv.wait_for(lk, std::chrono::seconds(5), [&] { return g_held >= 2; }))
            wrong("a batch waits for another thread's batch");
        g_hold = false;
        g_cv.notify_all();
    }
    for (std::thread *x : {&t, &u, &v}) x->join();
    a.check("held batch");
    b.check("second batch");
    end_world(w);
}

// any one call fails: the batch says so, and the next one is right
void batch_errors() {
    long k = 0;
    for (bool more = true; more && k < 2000; ) {
        ++k;
        VxWorld *w = make_world();
        Batch b(40000);
        g_failed = false;
        g_fail_at = k;
        const int rc = b.run(w);
        more = g_failed;
        g_fail_at = 0;
        if (more != (rc != VX_OK)) wrong("batch: call " + std::to_string(k) + " fails, the batch returns " + std::to_string(rc));
        Batch c(40000);
        if (c.run(w) != VX_OK) wrong("batch after a failed call");
        c.check("batch after a failed call");
        end_world(w);
    }
    if (k < 10) wrong("few calls to fail");
}

struct Frames {
    VxCamera cam{};
    VxTraceParams p{};
    std::vector<VxHitRecord> rec;
    std::vector<VxShadowRecord> sh;
    std::vector<VxCompactRecord> compact;
    explicit Frames(uint32_t width = 64, uint32_t height = 96) {
        vx_default_params(&p);
        const float pos[3] = {128.f, 32.f, 128.f};
        const int32_t o[3] = {0, 0, 0};
        vx_camera_from_pose(pos, 0.f, 0.f, 1.f, width, height, o, &cam);
        rec.resize((size_t)width * height);
        sh.resize((size_t)width * height);
        compact.resize((size_t)width * height);
    }
    int full(VxWorld *w) { return vx_render_primary_host(w, &cam, &p, rec.data(), sh.data()); }
    int small(VxWorld *w) { return vx_render_primary_host_compact(w, &cam, &p, compact.data()); }
    void check() {
        for (size_t i = 0; i < rec.size(); ++i)
            if (rec[i].voxel[0] != (int32_t)i) {
                wrong("frame: record " + std::to_string(i));
                return;
            }
    }
    void check_compact() {
        for (size_t i = 0; i < compact.size(); ++i)
            if (compact[i].w[0] != (uint32_t)i) {
                wrong("compact frame: record " + std::to_string(i));
                return;
            }
    }
};

// frames of every split into bands and streams, one after the other on one
// world: 4 bands on two streams, 6 on two, 4 on one, and fewer rows than bands
void frame_sizes() {
    VxWorld *w = make_world();
    const uint32_t sizes[][2] = {{640, 360}, {1, 8}, {7, 1}, {1111, 1264}, {1921, 1081}, {1280, 720},
                                 {1600, 1529}, {1600, 1530}, {2560, 1440}, {33, 9}, {1921, 1081}};
    for (auto &q : sizes) {
        Frames f(q[0], q[1]);
        for (int i = 0; i < 2; ++i) {
            std::memset(f.rec.data(), 0xFF, f.rec.size() * sizeof f.rec[0]);
            if (f.full(w) != VX_OK) wrong("frame");
            f.check();
            if (f.small(w) != VX_OK) wrong("compact frame");
            f.check_compact();
        }
    }
    end_world(w);
}

// any one call (with making: of those that make something) of a host frame
// fails: the frame says so, and the next ones use only streams and events that
// exist and wait for what the failed one left
void frames(bool making) {
    for (int warm = 0; warm < 3; ++warm) {
        long k = 0;
        for (bool more = true; more && k < 2000; ) {
            ++k;
            VxWorld *w = make_world();
            Frames f;
            for (int i = 0; i < warm; ++i)
                if (f.full(w) != VX_OK) wrong("frame");
            g_failed = false;
            g_making = making;
            g_fail_at = k;
            const int rc = (k & 1) ? f.full(w) : f.small(w);
            more = g_failed || k < 4;
            g_fail_at = 0;
            g_making = false;
            if (g_failed != (rc != VX_OK)) wrong("frame: call " + std::to_string(k) + " fails, the frame returns " + std::to_string(rc));
            for (int i = 0; i < 3; ++i) {
                if (f.full(w) != VX_OK) wrong("frame after a failed call");
                f.check();
                if (f.small(w) != VX_OK) wrong("compact frame after a failed call");
            }
            end_world(w);
        }
    }
}
void frame_handles() { frames(true); }
void frame_errors() { frames(false); }

// the same for an update of bricks
void update_handles() {
    long k = 0;
    for (bool more = true; more && k < 2000; ) {
        ++k;
        VxWorld *w = make_world();
        std::vector<uint32_t> idx = {3, 9, 3};
        std::vector<VxBrick> b(3);
        g_failed = false;
        g_making = true;
        g_fail_at = k;
        const int rc = vx_world_apply_dirty(w, idx.data(), b.data(), 3, nullptr);
        more = g_failed;
        g_fail_at = 0;
        g_making = false;
        if (g_failed != (rc != VX_OK)) wrong("update: call " + std::to_string(k) + " fails, the update returns " + std::to_string(rc));
        for (int i = 0; i < 3; ++i)
            if (vx_world_apply_dirty(w, idx.data(), b.data(), 3, nullptr) != VX_OK)
                wrong("update after a failed call");
        end_world(w);
    }
    if (k < 5) wrong("few calls to fail");
}
}  // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const std::map<std::string, void (*)()> all = {{"batch_memory", batch_memory},
                                                   {"batch_beside_others", batch_beside_others},
                                                   {"batch_errors", batch_errors},
                                                   {"frame_sizes", frame_sizes},
                                                   {"frame_handles", frame_handles},
                                                   {"update_handles", update_handles},
                                                   {"frame_errors", frame_errors}};
    auto it = all.find(what);
    if (it == all.end()) return 2;
    it->second();
    std::printf("%s: %d wrong\n", what.c_str(), g_wrong);
    return g_wrong == 0 ? 0 : 1;
}
