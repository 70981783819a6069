// vx_queue.cu -- the mixed ray queue: rays of different kinds and very
// uneven lengths (primary with spawned shadow, GI-probe, picking, any-hit
// line-of-sight, no-water) traced by ONE persistent launch.
//
// Every lane walks one ray at a time with the shared cascade step
// (vx_walk.cuh) and takes the next queue item when its ray ends; a primary
// that hits and carries VX_RAY_SPAWN_SHADOW continues in the same lane with
// its shadow ray (raymarch.wgsl:3953-3994).  Lanes of a warp refill together
// once `refill_min` of them are idle (a lone refill would stall 31 lanes
// through a ray set-up).  Optionally the queue is first reordered by a 22-bit
// coherence key -- kind, then the direction on a 1024x1024 octahedral grid in
// Morton order, crossed with the 64-voxel origin cell -- by a counting sort,
// so that a warp's rays head the same way from nearby origins: rays of one
// camera fall into pixel-sized direction cells, the rays of one probe site
// stay together.  Results do not depend on any of these choices; the
// autotuner checks that and keeps the fastest.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "vx_internal.h"
#include "vx_walk.cuh"

namespace vx {
namespace {

struct QueueArgs {
    TraceArgs ta;
    const VxRay *rays;
    const uint32_t *order;    // ray numbers by key, or nullptr (identity order)
    uint32_t n;
    VxHitRecord *out;
    VxShadowRecord *shadow;   // shadow records of spawning rays, or nullptr
    uint32_t *work;           // {next item, warps done}, self-resetting
    uint32_t refill_min;
};

__device__ __forceinline__ void load_ray(const VxRay *rays, uint32_t i, float &ox, float &oy,
                                         float &oz, float &dx, float &dy, float &dz, float &tmax,
                                         uint32_t &kind) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(rays + i));
    const float4 b = __ldg(reinterpret_cast<const float4 *>(rays + i) + 1);
    ox = a.x; oy = a.y; oz = a.z; dx = a.w; dy = b.x; dz = b.y; tmax = b.z;
    kind = __float_as_uint(b.w);
}

// The shadow ray of ray `ray` after its hit h (raymarch.wgsl:3953-3994: the
// origin p_hit + n*0.001, the sun direction jittered in its cone); the jitter
// is seeded by the ray index.
struct ShadowRay {
    float ox, oy, oz, dx, dy, dz;
};
__device__ __forceinline__ ShadowRay shadow_of(const VxTraceParams &p, uint32_t ray, float ox,
                                               float oy, float oz, float dx, float dy, float dz,
                                               const Hit &h) {
    ShadowRay r;
    const int ax = (int)(h.face >> 1);
    const float nv = (h.face & 1u) ? -1.0f : 1.0f;
    r.ox = (ox + dx * h.t) + (ax == 0 ? nv : 0.0f) * 0.001f;
    r.oy = (oy + dy * h.t) + (ax == 1 ? nv : 0.0f) * 0.001f;
    r.oz = (oz + dz * h.t) + (ax == 2 ? nv : 0.0f) * 0.001f;
    const float jit = ign((float)(ray & 0xFFFFu), (float)(ray >> 16), p.frame);
    const float theta = jit * 2.39996323f;
    const float radius = p.cone_tan * sqrtf(jit);
    float sn, cs;
    sincos_series(theta, sn, cs);
    r.dx = p.sun[0] + (p.sun_tangent[0] * cs + p.sun_bitangent[0] * sn) * radius;
    r.dy = p.sun[1] + (p.sun_tangent[1] * cs + p.sun_bitangent[1] * sn) * radius;
    r.dz = p.sun[2] + (p.sun_tangent[2] * cs + p.sun_bitangent[2] * sn) * radius;
    normalize3(r.dx, r.dy, r.dz);
    return r;
}

template <uint32_t FL>
__global__ void __launch_bounds__(256) k_queue(QueueArgs q) {
    constexpr uint32_t FULL = 0xFFFFFFFFu, IDLE = 0xFFFFFFFFu, DONE = 0xFFFFFFFEu;
    const uint32_t lane = threadIdx.x & 31u;
    const DevWorld &w = q.ta.w;
    const Ro ro{q.ta.ro[0], q.ta.ro[1], q.ta.ro[2]};
    const Geo g = geo_of<FL>(w.d, ro);
    const VxTraceParams &p = q.ta.p;
    uint64_t bytes = 0;
    Walk k;
    Hit h;
    uint32_t item = IDLE;     // queue slot being walked (IDLE / DONE otherwise)
    uint32_t ray = 0;         // index of the ray in q.rays
    uint32_t rkind = 0;       // kind word of that ray
    bool shadow_phase = false;
    float ox = 0.f, oy = 0.f, oz = 0.f;
    for (;;) {
        const bool need = item == IDLE;
        const unsigned ask = __ballot_sync(FULL, need);
        const unsigned busy = __ballot_sync(FULL, item < DONE);
        if (ask && ((uint32_t)__popc(ask) >= q.refill_min || busy == 0u)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(q.work, (uint32_t)__popc(ask));
            base = __shfl_sync(FULL, base, 0);
            if (need) {
                const uint32_t slot = base + (uint32_t)__popc(ask & ((1u << lane) - 1u));
                if (slot >= q.n) {
                    item = DONE;
                } else {
                    item = slot;
                    ray = q.order ? __ldg(q.order + slot) : slot;
                    float dx, dy, dz, tmax;
                    load_ray(q.rays, ray, ox, oy, oz, dx, dy, dz, tmax, rkind);
                    shadow_phase = false;
                    set_miss(h);
                    if (q.shadow) reinterpret_cast<uint2 *>(q.shadow)[ray] = make_uint2(0u, 0u);
                    const uint32_t kind = rkind & 3u;
                    if (!walk_init(w.d, ro, kind > 2u ? KIND_TRACE : kind, p, ox, oy, oz, dx, dy,
                                   dz, tmax, k)) {
                        if (kind == KIND_ANY) h.flags = 0u;
                        h.steps = 0;
                        store_record(q.out + ray, h);
                        item = IDLE;
                    }
                }
            }
        }
        if (__all_sync(FULL, item == DONE)) break;
        if (item < DONE) {
            const int r = walk_step<FL, false, -1>(w, g, p, ro, k, h, bytes);
            if (r != WALK_CONT) {
                item = IDLE;
                if (shadow_phase) {
                    reinterpret_cast<uint2 *>(q.shadow)[ray] =
                        make_uint2(k.iters, (r == WALK_HIT ? 1u : 0u) | (1u << 8));
                } else if (k.kind == KIND_ANY) {
                    set_miss(h);
                    h.flags = r == WALK_HIT ? 1u : 0u;
                    h.steps = k.iters;
                    store_record(q.out + ray, h);
                } else {
                    h.steps = k.iters;
                    store_record(q.out + ray, h);
                    if (q.shadow && (rkind & VX_RAY_SPAWN_SHADOW) && r == WALK_HIT) {
                        const ShadowRay sr =
                            shadow_of(p, ray, ox, oy, oz, k.s.dx, k.s.dy, k.s.dz, h);
                        if (walk_init(w.d, ro, KIND_ANY, p, sr.ox, sr.oy, sr.oz, sr.dx, sr.dy,
                                      sr.dz, p.shadow_max_dist, k)) {
                            shadow_phase = true;
                            item = 0u;
                        } else {
                            reinterpret_cast<uint2 *>(q.shadow)[ray] = make_uint2(0u, 1u << 8);
                        }
                    }
                }
            }
        }
    }
    if (lane == 0) {
        const uint32_t warps = gridDim.x * (blockDim.x >> 5);
        if (atomicAdd(q.work + 1, 1u) == warps - 1u) {
            q.work[0] = 0u;
            q.work[1] = 0u;
        }
    }
}

// Whole packets (refill_min 32: a warp refills when every lane is idle): a
// warp takes 32 queue items, walks their rays to the end, then their shadow
// rays.  No lane changes the kind of its ray inside a walk, so a warp of one
// kind walks in that kind's own loop, without the per-iteration votes and the
// kind tests of k_queue, whose lanes may hold any mix; a warp of several kinds,
// as an unsorted queue has them, in the mixed loop (one loop per kind in turn:
// 1.1 M unsorted rays of three kinds 646 us, 445 us as lane refill, 401 us here).
// A warp takes a packet when it has none: one asked for ahead kept others idle
// (90,000 unsorted rays, fewer packets than resident warps: 148 us, 97 without).
// Sorted 1080p mix (3.1M rays, 1.3M shadow rays), the queue with its sort: 777
// us as lane refill at 31, 676 here (690 with a packet asked for ahead).  At
// least 3 CTAs of 256 (70 registers): 2, 4 and 5 measured 3, 0.5 and 2 % slower.
template <uint32_t FL>
__global__ void __launch_bounds__(256, 3) k_queue_packet(QueueArgs q) {
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const DevWorld &w = q.ta.w;
    const Ro ro{q.ta.ro[0], q.ta.ro[1], q.ta.ro[2]};
    const VxTraceParams &p = q.ta.p;
    uint64_t bytes = 0;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(q.work, 32u);
        base = __shfl_sync(FULL, base, 0);
        if (base >= q.n) break;
        const uint32_t slot = base + lane;
        if (slot < q.n) {
            const uint32_t ray = q.order ? __ldg(q.order + slot) : slot;
            float ox, oy, oz, dx, dy, dz, tmax;
            uint32_t rkind;
            load_ray(q.rays, ray, ox, oy, oz, dx, dy, dz, tmax, rkind);
            const uint32_t kind = rkind & 3u;
            Hit h;
            uint32_t ssteps = 0, sword = 0;
            trace_ray_of_kind<FL>(w, p, ro, kind, ox, oy, oz, dx, dy, dz, tmax, h);
            if (q.shadow && kind != KIND_ANY && (rkind & VX_RAY_SPAWN_SHADOW) && (h.flags & 1u)) {
                const ShadowRay sr = shadow_of(p, ray, ox, oy, oz, dx, dy, dz, h);
                const bool occ = trace_any_ray<FL, false>(w, p, ro, sr.ox, sr.oy, sr.oz, sr.dx,
                                                          sr.dy, sr.dz, p.shadow_max_dist, ssteps,
                                                          bytes);
                sword = (occ ? 1u : 0u) | (1u << 8);
            }
            store_record(q.out + ray, h);
            if (q.shadow) reinterpret_cast<uint2 *>(q.shadow)[ray] = make_uint2(ssteps, sword);
        }
        __syncwarp();
    }
    if (lane == 0) {
        const uint32_t warps = gridDim.x * (blockDim.x >> 5);
        if (atomicAdd(q.work + 1, 1u) == warps - 1u) {
            q.work[0] = 0u;
            q.work[1] = 0u;
        }
    }
}

// ---- coherence reorder: a counting sort by a key of at most 22 bits
// key = kind(2) | Morton(octahedral direction, 10+10 bits) with the origin's
// 64-voxel cell XORed into its low 10 bits: rays of one origin stay in Morton
// order up to a reflection of blocks of 1024 cells, rays of one direction are
// parted by cell.  A launch of few rays drops low bits, to about four buckets
// a ray.
//
// What bounds it: the rays are read once (32 bytes each; the 1080p mix's 98 MB
// take 15 us at the copy rate); all else is in L2.  One pass counts, and the
// count a ray finds is its place in its bucket; the counts are summed up; one
// pass writes each ray's number to its place, 4 scattered bytes.  The order
// within a bucket is as the atomics fall: the records do not depend on it.
// 1080p mix, launches one by one: 212 us as four passes of a stable radix sort
// over 32-bit keys (histogram, row scan, scatter by digit runs each), 97 us
// so; the walks lose 15 us to the coarser order, the queue gains 87 (738 us to
// 651; 21 and 20 key bits: 666 and 660).
constexpr uint32_t kKeyBits = 22;
constexpr uint32_t kScanItems = 4096;    // buckets a CTA sums and scans

__device__ __forceinline__ uint32_t spread_bits(uint32_t x) {   // 10 bits -> even bits
    x &= 0x3FFu;
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}

__device__ __forceinline__ uint32_t ray_key(const VxRay *rays, uint32_t i, int32_t rox,
                                            int32_t roz) {
    float ox, oy, oz, dx, dy, dz, tmax;
    uint32_t kind;
    load_ray(rays, i, ox, oy, oz, dx, dy, dz, tmax, kind);
    // direction on the octahedral map, lower hemisphere folded out
    const float l1 = fabsf(dx) + fabsf(dy) + fabsf(dz);
    float u = l1 > 0.f ? dx / l1 : 0.f, v = l1 > 0.f ? dz / l1 : 0.f;
    if (dy < 0.f) {
        const float uu = (1.f - fabsf(v)) * (u < 0.f ? -1.f : 1.f);
        v = (1.f - fabsf(u)) * (v < 0.f ? -1.f : 1.f);
        u = uu;
    }
    const uint32_t qu = (uint32_t)min(1023, max(0, (int32_t)((u + 1.f) * 512.f)));
    const uint32_t qv = (uint32_t)min(1023, max(0, (int32_t)((v + 1.f) * 512.f)));
    const uint32_t morton = spread_bits(qu) | (spread_bits(qv) << 1);
    // origin cell of 64 voxels relative to the window corner (x, z) and in y
    auto cell = [](float o, int32_t corner) -> uint32_t {
        const float f = floorf(o);
        const int32_t c = f != f ? 0 : (int32_t)fminf(fmaxf(f - (float)corner, 0.f), 1e9f);
        return ((uint32_t)c >> 6) & 15u;
    };
    const uint32_t oc = cell(ox, rox) | (cell(oz, roz) << 4) | ((cell(oy, 0) & 3u) << 8);
    return ((kind & 3u) << 20) | (morton ^ oc);
}

// Each ray's bucket and its place in it.  Lanes of a warp with one bucket
// share an atomic, so rays that all share a few keys do not queue up.
__global__ void __launch_bounds__(256) k_sort_count(const VxRay *rays, uint32_t n, int32_t rox,
                                                    int32_t roz, uint32_t shift, uint32_t *counts,
                                                    uint2 *place) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < n;
    const unsigned lanes = __ballot_sync(0xFFFFFFFFu, live);
    if (!live) return;
    const uint32_t b = ray_key(rays, i, rox, roz) >> shift, lane = threadIdx.x & 31u;
    const unsigned peers = __match_any_sync(lanes, b);
    const int leader = __ffs((int)peers) - 1;
    uint32_t first = 0;
    if ((int)lane == leader) first = atomicAdd(counts + b, (uint32_t)__popc(peers));
    first = __shfl_sync(lanes, first, leader);
    place[i] = make_uint2(b, first + (uint32_t)__popc(peers & ((1u << lane) - 1u)));
}

__device__ __forceinline__ uint32_t block_sum256(uint32_t v, uint32_t *wsum) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    __syncthreads();                       // wsum may still be read by a previous call
    if (lane == 0) wsum[warp] = v;
    __syncthreads();
    uint32_t t = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8u; ++w) t += wsum[w];
    return t;
}

// sum of each CTA's 4096 buckets
__global__ void __launch_bounds__(256) k_sort_sums(const uint32_t *counts, uint32_t *sums) {
    __shared__ uint32_t wsum[8];
    const uint4 *c = reinterpret_cast<const uint4 *>(counts + (size_t)blockIdx.x * kScanItems);
    uint32_t v = 0;
#pragma unroll
    for (uint32_t k = 0; k < kScanItems / 1024u; ++k) {
        const uint4 q = c[threadIdx.x + 256u * k];
        v += (q.x + q.y) + (q.z + q.w);
    }
    v = block_sum256(v, wsum);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
}

// counts -> first place of each bucket, in place: 16 buckets a thread, from
// the sums of the CTAs before
__global__ void __launch_bounds__(256) k_sort_scan(uint32_t *counts, const uint32_t *sums) {
    __shared__ uint32_t wsum[8];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t base = 0;
    for (uint32_t k = tid; k < blockIdx.x; k += 256u) base += sums[k];
    base = block_sum256(base, wsum);
    uint4 *c = reinterpret_cast<uint4 *>(counts + (size_t)blockIdx.x * kScanItems) + tid * 4u;
    uint4 q[4];
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        q[k] = c[k];
        const uint32_t x = q[k].x, y = q[k].y, z = q[k].z, w = q[k].w;
        q[k] = make_uint4(run, run + x, run + x + y, run + x + y + z);
        run += (x + y) + (z + w);
    }
    uint32_t inc = run;                    // inclusive scan of thread totals in the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if ((int)lane >= o) inc += v;
    }
    __syncthreads();                       // wsum of the base is consumed
    if (lane == 31u) wsum[warp] = inc;
    __syncthreads();
    uint32_t first = base + inc - run;
#pragma unroll
    for (uint32_t w = 0; w < 8u; ++w) first += w < warp ? wsum[w] : 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        c[k] = make_uint4(first + q[k].x, first + q[k].y, first + q[k].z, first + q[k].w);
}

__global__ void __launch_bounds__(256) k_sort_place(const uint2 *place, uint32_t n,
                                                    const uint32_t *first, uint32_t *order) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint2 p = place[i];
    order[first[p.x] + p.y] = i;
}

// order-independent fingerprint of the outputs (autotuner consistency check)
__global__ void k_fingerprint(const uint32_t *a, size_t na, const uint32_t *b, size_t nb,
                              unsigned long long *out) {
    unsigned long long acc = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < na + nb;
         i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t v = i < na ? a[i] : b[i - na];
        unsigned long long x = ((unsigned long long)v << 32) ^ (unsigned long long)(i * 0x9E3779B97F4A7C15ull);
        x ^= x >> 29;
        x *= 0xBF58476D1CE4E5B9ull;
        x ^= x >> 32;
        acc += x;
    }
    atomicAdd(out, acc);
}

template <uint32_t FL>
struct QueueK {
    static void *fn() { return reinterpret_cast<void *>(&k_queue<FL>); }
};

template <uint32_t FL>
struct PacketK {
    static void *fn() { return reinterpret_cast<void *>(&k_queue_packet<FL>); }
};

void *queue_kernel(uint32_t fl, uint32_t refill_min) {
    return refill_min >= 32u ? pick_fl<PacketK>(fl) : pick_fl<QueueK>(fl);
}

}  // namespace

// key bits used for n rays: about four buckets a ray, a multiple of a CTA's
// share at least
static uint32_t sort_bits(size_t n) {
    uint32_t bits = 12;
    while (bits < kKeyBits && ((size_t)1 << bits) < 4 * n) ++bits;
    return bits;
}

cudaError_t QueueScratch::reserve(size_t n) {
    if (!work) {
        cudaError_t e = cudaMalloc(&work, 2 * sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaMemset(work, 0, 2 * sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaMalloc(&fp, sizeof(unsigned long long));
        if (e != cudaSuccess) return e;
    }
    if (cap >= n && place) return cudaSuccess;
    cudaFree(place);
    cudaFree(order);
    cudaFree(counts);
    place = nullptr;
    order = counts = nullptr;
    cap = 0;
    const size_t m = std::max<size_t>(n, 1), buckets = (size_t)1 << sort_bits(m);
    cudaError_t e = cudaMalloc(&place, m * sizeof(uint2));
    if (e == cudaSuccess) e = cudaMalloc(&order, m * sizeof(uint32_t));
    // the buckets, then the sums of kScanItems of them
    if (e == cudaSuccess)
        e = cudaMalloc(&counts, (buckets + buckets / kScanItems) * sizeof(uint32_t));
    if (e == cudaSuccess) cap = n;
    return e;
}

void QueueScratch::release() {
    cudaFree(work);
    cudaFree(place);
    cudaFree(order);
    cudaFree(counts);
    cudaFree(fp);
    *this = QueueScratch();
}

cudaError_t launch_queue(const TraceArgs &ta, const VxRay *rays, size_t n, VxHitRecord *out,
                         VxShadowRecord *shadow, const VxQueueTuning &t, QueueScratch &sc,
                         cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint32_t nn = (uint32_t)n;
    const uint32_t *order = nullptr;
    if (t.sort) {
        const uint32_t bits = sort_bits(n), buckets = 1u << bits;
        uint32_t *sums = sc.counts + buckets;
        cudaError_t e = cudaMemsetAsync(sc.counts, 0, (size_t)buckets * sizeof(uint32_t), s);
        if (e != cudaSuccess) return e;
        k_sort_count<<<(nn + 255) / 256, 256, 0, s>>>(rays, nn, ta.ro[0], ta.ro[2],
                                                      kKeyBits - bits, sc.counts, sc.place);
        k_sort_sums<<<buckets / kScanItems, 256, 0, s>>>(sc.counts, sums);
        k_sort_scan<<<buckets / kScanItems, 256, 0, s>>>(sc.counts, sums);
        k_sort_place<<<(nn + 255) / 256, 256, 0, s>>>(sc.place, nn, sc.counts, sc.order);
        order = sc.order;
    }
    QueueArgs q;
    q.ta = ta;
    q.rays = rays;
    q.order = order;
    q.n = nn;
    q.out = out;
    q.shadow = shadow;
    q.work = sc.work;
    q.refill_min = (uint32_t)std::min(32, std::max(1, t.refill_min));
    void *fn = queue_kernel((ta.p.flags & 7u) | pow2_bit(ta.w.d), q.refill_min);
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, t.block_threads, 0);
    if (e != cudaSuccess) return e;
    if (t.ctas_per_sm > 0) per_sm = std::min(per_sm, t.ctas_per_sm);
    per_sm = std::max(per_sm, 1);
    void *args[] = {&q};
    return cudaLaunchKernel(fn, dim3((unsigned)(sms * per_sm)), dim3((unsigned)t.block_threads),
                            args, 0, s);
}

cudaError_t queue_fingerprint(const VxHitRecord *out, size_t n, const VxShadowRecord *shadow,
                              QueueScratch &sc, cudaStream_t s, unsigned long long *host) {
    cudaError_t e = cudaMemsetAsync(sc.fp, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    k_fingerprint<<<296, 256, 0, s>>>(reinterpret_cast<const uint32_t *>(out), n * 6,
                                      reinterpret_cast<const uint32_t *>(shadow),
                                      shadow ? n * 2 : 0, sc.fp);
    e = cudaMemcpyAsync(host, sc.fp, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e;
}

}  // namespace vx
