// vx_world.cu -- device-resident world pyramid: layout conversion, seeded
// terrain generation, mask/LUT construction and the incremental dirty-brick
// update.  Compiled with --fmad=false (the terrain noise must match the CPU
// restatement bit for bit).
//
// Semantics follow src/voxel.rs: brick_uniform_of :233-247, tile_uniform_of
// :253-272, rebuild_all_uniform :946-957, rebuild_all_masks :958-1000,
// refresh_masks_for_brick :879-914 (the incremental update recomputes each
// touched tile/chunk/L4 word from its 64 children, which equals the value
// the reference's incremental bit maintenance keeps), noise :1163-1232,
// :1999-2021.
#include <cuda_runtime.h>

#include "vx_internal.h"
#include "vx_noise.cuh"

namespace vx {
namespace {

__device__ __forceinline__ int32_t f2i(float x) {
    if (x != x) return 0;
    if (x >= 1073741824.0f) return 1073741824;
    if (x <= -1073741824.0f) return -1073741824;
    return (int32_t)x;
}
__device__ __forceinline__ int child_bit(int lx, int ly, int lz) { return lx + lz * 4 + ly * 16; }

// ------------------------------------------------------------- layout
// voxelG's 72-byte Brick (AoS) <-> occupancy array + 64-byte material rows.
__global__ void k_aos_to_soa(DevWorld w, const VxBrick *__restrict__ aos, int64_t first,
                             int64_t count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint2 *src = reinterpret_cast<const uint2 *>(aos + i);
    const uint2 o = src[0];
    w.occ[first + i] = (uint64_t)o.x | ((uint64_t)o.y << 32);
    uint2 *dst = reinterpret_cast<uint2 *>(w.mat + (first + i) * 64);
#pragma unroll
    for (int k = 0; k < 8; ++k) dst[k] = src[1 + k];
}

__global__ void k_soa_to_aos(DevWorld w, VxBrick *__restrict__ aos, int64_t first,
                             int64_t count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    uint2 *dst = reinterpret_cast<uint2 *>(aos + i);
    const uint64_t o = w.occ[first + i];
    dst[0] = make_uint2((uint32_t)o, (uint32_t)(o >> 32));
    const uint2 *src = reinterpret_cast<const uint2 *>(w.mat + (first + i) * 64);
#pragma unroll
    for (int k = 0; k < 8; ++k) dst[1 + k] = src[k];
}

// brick_uniform_of, voxel.rs:233-247
__device__ __forceinline__ uint8_t uniform_of(uint64_t occ, const uint8_t *row) {
    if (occ != ~0ull) return 0;
    const uint4 *r = reinterpret_cast<const uint4 *>(row);
    const uint8_t m0 = row[0];
    if (m0 == 0) return 0;
    const uint32_t rep = 0x01010101u * m0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint4 q = r[k];
        if (q.x != rep || q.y != rep || q.z != rep || q.w != rep) return 0;
    }
    return m0;
}

// ------------------------------------------------------------- terrain
using noise::fbm_2d;
using noise::value_noise_3d;

struct GenArgs {
    DevWorld w;
    VxTerrainParams t;
    float off_x, off_z;   // seed_offset_xz, voxel.rs:1163-1167
    int16_t *heights;     // vx * vz column heights
};

__global__ void k_heights(GenArgs g) {
    const Dims &d = g.w.d;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)d.vx * d.vz) return;
    const int32_t x = (int32_t)(i % d.vx), z = (int32_t)(i / d.vx);
    const float fx = (float)x + g.off_x, fz = (float)z + g.off_z;
    const float n = fbm_2d(fx * g.t.inv_wavelength, fz * g.t.inv_wavelength, g.t.octaves);
    int32_t h = f2i(floorf(g.t.base_height + g.t.amplitude * n));
    if (h < 1) h = 1;
    if (h > d.vy - 1) h = d.vy - 1;
    g.heights[i] = (int16_t)h;
}

// One thread per brick: 64 voxels from the column heights + cave noise.
__global__ void k_gen_bricks(GenArgs g) {
    const Dims &d = g.w.d;
    const int64_t bi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (bi >= d.n_bricks) return;
    const int32_t bx = (int32_t)(bi % d.bx);
    const int32_t by = (int32_t)((bi / d.bx) % d.by);
    const int32_t bz = (int32_t)(bi / ((int64_t)d.bx * d.by));
    uint64_t occ = 0;
    uint32_t words[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) words[k] = 0;
    const float cinv = g.t.cave_inv_wavelength;
    for (int lz = 0; lz < 4; ++lz) {
        for (int lx = 0; lx < 4; ++lx) {
            const int32_t x = bx * 4 + lx, z = bz * 4 + lz;
            const int32_t h = g.heights[(int64_t)z * d.vx + x];
            const float fx = (float)x + g.off_x, fz = (float)z + g.off_z;
            for (int ly = 0; ly < 4; ++ly) {
                const int32_t y = by * 4 + ly;
                uint32_t m = 0;
                if (y <= h) {
                    bool cave = false;
                    if (y > 4 && y + 3 < h)
                        cave = value_noise_3d(fx * cinv, (float)y * cinv, fz * cinv) >
                               g.t.cave_threshold;
                    if (!cave) m = (y == h) ? 2u : ((y + g.t.dirt_depth >= h) ? 3u : 4u);
                } else if (y <= g.t.water_level) {
                    m = 12u;
                }
                if (m != 0u) {
                    const int vi = child_bit(lx, ly, lz);
                    occ |= 1ull << vi;
                    // vi is not a compile-time index here; build the word by shifts
                    const int wi = vi >> 2, sh = (vi & 3) * 8;
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        if (k == wi) words[k] |= m << sh;
                }
            }
        }
    }
    g.w.occ[bi] = occ;
    uint4 *row = reinterpret_cast<uint4 *>(g.w.mat + bi * 64);
#pragma unroll
    for (int k = 0; k < 4; ++k)
        row[k] = make_uint4(words[4 * k], words[4 * k + 1], words[4 * k + 2], words[4 * k + 3]);
    uint8_t u = 0;
    if (occ == ~0ull) {
        const uint32_t m0 = words[0] & 0xFFu;
        const uint32_t rep = 0x01010101u * m0;
        bool same = m0 != 0u;
#pragma unroll
        for (int k = 0; k < 16; ++k) same = same && (words[k] == rep);
        u = same ? (uint8_t)m0 : 0;
    }
    g.w.brick_uniform[bi] = u;
}

// ------------------------------------------------------------- pyramid
// A word of 64 child bits by one warp: lane i tests children i and i + 32
// (child bit x + z*4 + y*16), so the 64 loads leave in one round instead of
// one after the other (a thread per word: 16 us for a level of 4,096 chunks,
// 17 us for 64 L4 cells, the latency of 64 loads in turn; a warp: 5 us).
template <typename F>
__device__ __forceinline__ uint64_t warp_child_mask(F test) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lo = __ballot_sync(0xFFFFFFFFu, test((int32_t)lane));
    const uint32_t hi = __ballot_sync(0xFFFFFFFFu, test((int32_t)lane + 32));
    return (uint64_t)lo | ((uint64_t)hi << 32);
}

// the same by one thread, its 64 loads in turn
template <typename F>
__device__ __forceinline__ uint64_t thread_child_mask(F test) {
    uint64_t mask = 0;
    for (int32_t c = 0; c < 64; ++c)
        if (test(c)) mask |= 1ull << c;
    return mask;
}

// tile word + tile LUT from the 64 child bricks (voxel.rs:253-272, :964-972),
// one warp
__device__ __forceinline__ void build_tile(const DevWorld &w, int64_t ti) {
    const Dims &d = w.d;
    const int32_t tx = (int32_t)(ti % d.tx);
    const int32_t ty = (int32_t)((ti / d.tx) % d.ty);
    const int32_t tz = (int32_t)(ti / ((int64_t)d.tx * d.ty));
    const int64_t b0 = (int64_t)(tx * 4) + (int64_t)(ty * 4) * d.bx + (int64_t)(tz * 4) * d.bx * d.by;
    uint32_t u[2];
    uint64_t occ[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int32_t c = (int32_t)(threadIdx.x & 31u) + 32 * h;
        const int64_t bi = b0 + (c & 3) + (int64_t)(c >> 4) * d.bx + (int64_t)((c >> 2) & 3) * d.bx * d.by;
        occ[h] = w.occ[bi];
        u[h] = w.brick_uniform[bi];
    }
    const uint32_t lo = __ballot_sync(0xFFFFFFFFu, occ[0] != 0ull);
    const uint32_t hi = __ballot_sync(0xFFFFFFFFu, occ[1] != 0ull);
    const uint32_t m0 = __shfl_sync(0xFFFFFFFFu, u[0], 0);
    const bool uni = __all_sync(0xFFFFFFFFu, m0 != 0u && u[0] == m0 && u[1] == m0);
    if ((threadIdx.x & 31u) == 0u) {
        w.tile_mask[ti] = (uint64_t)lo | ((uint64_t)hi << 32);
        w.tile_uniform[ti] = uni ? (uint8_t)m0 : 0;
    }
}

// chunk word from its (up to 64) child tiles (voxel.rs:973-981), one warp or
// one thread
template <bool THREAD = false>
__device__ __forceinline__ void build_chunk(const DevWorld &w, int64_t ci) {
    const Dims &d = w.d;
    const int32_t cx = (int32_t)(ci % d.cx);
    const int32_t cy = (int32_t)((ci / d.cx) % d.cy);
    const int32_t cz = (int32_t)(ci / ((int64_t)d.cx * d.cy));
    const auto test = [&](int32_t c) {
        const int32_t tx = cx * 4 + (c & 3), ty = cy * 4 + (c >> 4), tz = cz * 4 + ((c >> 2) & 3);
        return tx < d.tx && ty < d.ty && tz < d.tz &&
               w.tile_mask[tx + (int64_t)ty * d.tx + (int64_t)tz * d.tx * d.ty] != 0ull;
    };
    const uint64_t mask = THREAD ? thread_child_mask(test) : warp_child_mask(test);
    if (THREAD || (threadIdx.x & 31u) == 0u) w.chunk_mask[ci] = mask;
}

// L4 word from its child chunks (voxel.rs:982-990), one warp or one thread
template <bool THREAD = false>
__device__ __forceinline__ void build_l4(const DevWorld &w, int64_t li) {
    const Dims &d = w.d;
    const int32_t x = (int32_t)(li % d.lx);
    const int32_t y = (int32_t)((li / d.lx) % d.ly);
    const int32_t z = (int32_t)(li / ((int64_t)d.lx * d.ly));
    const auto test = [&](int32_t c) {
        const int32_t cx = x * 4 + (c & 3), cy = y * 4 + (c >> 4), cz = z * 4 + ((c >> 2) & 3);
        return cx < d.cx && cy < d.cy && cz < d.cz &&
               w.chunk_mask[cx + (int64_t)cy * d.cx + (int64_t)cz * d.cx * d.cy] != 0ull;
    };
    const uint64_t mask = THREAD ? thread_child_mask(test) : warp_child_mask(test);
    if (THREAD || (threadIdx.x & 31u) == 0u) w.l4_mask[li] = mask;
}

// The same words by one thread each, its 64 loads in turn: fewer instructions
// for each word, enough where there are words to fill the device with.
__device__ __forceinline__ void build_tile_thread(const DevWorld &w, int64_t ti) {
    const Dims &d = w.d;
    const int32_t tx = (int32_t)(ti % d.tx);
    const int32_t ty = (int32_t)((ti / d.tx) % d.ty);
    const int32_t tz = (int32_t)(ti / ((int64_t)d.tx * d.ty));
    uint64_t mask = 0;
    const int64_t b0 = (int64_t)(tx * 4) + (int64_t)(ty * 4) * d.bx + (int64_t)(tz * 4) * d.bx * d.by;
    const uint8_t m0 = w.brick_uniform[b0];
    bool uni = m0 != 0;
    for (int lz = 0; lz < 4; ++lz)
        for (int ly = 0; ly < 4; ++ly)
            for (int lx = 0; lx < 4; ++lx) {
                const int64_t bi = b0 + lx + (int64_t)ly * d.bx + (int64_t)lz * d.bx * d.by;
                if (w.occ[bi] != 0ull) mask |= 1ull << child_bit(lx, ly, lz);
                uni = uni && (w.brick_uniform[bi] == m0);
            }
    w.tile_mask[ti] = mask;
    w.tile_uniform[ti] = uni ? m0 : 0;
}
// Every tile of a large world, one thread each: neighbouring threads read
// neighbouring bricks, so the 64 loads in turn stream the occupancy words
// (2048x256x2048: 27 us for 151 MB, near the copy rate; a warp per tile 57 us,
// bound by its index arithmetic).
__global__ void __launch_bounds__(128) k_build_tiles_stream(DevWorld w) {
    const int64_t ti = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (ti < w.d.n_tiles) build_tile_thread(w, ti);
}
// one warp per cell
__global__ void __launch_bounds__(256) k_build_tiles(DevWorld w) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i < w.d.n_tiles) build_tile(w, i);
}
__global__ void __launch_bounds__(256) k_build_chunks(DevWorld w) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i < w.d.n_chunks) build_chunk(w, i);
}
__global__ void __launch_bounds__(256) k_build_l4(DevWorld w) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i < w.d.n_l4) build_l4(w, i);
}

// ------------------------------------------------------------- dirty
// A 72-byte brick is 8-byte aligned, so it is read in 8-byte words throughout.
__device__ __forceinline__ void scatter_brick(const DevWorld &w, int64_t bi, const VxBrick *b) {
    const uint2 *src = reinterpret_cast<const uint2 *>(b);
    uint2 v[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = src[k];
    const uint64_t occ = (uint64_t)v[0].x | ((uint64_t)v[0].y << 32);
    w.occ[bi] = occ;
    uint4 *dst = reinterpret_cast<uint4 *>(w.mat + bi * 64);
#pragma unroll
    for (int k = 0; k < 4; ++k)
        dst[k] = make_uint4(v[2 * k + 1].x, v[2 * k + 1].y, v[2 * k + 2].x, v[2 * k + 2].y);
    // brick_uniform_of, voxel.rs:233-247
    const uint32_t m0 = v[1].x & 0xFFu, rep = 0x01010101u * m0;
    bool same = occ == ~0ull;
#pragma unroll
    for (int k = 1; k < 9; ++k) same = same && v[k].x == rep && v[k].y == rep;
    w.brick_uniform[bi] = same ? (uint8_t)m0 : 0;
}

// The steps of a dirty-brick update.  Duplicate brick indices in one update,
// last entry wins: each entry claims its brick with its position + 1 (the
// largest wins), only the winner writes, and the claims are cleared again.
// Then each dirty brick re-derives its parent words, one warp per entry;
// warps that share a parent write the same value.  win == nullptr: the
// entries name distinct bricks.
__device__ __forceinline__ void dirty_claim(uint32_t *win, const uint32_t *idx, size_t i) {
    atomicMax(win + idx[i], (uint32_t)(i + 1));
}
__device__ __forceinline__ void dirty_scatter(const DevWorld &w, const uint32_t *win,
                                              const uint32_t *idx, const VxBrick *bricks,
                                              size_t i) {
    const uint32_t bi = idx[i];
    if (win && __ldcg(win + bi) != (uint32_t)(i + 1)) return;
    scatter_brick(w, bi, bricks + i);
}
struct BrickPos {
    int32_t x, y, z;
};
__device__ __forceinline__ BrickPos brick_pos(const Dims &d, int64_t bi) {
    return {(int32_t)(bi % d.bx), (int32_t)((bi / d.bx) % d.by),
            (int32_t)(bi / ((int64_t)d.bx * d.by))};
}
template <bool THREAD = false>
__device__ __forceinline__ void dirty_tile(const DevWorld &w, int64_t bi) {
    const Dims &d = w.d;
    const BrickPos b = brick_pos(d, bi);
    const int64_t ti = (b.x / 4) + (int64_t)(b.y / 4) * d.tx + (int64_t)(b.z / 4) * d.tx * d.ty;
    if (THREAD) build_tile_thread(w, ti);
    else build_tile(w, ti);
}
template <bool THREAD = false>
__device__ __forceinline__ void dirty_chunk(const DevWorld &w, int64_t bi) {
    const Dims &d = w.d;
    const BrickPos b = brick_pos(d, bi);
    build_chunk<THREAD>(w, (b.x / 16) + (int64_t)(b.y / 16) * d.cx + (int64_t)(b.z / 16) * d.cx * d.cy);
}
template <bool THREAD = false>
__device__ __forceinline__ void dirty_l4(const DevWorld &w, int64_t bi) {
    const Dims &d = w.d;
    const BrickPos b = brick_pos(d, bi);
    build_l4<THREAD>(w, (b.x / 64) + (int64_t)(b.y / 64) * d.lx + (int64_t)(b.z / 64) * d.lx * d.ly);
}

// Any number of entries: one launch per step.
__global__ void k_dirty_claim(uint32_t *win, const uint32_t *idx, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dirty_claim(win, idx, i);
}
__global__ void k_dirty_scatter(DevWorld w, const uint32_t *win, const uint32_t *idx,
                                const VxBrick *bricks, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dirty_scatter(w, win, idx, bricks, i);
}
// an entry's words by one warp, or by one thread
template <bool THREAD>
__device__ __forceinline__ size_t dirty_entry() {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    return THREAD ? t : t >> 5;
}
template <bool THREAD>
__global__ void __launch_bounds__(256) k_dirty_tiles(DevWorld w, uint32_t *win,
                                                     const uint32_t *idx, size_t n) {
    const size_t i = dirty_entry<THREAD>();
    if (i >= n) return;
    if (win && (THREAD || (threadIdx.x & 31u) == 0u)) win[idx[i]] = 0u;
    dirty_tile<THREAD>(w, idx[i]);
}
template <bool THREAD>
__global__ void __launch_bounds__(256) k_dirty_chunks(DevWorld w, const uint32_t *idx, size_t n) {
    const size_t i = dirty_entry<THREAD>();
    if (i < n) dirty_chunk<THREAD>(w, idx[i]);
}
template <bool THREAD>
__global__ void __launch_bounds__(256) k_dirty_l4(DevWorld w, const uint32_t *idx, size_t n) {
    const size_t i = dirty_entry<THREAD>();
    if (i < n) dirty_l4<THREAD>(w, idx[i]);
}

// A frame's worth of entries: the same steps in one launch of one cluster,
// its barrier between them.  Each step is a round or two of memory latency:
// 175 entries take 20 us, cold, against 71 us for six launches of one thread
// per entry, most of it the 64 loads in turn and the starts and drains.  The
// cluster's 128 warps take a round for every 128 entries, and each level's
// rounds follow one another.  Whole update, us, cluster / launches of a warp
// per word: 32 entries 36 / 44, 175 42 / 45, 256 43 / 46, 512 54 / 49, 1,000
// 69 / 52.
constexpr uint32_t kDirtyCtas = 8, kDirtyThreads = 512;
constexpr uint32_t kDirtyClusterMax = 384;    // entries: three rounds

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;"
                 ::: "memory");
}

__global__ void __cluster_dims__(kDirtyCtas, 1, 1) __launch_bounds__(kDirtyThreads)
    k_dirty_cluster(DevWorld w, uint32_t *win, const uint32_t *idx, const VxBrick *bricks,
                    uint32_t n) {
    const uint32_t t = blockIdx.x * kDirtyThreads + threadIdx.x, warp = t >> 5;
    constexpr uint32_t threads = kDirtyCtas * kDirtyThreads, warps = threads / 32u;
    if (win) {
        for (uint32_t i = t; i < n; i += threads) dirty_claim(win, idx, i);
        cluster_barrier();
    }
    for (uint32_t i = t; i < n; i += threads) dirty_scatter(w, win, idx, bricks, i);
    cluster_barrier();
    if (win)
        for (uint32_t i = t; i < n; i += threads) win[idx[i]] = 0u;
    for (uint32_t i = warp; i < n; i += warps) dirty_tile(w, idx[i]);
    cluster_barrier();
    for (uint32_t i = warp; i < n; i += warps) dirty_chunk(w, idx[i]);
    cluster_barrier();
    for (uint32_t i = warp; i < n; i += warps) dirty_l4(w, idx[i]);
}

// Persistent edits (apply_edit / replay_edits_for_chunk, voxel.rs:448-474,
// :571-603): edit i sets voxel (ed[i].y & 63) of brick ed[i].x to material
// ed[i].y >> 8, Brick::set semantics (voxel.rs:315-325: material 0 clears the
// occupancy bit).  The edits of one batch name distinct voxels; several may
// share a brick, so the occupancy word is updated atomically.
__global__ void k_edit_voxels(DevWorld w, const uint2 *__restrict__ ed, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint2 e = ed[i];
    const uint32_t vi = e.y & 63u, mat = e.y >> 8;
    w.mat[(size_t)e.x * 64u + vi] = (uint8_t)mat;
    unsigned long long *occ = reinterpret_cast<unsigned long long *>(w.occ + e.x);
    if (mat != 0u) atomicOr(occ, 1ull << vi);
    else atomicAnd(occ, ~(1ull << vi));
}
// the uniform byte of each edited brick, once all its voxels are written
__global__ void k_edit_uniform(DevWorld w, const uint32_t *__restrict__ idx, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t bi = idx[i];
    w.brick_uniform[bi] = uniform_of(w.occ[bi], w.mat + bi * 64);
}

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }
// CTAs of 256 threads for one warp per item
inline unsigned warp_blocks(int64_t n) { return (unsigned)((n + 7) / 8); }

// The parent words of n dirty bricks: a warp to a word while the entries are too
// few to fill the device with one thread each, whose 64 loads in turn are a few
// times the instructions cheaper.  Whole update, us, warp / thread: 8,000
// entries 98-103 / 118, 16,000 167 / 175, 32,000 294 / 284, 50,000 419 / 384,
// 200,000 1531 / 1343.
constexpr size_t kDirtyWarpMax = 20000;
template <bool THREAD>
void dirty_parents_by(const DevWorld &w, uint32_t *win, const uint32_t *idx, size_t n,
                      cudaStream_t s) {
    const unsigned b = THREAD ? blocks_for((int64_t)n, 256) : warp_blocks((int64_t)n);
    k_dirty_tiles<THREAD><<<b, 256, 0, s>>>(w, win, idx, n);
    k_dirty_chunks<THREAD><<<b, 256, 0, s>>>(w, idx, n);
    k_dirty_l4<THREAD><<<b, 256, 0, s>>>(w, idx, n);
}
void dirty_parents(const DevWorld &w, uint32_t *win, const uint32_t *idx, size_t n,
                   cudaStream_t s) {
    if (n > kDirtyWarpMax) dirty_parents_by<true>(w, win, idx, n, s);
    else dirty_parents_by<false>(w, win, idx, n, s);
}

}  // namespace

cudaError_t launch_edits(const DevWorld &w, const uint2 *ed, size_t n_edits, const uint32_t *idx,
                         size_t n_bricks, cudaStream_t s) {
    if (n_edits == 0) return cudaSuccess;
    k_edit_voxels<<<blocks_for((int64_t)n_edits, 128), 128, 0, s>>>(w, ed, n_edits);
    const unsigned b = blocks_for((int64_t)n_bricks, 128);
    k_edit_uniform<<<b, 128, 0, s>>>(w, idx, n_bricks);
    dirty_parents(w, nullptr, idx, n_bricks, s);
    return launch_tile_meta(w, s);
}

cudaError_t launch_bricks_from_aos(const DevWorld &w, const VxBrick *aos, int64_t first,
                                   int64_t count, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    k_aos_to_soa<<<blocks_for(count, 256), 256, 0, s>>>(w, aos, first, count);
    return cudaGetLastError();
}

cudaError_t launch_bricks_to_aos(const DevWorld &w, VxBrick *aos, int64_t first, int64_t count,
                                 cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    k_soa_to_aos<<<blocks_for(count, 256), 256, 0, s>>>(w, aos, first, count);
    return cudaGetLastError();
}

cudaError_t launch_rebuild_pyramid(const DevWorld &w, bool tiles, cudaStream_t s) {
    // one thread per tile needs enough tiles to hide its chain of loads
    // (16,384 tiles: 17 us against 8 us for a warp each)
    if (tiles && w.d.n_tiles > 65536)
        k_build_tiles_stream<<<blocks_for(w.d.n_tiles, 128), 128, 0, s>>>(w);
    else if (tiles)
        k_build_tiles<<<warp_blocks(w.d.n_tiles), 256, 0, s>>>(w);
    k_build_chunks<<<warp_blocks(w.d.n_chunks), 256, 0, s>>>(w);
    k_build_l4<<<warp_blocks(w.d.n_l4), 256, 0, s>>>(w);
    return launch_tile_meta(w, s);
}



cudaError_t launch_generate(const DevWorld &w, const VxTerrainParams &t, int16_t *heights,
                            cudaStream_t s) {
    GenArgs g;
    g.w = w;
    g.t = t;
    // seed_offset_xz, voxel.rs:1163-1167 (same float ops as the device would do)
    const float hi = (float)(int32_t)(uint32_t)(t.seed >> 32);
    const float lo = (float)(int32_t)(uint32_t)(t.seed & 0xFFFFFFFFull);
    g.off_x = hi * 0.01734f;
    g.off_z = lo * 0.02153f;
    g.heights = heights;
    k_heights<<<blocks_for((int64_t)w.d.vx * w.d.vz, 256), 256, 0, s>>>(g);
    k_gen_bricks<<<blocks_for(w.d.n_bricks, 128), 128, 0, s>>>(g);
    return launch_rebuild_pyramid(w, true, s);
}

// win: a claim word per brick, zero between updates (the last of an update's
// entries for one brick wins), or nullptr when the entries are distinct
static cudaError_t apply_dirty(const DevWorld &w, uint32_t *win, const uint32_t *idx,
                               const VxBrick *bricks, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (n <= kDirtyClusterMax) {
        k_dirty_cluster<<<kDirtyCtas, kDirtyThreads, 0, s>>>(w, win, idx, bricks, (uint32_t)n);
        return launch_tile_meta(w, s);
    }
    const unsigned b = blocks_for((int64_t)n, 128);
    if (win) k_dirty_claim<<<b, 128, 0, s>>>(win, idx, n);
    k_dirty_scatter<<<b, 128, 0, s>>>(w, win, idx, bricks, n);
    dirty_parents(w, win, idx, n, s);
    return launch_tile_meta(w, s);
}

cudaError_t launch_apply_dirty_last_wins(const DevWorld &w, uint32_t *win, const uint32_t *idx,
                                         const VxBrick *bricks, size_t n, cudaStream_t s) {
    return apply_dirty(w, win, idx, bricks, n, s);
}

cudaError_t launch_apply_dirty(const DevWorld &w, const uint32_t *idx, const VxBrick *bricks,
                               size_t n, cudaStream_t s) {
    return apply_dirty(w, nullptr, idx, bricks, n, s);
}

}  // namespace vx
