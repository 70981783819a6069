// vx_slotgen.cu -- the reference's storage-chunk generator gen_slot_bricks
// (src/voxel.rs:1322-1500) on the device: terrain columns, biomes, ores,
// surface decoration and the branched trees of the chunk and its eight xz
// neighbours, written straight into the world's toroidal slots.  Compiled
// with --fmad=false so every binary32 operation rounds as the CPU's does.
//
// The reference recomputes, for every storage chunk, the terrain of its
// 32x32 columns and the trees of its 3x3 neighbourhood.  Both depend only on
// x and z, so a batch of chunks is generated by two kernels:
//   k_gen_xz       one thread per column of each distinct xz chunk --
//                  sample_terrain (:1244-1316), the biome (:1342-1344) and
//                  the surface decoration (:1394-1459) packed in one word --
//                  and one thread per tree candidate of each distinct source
//                  chunk (trees_for_chunk, :1537-1591), expanded into its
//                  paint primitives (paint_tree, :1605-1710);
//   k_gen_slot     one 256-thread CTA per storage chunk, three per SM: the
//                  voxels of its columns in shared memory (ore noise from
//                  tables of the chunk's lattice hashes), then the
//                  primitives of the 3x3 source chunks in the reference's
//                  order -- source chunk (z, x), tree, primitive.  Each warp
//                  paints a slab of four z levels by itself: it takes the
//                  primitives that reach the slab in order, and every write
//                  of one primitive carries one material, so the order among
//                  its voxels cannot change what try_write_tree_voxel
//                  (:1500-1525) leaves.  Last the 512 bricks, their occupancy
//                  words (occupancy == material != 0, the invariant
//                  Brick::set keeps, :315-325) and uniform bytes go to the
//                  slot's bricks, and the chunk's eight tile words and LUT
//                  bytes with them.
// What bounds k_gen_slot: the ore noise of the voxels below ground (two value
// noises each) and, before, the walk over the trees.  For a window of
// 2048x256x2048 moved by (8, 3) chunks, 5,440 of them: 630-700 us with the
// noise hashed column by column (526 M warp instructions), all 256 threads on
// one primitive at a time behind a barrier and the 108 tree headers read one
// after the other; 620 us with the lattice tables, 455 us with the slabs,
// 392 us with the chunks below ground started first (288 M); 355 us with a
// tree's four levels of a slab painted at once, 350 us with two columns' noise
// in one loop (three CTAs of 80 registers; 438 us with four of 64, which
// spill in it), 325 us with the two columns in packed arithmetic (207 M).
// All-air chunks only write, and caves read tables like the ores (302 M -> 275).
// powf, cosf and sinf give the host C library's binary32 results, as the
// reference's f32::powf / cos / sin do: vx_gmath.h's functions, corrected
// by the exception table (Seed::lmx) on the generator's domains.
#include <cuda_runtime.h>

#include "vx_gmath.h"
#include "vx_internal.h"
#include "vx_noise.cuh"

namespace vx {
namespace {

using noise::fbm_2d;
using noise::hash3;
using noise::value_noise_3d;

constexpr int kCV = 32;          // STORAGE_CHUNK_VOXELS
constexpr int kSea = 64;         // sea_level
constexpr int kWorldY = 256;     // WORLD_VOXELS_Y the generator is written for
constexpr int kCand = 12;        // trees_for_chunk yields at most round(1.2*5)*2
constexpr int kTrees = 9 * kCand;
constexpr int kPrims = 16;       // primitives of one tree (oak: 1 + 4*3 + 2)

enum : uint8_t {
    M_SAND = 1, M_GRASS = 2, M_DIRT = 3, M_STONE = 4, M_WATER = 12, M_WOOD = 13,
    M_LEAVES = 14, M_SNOW = 15, M_COAL = 19, M_IRON = 20, M_GOLD = 21, M_DIAMOND = 22,
    M_WOOD_BIRCH = 23, M_WOOD_PINE = 24, M_LEAVES_BIRCH = 25, M_LEAVES_PINE = 26,
    M_LEAVES_AUTUMN = 27, M_FLOWER = 30, M_TALL_GRASS = 31, M_CACTUS = 32, M_FRINGE = 33,
    M_GRASS_DRY = 34, M_BUSH = 36
};
enum { B_TUNDRA, B_PLAINS, B_FOREST, B_JUNGLE, B_SAVANNA, B_DESERT, B_BEACH, B_MOUNTAIN };

__device__ __forceinline__ int32_t f2i(float x) {
    if (x != x) return 0;
    if (x >= 1073741824.0f) return 1073741824;
    if (x <= -1073741824.0f) return -1073741824;
    return (int32_t)x;
}
__device__ __forceinline__ float fmaxr(float a, float b) { return a < b ? b : a; }
__device__ __forceinline__ float fminr(float a, float b) { return b < a ? b : a; }
// the C library's powf(x, 1.15f), powf(x, 0.85f), cosf, sinf (vx_gmath.h)
__device__ __forceinline__ float pow115(const uint32_t *lmx, float x) {
    return gm::lmx_fix(lmx, gm::LMX_POW115, x, gm::pow01(x, 1.15f));
}
__device__ __forceinline__ float pow085(const uint32_t *lmx, float x) {
    return gm::lmx_fix(lmx, gm::LMX_POW085, x, gm::pow01(x, 0.85f));
}
__device__ __forceinline__ float cos_f(const uint32_t *lmx, float a) {
    return gm::lmx_fix(lmx, gm::LMX_COS, a, gm::cos_small(a));
}
__device__ __forceinline__ float sin_f(const uint32_t *lmx, float a) {
    return gm::lmx_fix(lmx, gm::LMX_SIN, a, gm::sin_small(a));
}

struct Seed {
    uint64_t seed;
    float offx, offz;      // seed_offset_xz, voxel.rs:1163-1167
    const uint32_t *lmx;   // exception table of vx_gmath.h (device copy)
};

// sample_terrain, voxel.rs:1244-1316 (ravine cut 0, rivers off)
__device__ int32_t sample_terrain(float wx, float wz, float offx, float offz, const uint32_t *lmx,
                                  int32_t *water_top) {
    const float px = wx + offx, pz = wz + offz;
    const float warp_x = fbm_2d(px * 0.005f, pz * 0.005f, 2) * 8.0f;
    const float warp_z = fbm_2d(px * 0.005f + 50.0f, pz * 0.005f + 50.0f, 2) * 8.0f;
    const float wpx = px + warp_x, wpz = pz + warp_z;
    const float base = fbm_2d(wpx * 0.012f, wpz * 0.012f, 4) * 22.0f;
    const float mountain_mask = fmaxr(fbm_2d(wpx * 0.0028f, wpz * 0.0028f, 2) + 0.2f, 0.0f);
    const float mountain_amp = fminr(mountain_mask, 1.0f);
    // both factors are finite and not negative, so a zero one makes the
    // product +0 whatever the other is
    float mountain_h = 0.0f;
    if (mountain_amp > 0.0f) {
        const float m = fmaxr(fbm_2d(wpx * 0.009f, wpz * 0.009f, 5), 0.0f);
        if (m > 0.0f) mountain_h = pow115(lmx, m) * mountain_amp * 110.0f;
    }
    const float base_h = 64.0f + 8.0f + base + mountain_h - 0.0f;
    const float h = base_h < 2.0f ? 2.0f : (base_h > 255.0f ? 255.0f : base_h);
    const int32_t hi = f2i(h);
    *water_top = hi < kSea ? kSea : 0;
    return hi;
}

// pick_biome and the Biome tables, voxel.rs:1822-1903
__device__ __forceinline__ int pick_biome(float temp, float humid, uint32_t h) {
    if (h > kSea + 36) return B_MOUNTAIN;
    if (h <= kSea + 1) return B_BEACH;
    if (temp < -0.20f) return B_TUNDRA;
    if (temp > 0.25f && humid < -0.05f) return B_DESERT;
    if (temp > 0.15f && humid > 0.25f) return B_JUNGLE;
    if (temp > 0.10f && humid < 0.10f) return B_SAVANNA;
    if (humid > 0.20f) return B_FOREST;
    return B_PLAINS;
}
__device__ __forceinline__ uint8_t top_block(int b, uint32_t h) {
    if (b == B_TUNDRA) return M_SNOW;
    if (b == B_DESERT || b == B_BEACH || b == B_SAVANNA) return M_SAND;
    if (b == B_MOUNTAIN) return h > kSea + 55 ? M_SNOW : M_STONE;
    return M_GRASS;
}
__device__ __forceinline__ uint8_t subsoil(int b) {
    if (b == B_DESERT || b == B_BEACH) return M_SAND;
    if (b == B_MOUNTAIN) return M_STONE;
    return M_DIRT;
}
__device__ __forceinline__ uint32_t tree_type(int b, uint32_t hash) {
    if (b == B_TUNDRA || b == B_MOUNTAIN) return 2;
    if (b == B_PLAINS) return hash % 3 == 0 ? 1 : 0;
    if (b == B_FOREST) {
        const uint32_t k = hash % 4;
        return k == 0 ? 1 : (k == 1 ? 3 : 0);
    }
    if (b == B_JUNGLE) return hash % 4 == 0 ? 3 : 0;
    return 0;
}
__device__ __forceinline__ float tree_density(int b) {
    switch (b) {
    case B_JUNGLE: return 1.2f;
    case B_FOREST: return 0.55f;
    case B_TUNDRA: return 0.30f;
    case B_PLAINS: return 0.20f;
    case B_MOUNTAIN: return 0.14f;
    case B_DESERT: return 0.20f;
    default: return 0.0f;
    }
}

// shared-memory chunk: brick (x + y*8 + z*64) * 64 + x + z*4 + y*16
__device__ __forceinline__ uint32_t vox(uint32_t dx, uint32_t dy, uint32_t dz) {
    return (((dx >> 2) + (dy >> 2) * 8u + (dz >> 2) * 64u) << 6) +
           ((dx & 3u) + (dz & 3u) * 4u + (dy & 3u) * 16u);
}

// ------------------------------------------------------------------ trees
struct Tree {
    int32_t x, y, z;
    uint32_t ttype, hash;
};

// candidate i of trees_for_chunk(cx, cz) (voxel.rs:1537-1591); false when
// the reference's loop yields no tree for it
__device__ bool tree_candidate(int32_t cx, int32_t cz, uint32_t i, const Seed &g, Tree &t) {
    const float ccx = ((float)cx + 0.5f) * 32.0f, ccz = ((float)cz + 0.5f) * 32.0f;
    const float temperature = fbm_2d((ccx + g.offx) * 0.0006f, (ccz + g.offz) * 0.0006f, 3);
    const float humidity =
        fbm_2d((ccx + g.offx) * 0.0008f + 100.0f, (ccz + g.offz) * 0.0008f + 100.0f, 3);
    const int biome = pick_biome(temperature, humidity, kSea + 10);
    const uint32_t n_cand = (uint32_t)f2i(roundf(tree_density(biome) * 5.0f));
    if (i >= n_cand * 2u) return false;  // n <= n_cand * patch_mul <= 2 n_cand
    float patch_mul = 1.0f;
    if (biome != B_DESERT) {
        const float patch_raw = fbm_2d(ccx * 0.0035f, ccz * 0.0035f, 2);
        patch_mul = fminr(fmaxr(patch_raw + 0.4f, 0.0f) * 1.6f, 2.0f);
    }
    const uint32_t n = (uint32_t)f2i((float)n_cand * patch_mul);
    if (i >= n) return false;
    // hash_chunk, voxel.rs:1593-1601
    const uint32_t s = (uint32_t)g.seed ^ (uint32_t)(g.seed >> 32);
    uint32_t ch = (uint32_t)cx * 0x9E3779B1u;
    ch = ch + (uint32_t)cz * 0x85EBCA77u;
    ch = ch + s * 0xC2B2AE3Du;
    ch = ch ^ (ch >> 16);
    ch = ch * 0xD2B74407u;
    ch = ch ^ (ch >> 13);
    const uint32_t h = ch * 2654435761u + i * 7919u;
    const int32_t wx = cx * kCV + (int32_t)(h & 31u), wz = cz * kCV + (int32_t)((h >> 5) & 31u);
    int32_t wt;
    const int32_t th = sample_terrain((float)wx, (float)wz, g.offx, g.offz, g.lmx, &wt);
    if ((uint32_t)th <= (uint32_t)(kSea + 1)) return false;
    if (th + 22 >= kWorldY) return false;
    const float lt = fbm_2d(((float)wx + g.offx) * 0.0006f, ((float)wz + g.offz) * 0.0006f, 3);
    const float lh = fbm_2d(((float)wx + g.offx) * 0.0008f + 100.0f,
                            ((float)wz + g.offz) * 0.0008f + 100.0f, 3);
    const int lb = pick_biome(lt, lh, (uint32_t)th);
    if (lb == B_BEACH || lb == B_SAVANNA) return false;
    t.x = wx; t.y = th + 1; t.z = wz;
    t.ttype = lb == B_DESERT ? 4u : tree_type(lb, h);
    t.hash = h;
    return true;
}

enum : uint32_t { PR_LINE = 0, PR_SHELL = 1, PR_SPHERE = 2 };
struct __align__(16) Prim {
    int32_t a[3];    // line start / shell or sphere centre
    int32_t b[3];    // line end; b[0] = radius of a shell or sphere
    uint32_t kind_mat;
    int32_t steps;   // line: ceil(len * 1.5)
};

// Appends a tree's primitives in paint_tree order.
struct Emit {
    Prim *out;
    int n;
    // paint_line with thickness 0, voxel.rs:1744-1776
    __device__ void line(int32_t ax, int32_t ay, int32_t az, int32_t bx, int32_t by, int32_t bz,
                         uint8_t mat) {
        const int32_t d0 = bx - ax, d1 = by - ay, d2 = bz - az;
        const float len = sqrtf((float)(d0 * d0 + d1 * d1 + d2 * d2));
        Prim &p = out[n++];
        p.a[0] = ax; p.a[1] = ay; p.a[2] = az;
        p.b[0] = bx; p.b[1] = by; p.b[2] = bz;
        p.kind_mat = (PR_LINE << 8) | mat;
        p.steps = f2i(ceilf(len * 1.5f));
    }
    // paint_fringe_shell(c, r + 1) then paint_sphere(c, r): paint_canopy,
    // voxel.rs:1715-1742, :1778-1789
    __device__ void canopy(int32_t cx, int32_t cy, int32_t cz, int32_t r, uint8_t mat) {
        Prim &f = out[n++];
        f.a[0] = cx; f.a[1] = cy; f.a[2] = cz;
        f.b[0] = r + 1; f.b[1] = f.b[2] = 0;
        f.kind_mat = (PR_SHELL << 8) | M_FRINGE;
        f.steps = 0;
        Prim &p = out[n++];
        p.a[0] = cx; p.a[1] = cy; p.a[2] = cz;
        p.b[0] = r; p.b[1] = p.b[2] = 0;
        p.kind_mat = (PR_SPHERE << 8) | mat;
        p.steps = 0;
    }
};

// The box of the voxels a primitive can write: its segment (rounding a + d t
// with t in [0, 1] stays between the ends), c +- (r + 1, r, r + 1) for a
// shell, c +- r for a sphere.
__device__ __forceinline__ void prim_box(const Prim &p, int32_t mn[3], int32_t mx[3]) {
    const uint32_t kind = p.kind_mat >> 8;
    if (kind == PR_LINE) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            mn[k] = min(p.a[k], p.b[k]);
            mx[k] = max(p.a[k], p.b[k]);
        }
    } else {
        const int32_t r = p.b[0], rh = kind == PR_SHELL ? r + 1 : r;
        mn[0] = p.a[0] - rh; mx[0] = p.a[0] + rh;
        mn[1] = p.a[1] - r;  mx[1] = p.a[1] + r;
        mn[2] = p.a[2] - rh; mx[2] = p.a[2] + rh;
    }
}
// A tree's voxels lie within kTreeReach of its base in x and z: the longest
// branch (5) and the shell of a branch canopy (radius 3 + 1, widened by 1);
// pine canopies reach 4 + 1 + 1, cactus arms 2.
constexpr int32_t kTreeReach = 10;

// branch_jitter, voxel.rs:1791-1797
__device__ __forceinline__ float branch_jitter(uint32_t hash, uint32_t b) {
    const uint32_t h = hash * 0x9E3779B1u + b * 2654435761u;
    return ((float)(h & 0xFFFFu) / 65535.0f) * 2.0f - 1.0f;
}

// paint_tree, voxel.rs:1605-1710
__device__ void tree_prims(const Tree &t, const uint32_t *lmx, Emit &e) {
    const float tau = 6.28318548202514648f;  // std::f32::consts::TAU
    const uint32_t h = t.hash;
    if (t.ttype == 2) {
        const int32_t trunk_h = 10 + (int32_t)(h % 6);
        e.line(t.x, t.y, t.z, t.x, t.y + trunk_h, t.z, M_WOOD_PINE);
        for (int32_t i = 0; i < 6; ++i) {
            const float tf = (float)i / 6.0f;
            const int32_t y = t.y + f2i((float)trunk_h * (0.35f + tf * 0.78f));
            const int32_t r = f2i(pow085(lmx, 1.0f - tf) * 3.5f + 1.0f);
            e.canopy(t.x, y, t.z, r, M_LEAVES_PINE);
        }
    } else if (t.ttype == 1) {
        const int32_t trunk_h = 8 + (int32_t)(h % 5);
        e.line(t.x, t.y, t.z, t.x, t.y + trunk_h, t.z, M_WOOD_BIRCH);
        const int32_t n = 2 + (int32_t)(h % 2);
        for (int32_t b = 0; b < n; ++b) {
            const float angle = ((float)b / (float)n) * tau + branch_jitter(h, (uint32_t)b) * 0.5f;
            const int32_t len = 2 + (int32_t)((h * ((uint32_t)b + 1u)) % 3u);
            const int32_t sy = t.y + f2i((float)trunk_h * 0.7f);
            const int32_t ex = t.x + f2i(cos_f(lmx, angle) * (float)len);
            const int32_t ez = t.z + f2i(sin_f(lmx, angle) * (float)len);
            e.line(t.x, sy, t.z, ex, sy + 1, ez, M_WOOD_BIRCH);
            e.canopy(ex, sy + 1, ez, 2, M_LEAVES_BIRCH);
        }
        e.canopy(t.x, t.y + trunk_h, t.z, 3, M_LEAVES_BIRCH);
    } else if (t.ttype == 4) {
        // arm directions per h & 3: [(1,0),(0,1)] [(-1,0),(0,-1)] [(0,1),(-1,0)] [(0,-1),(1,0)]
        const int32_t sets[4][2][2] = {{{1, 0}, {0, 1}}, {{-1, 0}, {0, -1}},
                                       {{0, 1}, {-1, 0}}, {{0, -1}, {1, 0}}};
        const int32_t col_h = 3 + (int32_t)(h % 6);
        e.line(t.x, t.y, t.z, t.x, t.y + col_h, t.z, M_CACTUS);
        const int32_t n_arms = (int32_t)(h % 3);
        const uint32_t si = h & 3u;
        for (int32_t a = 0; a < n_arms; ++a) {
            const int32_t dx = sets[si][a % 2][0], dz = sets[si][a % 2][1];
            const int32_t sy = t.y + f2i((float)col_h * 0.4f);
            const int32_t arm_top = t.y + f2i((float)col_h * 0.9f);
            const int32_t ax = t.x + dx * 2, az = t.z + dz * 2;
            e.line(t.x, sy, t.z, ax, sy, az, M_CACTUS);
            e.line(ax, sy, az, ax, arm_top, az, M_CACTUS);
        }
    } else {
        const uint8_t leaf = t.ttype == 3 ? M_LEAVES_AUTUMN : M_LEAVES;
        const int32_t trunk_h = 8 + (int32_t)(h % 5);
        e.line(t.x, t.y, t.z, t.x, t.y + trunk_h, t.z, M_WOOD);
        const int32_t n = 3 + (int32_t)(h % 2);
        for (int32_t b = 0; b < n; ++b) {
            const float angle = ((float)b / (float)n) * tau + branch_jitter(h, (uint32_t)b) * 0.6f;
            const int32_t len = 3 + (int32_t)((h * ((uint32_t)b + 7u)) % 3u);
            const int32_t sy = t.y + f2i((float)trunk_h * 0.65f);
            const int32_t ex = t.x + f2i(cos_f(lmx, angle) * (float)len);
            const int32_t ey = sy + f2i((float)len * 0.5f);
            const int32_t ez = t.z + f2i(sin_f(lmx, angle) * (float)len);
            e.line(t.x, sy, t.z, ex, ey, ez, M_WOOD);
            e.canopy(ex, ey, ez, 3, leaf);
        }
        e.canopy(t.x, t.y + trunk_h, t.z, 4, leaf);
    }
}

// try_write_tree_voxel, voxel.rs:1500-1525, on the shared chunk; (x, y, z)
// inside it
__device__ __forceinline__ void tree_voxel(uint8_t *s_mat, uint32_t dx, uint32_t dy, uint32_t dz,
                                           uint8_t mat) {
    const uint32_t v = vox(dx, dy, dz);
    const uint8_t cur = s_mat[v];
    if (cur == 0 || (cur == M_FRINGE && mat != M_FRINGE)) s_mat[v] = mat;
}

// One warp paints a primitive's voxels in the slab [zlo, zhi = zlo + 4) of the
// chunk at lo (any order: one primitive writes one material).
__device__ __forceinline__ void paint_prim(uint8_t *s_mat, const int32_t lo[3], int32_t zlo,
                                           int32_t zhi, const Prim &p) {
    const uint32_t kind = p.kind_mat >> 8;
    const uint8_t mat = (uint8_t)(p.kind_mat & 0xFFu);
    const int32_t lane = (int32_t)(threadIdx.x & 31u);
    if (kind == PR_LINE) {
        const int32_t d0 = p.b[0] - p.a[0], d1 = p.b[1] - p.a[1], d2 = p.b[2] - p.a[2];
        const int32_t steps = max(p.steps, 0);     // no steps: the point a
        for (int32_t s = lane; s <= steps; s += 32) {
            const float t = steps > 0 ? (float)s / (float)steps : 0.0f;
            const int32_t x = f2i(roundf((float)p.a[0] + (float)d0 * t));
            const int32_t y = f2i(roundf((float)p.a[1] + (float)d1 * t));
            const int32_t z = f2i(roundf((float)p.a[2] + (float)d2 * t));
            if ((uint32_t)(x - lo[0]) < (uint32_t)kCV && (uint32_t)(y - lo[1]) < (uint32_t)kCV &&
                z >= zlo && z < zhi)
                tree_voxel(s_mat, (uint32_t)(x - lo[0]), (uint32_t)(y - lo[1]),
                           (uint32_t)(z - lo[2]), mat);
        }
        return;
    }
    // shell: max(|dx| - 1, 0)^2 + dy^2 + max(|dz| - 1, 0)^2 <= r^2; sphere
    // without the widening.  Two rows of 16 voxels a round.
    const int32_t wide = kind == PR_SHELL ? 1 : 0, r = p.b[0], r2 = r * r;
    const int32_t ya = max(p.a[1] - r, lo[1]), yb = min(p.a[1] + r, lo[1] + kCV - 1);
    // the slab's four levels at once (they lie in one brick layer), so the
    // reads of a row do not wait for the writes of the level before
    int32_t hz2[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int32_t hz = max(abs(zlo + k - p.a[2]) - wide, 0);
        hz2[k] = hz * hz;
    }
    for (int32_t y = ya + (lane >> 4); y <= yb; y += 2) {
        const int32_t dy = y - p.a[1], rest_y = r2 - dy * dy;
        for (int32_t dx = (lane & 15) - r - wide; dx <= r + wide; dx += 16) {
            const int32_t hx = max(abs(dx) - wide, 0), rest = rest_y - hx * hx;
            const uint32_t x = (uint32_t)(p.a[0] + dx - lo[0]);
            if (rest < 0 || x >= (uint32_t)kCV) continue;
            uint8_t *v = s_mat + vox(x, (uint32_t)(y - lo[1]), (uint32_t)(zlo - lo[2]));
            uint8_t cur[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) cur[k] = v[4 * k];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (hz2[k] <= rest && (cur[k] == 0 || (cur[k] == M_FRINGE && mat != M_FRINGE)))
                    v[4 * k] = mat;
        }
    }
}

// ------------------------------------------------------------------ columns
// Column word: bits 0-7 h, 8 water (water_top = sea level), 9-11 biome,
// 12-17 decoration material (0: none), 18 the decoration is a big bush.
// pos_mod(a, n), n > 0
__device__ __forceinline__ int32_t wrap(int32_t a, int32_t n) { return ((a % n) + n) % n; }

// The world chunk (x, z) of column chunk k / source chunk k of a plan.
__device__ __forceinline__ void col_chunk(const GenPlan &p, const Dims &d, uint32_t k,
                                          int32_t &cx, int32_t &cz) {
    if (p.window) {
        const int32_t sxn = d.bx / 8, szn = d.bz / 8;
        const int32_t sx = (int32_t)k % sxn, sz = (int32_t)k / sxn;
        cx = p.ox + wrap(sx - p.ox, sxn);
        cz = p.oz + wrap(sz - p.oz, szn);
    } else {
        cx = p.cols[2 * k];
        cz = p.cols[2 * k + 1];
    }
}
__device__ __forceinline__ void src_chunk(const GenPlan &p, const Dims &d, uint32_t k,
                                          int32_t &cx, int32_t &cz) {
    if (p.window) {
        const int32_t w = d.bx / 8 + 2;
        cx = p.ox - 1 + (int32_t)k % w;
        cz = p.oz - 1 + (int32_t)k / w;
    } else {
        cx = p.srcs[2 * k];
        cz = p.srcs[2 * k + 1];
    }
}

__device__ void gen_column(const GenPlan &p, const Dims &d, const Seed &g, uint32_t c) {
    if (c >= p.n_cols * (uint32_t)(kCV * kCV)) return;
    const uint32_t k = c >> 10, col = c & 1023u;
    int32_t ccx, ccz;
    col_chunk(p, d, k, ccx, ccz);
    const int32_t wxi = ccx * kCV + (int32_t)(col & 31u);
    const int32_t wzi = ccz * kCV + (int32_t)(col >> 5);
    const float wx = (float)wxi, wz = (float)wzi;
    int32_t water_top;
    const int32_t h = sample_terrain(wx, wz, g.offx, g.offz, g.lmx, &water_top);
    const uint32_t hu = (uint32_t)h;
    const float temperature = fbm_2d((wx + g.offx) * 0.0006f, (wz + g.offz) * 0.0006f, 3);
    const float humidity =
        fbm_2d((wx + g.offx) * 0.0008f + 100.0f, (wz + g.offz) * 0.0008f + 100.0f, 3);
    const int biome = pick_biome(temperature, humidity, hu);
    uint32_t dec = 0, big = 0;
    if (water_top == 0 && hu < (uint32_t)(kWorldY - 1)) {
        const uint8_t surface = top_block(biome, hu);
        const int32_t dec_y = h + 1;
        const float v = hash3(wxi, dec_y, wzi) * 0.5f + 0.5f;
        const bool big_lattice = hash3(wxi & ~1, 977, wzi & ~1) * 0.5f + 0.5f > 0.9955f;
        if (surface == M_GRASS) {
            float fp, gp;
            if (biome == B_PLAINS) { fp = 0.020f; gp = 0.08f; }
            else if (biome == B_FOREST) { fp = 0.010f; gp = 0.065f; }
            else if (biome == B_JUNGLE) { fp = 0.012f; gp = 0.09f; }
            else { fp = 0.015f; gp = 0.065f; }
            if (fbm_2d((float)wxi * 0.02f + 7.0f, (float)wzi * 0.02f - 3.0f, 2) > 0.30f) {
                fp *= 3.0f;
                gp *= 12.0f;
            }
            if (v > 1.0f - fp) dec = M_FLOWER;
            else if (v > 1.0f - fp - gp) dec = M_TALL_GRASS;
            else if (big_lattice) dec = M_BUSH;
            else if (v > 1.0f - fp - gp - 0.004f) dec = M_BUSH;
        } else if (surface == M_SAND && (biome == B_DESERT || biome == B_SAVANNA)) {
            if (v > 0.99f) dec = M_GRASS_DRY;
        } else if (surface == M_SNOW && biome == B_TUNDRA) {
            if (v > 0.995f) dec = M_GRASS_DRY;
        }
        big = (dec == M_BUSH && big_lattice) ? 1u : 0u;
    }
    p.colw[c] = hu | ((water_top != 0 ? 1u : 0u) << 8) | ((uint32_t)biome << 9) | (dec << 12) |
             (big << 18);
}

// ------------------------------------------------------------------ trees
// Per source chunk: kCand headers (primitive count | x in the chunk << 8 |
// z << 13 | base y << 18; 0 when the candidate yields no tree) and kCand x
// kPrims primitives.
__device__ void gen_tree(const GenPlan &p, const Dims &d, const Seed &g, uint32_t c) {
    if (c >= p.n_srcs * (uint32_t)kCand) return;
    const uint32_t k = c / kCand, i = c % kCand;
    int32_t scx, scz;
    src_chunk(p, d, k, scx, scz);
    Tree t;
    int32_t h = 0;
    if (tree_candidate(scx, scz, i, g, t)) {
        Emit e;
        e.out = reinterpret_cast<Prim *>(p.prims) + (size_t)c * kPrims;
        e.n = 0;
        tree_prims(t, g.lmx, e);
        h = e.n | ((t.x - scx * kCV) << 8) | ((t.z - scz * kCV) << 13) | (t.y << 18);
    }
    p.hdr[c] = h;
}

// The columns and the trees in one launch: the trees are few threads with a
// long chain of work each (35-40 us as a launch of their own), so their CTAs
// go first and the columns' run beside them.
__global__ void __launch_bounds__(256) k_gen_xz(GenPlan p, Dims d, Seed g, uint32_t tree_ctas) {
    if (blockIdx.x < tree_ctas) gen_tree(p, d, g, blockIdx.x * blockDim.x + threadIdx.x);
    else gen_column(p, d, g, (blockIdx.x - tree_ctas) * blockDim.x + threadIdx.x);
}

// ------------------------------------------------------------------ chunks
constexpr int kSlotThreads = 256;   // three CTAs per SM overlap each other's barriers
static_assert(kTrees <= 9 * kCand && (512 % kSlotThreads) == 0, "write-out covers 512 bricks");

// Job b of a plan (kGenJobInts ints, the layout of explicit plans).
__device__ __forceinline__ void job_of(const GenPlan &p, const Dims &d, uint32_t b,
                                      int32_t job[kGenJobInts]) {
    if (!p.window) {
#pragma unroll
        for (int k = 0; k < kGenJobInts; ++k) job[k] = p.jobs[(size_t)b * kGenJobInts + k];
        return;
    }
    const int32_t sxn = d.bx / 8, szn = d.bz / 8;
    // y slowest: the chunks below ground, which take longest, start first
    const int32_t sx = (int32_t)b % sxn, sz = ((int32_t)b / sxn) % szn,
                  sy = (int32_t)b / (sxn * szn);
    const int32_t cx = p.ox + wrap(sx - p.ox, sxn), cz = p.oz + wrap(sz - p.oz, szn);
    job[0] = cx; job[1] = sy; job[2] = cz;
    job[3] = sx; job[4] = sy; job[5] = sz;
    job[6] = sx + sz * sxn;
#pragma unroll
    for (int k = 0; k < 9; ++k)
        job[7 + k] = (cx + k % 3 - 1 - (p.ox - 1)) + (cz + k / 3 - 1 - (p.oz - 1)) * (sxn + 2);
}

// The two ore noises of stone_or_ore (voxel.rs:1906-1916) and the two of the
// caves (:1333-1461) over half a chunk, 16 levels at a time: the
// hashes of the lattice points the half can touch lie in shared memory, and
// what depends on y alone -- the lattice row and the smoothed fraction -- in
// tables of the chunk's 32 levels.
// A voxel column by itself hashes each of its lattice cells' new corners (36
// and 74 hashes per column for the ore frequencies, 1,024 columns); a half
// has 847 and 4,400 lattice points, and 64 and 108 of the caves'.
constexpr float kOreF1 = 0.27f, kOreF2 = 0.55f;
constexpr float kCaveF1 = 0.045f, kCaveF2 = 0.110f, kCaveY1 = 0.085f, kCaveY2 = 0.060f;
constexpr int kHalf = 16;
// points: 31 f + 2 in x and z, 15 f + 2 in y, rounded up
constexpr int kN1 = 11, kY1 = 7, kN2 = 20, kY2 = 11, kN3 = 4, kY3 = 4, kN4 = 6, kY4 = 3;
struct __align__(16) NoiseLevel {
    float yf, yf2, yg, yg2;     // smoothed fraction and 1 - it, twice each
};
struct SlotShared {
    uint8_t mat[kCV * kCV * kCV];
    float t1[kY1 * kN1 * kN1], t2[kY2 * kN2 * kN2], t3[kY3 * kN3 * kN3], t4[kY4 * kN4 * kN4];
    NoiseLevel l[4][kCV];
    int32_t row[4][kCV];            // lattice row of each level
    float one[2];                   // 1
    uint32_t step[4];               // bit y: its row is the one after level y - 1's
    int32_t job[kGenJobInts];
    int32_t x0[4], z0[4];           // first cells of the tables
    // per brick: uniform byte, any voxel (once the tables are done with)
    __device__ uint8_t *uni() { return reinterpret_cast<uint8_t *>(t2); }
    __device__ uint8_t *solid() { return uni() + 512; }
};
static_assert(3 * (sizeof(SlotShared) + 1024) <= 228 * 1024, "three CTAs per SM");
// one noise of a column, read from the lattice table: value_noise_3d's
// operations on the same hashes
template <int N>
struct TableColumn {
    int32_t at;         // the column's lattice cell in lattice row 0 of the table
    float xf, zf, zg;
    float a, b, c, d;
    int32_t yi;
    // x and z times the frequency; the table's first cell
    __device__ __forceinline__ void init(float x, float z, int32_t x0, int32_t y0, int32_t z0) {
        const int32_t xi = noise::floor_i(x), zi = noise::floor_i(z);
        xf = noise::smooth(x - (float)xi);
        zf = noise::smooth(z - (float)zi);
        zg = 1.0f - zf;
        at = ((zi - z0) - y0 * N) * N + (xi - x0);
        yi = INT32_MIN;
    }
    __device__ __forceinline__ float lerp(const float *q) const {
        return q[0] * (1.0f - xf) + q[1] * xf;
    }
    __device__ __forceinline__ float eval(const float *t, const NoiseLevel &l, int32_t row) {
        if (row != yi) {
            const float *q = t + (at + row * (N * N));
            if (row == yi + 1) {
                a = b;
                c = d;
            } else {
                a = lerp(q);
                c = lerp(q + N);
            }
            b = lerp(q + N * N);
            d = lerp(q + N * N + N);
            yi = row;
        }
        const float ab = a * l.yg + b * l.yf;
        const float cd = c * l.yg + d * l.yf;
        return ab * zg + cd * zf;
    }
};
// Two columns at once, of one x and two z: the same operations, two to an
// instruction (each half of a float pair rounds by itself).  Their y levels go
// up one by one from the half's first.
// A pair's mul and add came out contracted into one rounding (one ore voxel of
// a 512x256x512 window fell on the other side of its threshold), so sums are
// a * one + b, with a one that the compiler does not know: a's product is
// rounded before it is multiplied, and times one is exact.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pair(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpair(f2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b, f2 one) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(one), "l"(b));
    return r;
}
template <int N>
struct TablePair {
    const float *q0, *q1;   // the columns' cells in the upper lattice row
    float xf, xg;
    f2 zf, zg, a, b, c, d;
    __device__ __forceinline__ f2 lerp(int o, f2 one) const {
        return add2(mul2(pair(q0[o], q1[o]), pair(xg, xg)),
                    mul2(pair(q0[o + 1], q1[o + 1]), pair(xf, xf)), one);
    }
    __device__ __forceinline__ void init(const float *t, float x, float za, float zb, int32_t x0,
                                         int32_t z0, f2 one) {
        const int32_t xi = noise::floor_i(x), zi = noise::floor_i(za), zj = noise::floor_i(zb);
        xf = noise::smooth(x - (float)xi);
        xg = 1.0f - xf;
        const float fa = noise::smooth(za - (float)zi), fb = noise::smooth(zb - (float)zj);
        zf = pair(fa, fb);
        zg = pair(1.0f - fa, 1.0f - fb);
        q0 = t + (zi - z0) * N + (xi - x0);
        q1 = t + (zj - z0) * N + (xi - x0);
        a = lerp(0, one);
        c = lerp(N, one);
        q0 += N * N;
        q1 += N * N;
        b = lerp(0, one);
        d = lerp(N, one);
    }
    __device__ __forceinline__ void step(f2 one) {
        q0 += N * N;
        q1 += N * N;
        a = b;
        c = d;
        b = lerp(0, one);
        d = lerp(N, one);
    }
    __device__ __forceinline__ f2 eval(const NoiseLevel &l, f2 one) const {
        const f2 yf = pair(l.yf, l.yf2), yg = pair(l.yg, l.yg2);
        const f2 ab = add2(mul2(a, yg), mul2(b, yf), one);
        const f2 cd = add2(mul2(c, yg), mul2(d, yf), one);
        return add2(mul2(ab, zg), mul2(cd, zf), one);
    }
};
__device__ __forceinline__ uint8_t ore_of(float combined, int32_t depth) {
    if (depth > 30 && combined > 0.50f) return M_DIAMOND;
    if (depth > 20 && combined > 0.36f) return M_GOLD;
    if (depth > 10 && combined > 0.24f) return M_IRON;
    if (combined > 0.32f) return M_COAL;
    return M_STONE;
}

// The two kinds of column that few chunks have are calls, so their noises'
// registers are not the kernel's (inlined: 334 us against 325 for an 8 x 3
// chunk step of a 2048x2048 window).
//
// Levels [y, end) of stone and ore with caves below `seal`, from the tables.
__device__ __noinline__ void cave_column(SlotShared &sh, float wx, float wz, uint32_t dx,
                                         uint32_t dz, int32_t y0, int half, int32_t end,
                                         int32_t seal, int32_t h) {
    const int first = half * kHalf;
    TableColumn<kN1> o1;
    TableColumn<kN2> o2;
    TableColumn<kN3> c1;
    TableColumn<kN4> c2;
    o1.init(wx * kOreF1, wz * kOreF1, sh.x0[0], sh.row[0][first], sh.z0[0]);
    o2.init(wx * kOreF2, wz * kOreF2, sh.x0[1], sh.row[1][first], sh.z0[1]);
    c1.init(wx * kCaveF1, wz * kCaveF1, sh.x0[2], sh.row[2][first], sh.z0[2]);
    c2.init(wx * kCaveF2, wz * kCaveF2, sh.x0[3], sh.row[3][first], sh.z0[3]);
    for (int32_t y = y0 + first; y < end; ++y) {
        const int l = y - y0;
        if (y < seal && y > 4) {
            const float cn = c1.eval(sh.t3, sh.l[2][l], sh.row[2][l]);
            const float cn2 = c2.eval(sh.t4, sh.l[3][l], sh.row[3][l]);
            if ((cn + cn2 * 0.6f) > 0.30f) continue;
        }
        const float n1 = o1.eval(sh.t1, sh.l[0][l], sh.row[0][l]);
        const float n2 = o2.eval(sh.t2, sh.l[1][l], sh.row[1][l]);
        sh.mat[vox(dx, (uint32_t)l, dz)] = ore_of(n1 + n2 * 0.30f, h - y);
    }
}

// Levels [y, end) up to the surface of a column beyond the tables.
__device__ __noinline__ void direct_column(uint8_t *s_mat, float wx, float wz, uint32_t dx,
                                           uint32_t dz, int32_t y0, int32_t y, int32_t end,
                                           int32_t seal, int32_t h, int biome) {
    noise::ColumnNoise3 ore1, ore2, cave1, cave2;
    ore1.init(wx * kOreF1, wz * kOreF1);
    ore2.init(wx * kOreF2, wz * kOreF2);
    cave1.init(wx * kCaveF1, wz * kCaveF1);
    cave2.init(wx * kCaveF2, wz * kCaveF2);
    for (; y < end && y <= h; ++y) {
        if (!(y >= seal) && y > 4 && y + 3 < h) {
            const float cn = cave1.eval((float)y * kCaveY1);
            const float cn2 = cave2.eval((float)y * kCaveY2);
            if ((cn + cn2 * 0.6f) > 0.30f) continue;
        }
        uint8_t mat;
        if (y >= h) {
            mat = top_block(biome, (uint32_t)h);
        } else if (y + 4 >= h) {
            mat = subsoil(biome);
        } else {
            const float n1 = ore1.eval((float)y * kOreF1), n2 = ore2.eval((float)y * kOreF2);
            mat = ore_of(n1 + n2 * 0.30f, h - y);
        }
        s_mat[vox(dx, (uint32_t)(y - y0), dz)] = mat;
    }
}

__global__ void __launch_bounds__(kSlotThreads, 3) k_gen_slot(DevWorld w, GenPlan pl) {
    extern __shared__ __align__(16) uint8_t s_raw[];
    SlotShared &sh = *reinterpret_cast<SlotShared *>(s_raw);
    uint8_t *s_mat = sh.mat;
    int32_t *s_job = sh.job;
    if (threadIdx.x == 0) {
        int32_t j[kGenJobInts];
        job_of(pl, w.d, blockIdx.x, j);
#pragma unroll
        for (int k = 0; k < kGenJobInts; ++k) s_job[k] = j[k];
    }
    const uint32_t tid = threadIdx.x;
    const Prim *prims = reinterpret_cast<const Prim *>(pl.prims);

    __syncthreads();
    const int32_t *job = s_job;
    const int32_t lo[3] = {job[0] * kCV, job[1] * kCV, job[2] * kCV};
    const uint32_t *colw = pl.colw + (size_t)job[6] * (kCV * kCV);
    const uint32_t sbx = (uint32_t)job[3] * 8u, sby = (uint32_t)job[4] * 8u,
                   sbz = (uint32_t)job[5] * 8u;
    int32_t h_max = -1;
    {
        bool any = false;               // can anything be in this chunk?
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t word = __ldg(colw + tid + kSlotThreads * i);
            const int32_t h = (int32_t)(word & 0xFFu);
            h_max = max(h_max, h);
            // two levels of decoration over the column, or its water
            any = any || max(h + 2, (word >> 8) & 1u ? kSea : 0) >= lo[1];
        }
        if (tid < (uint32_t)kTrees) {
            const int32_t hd = __ldg(pl.hdr + (size_t)job[7 + tid / kCand] * kCand + tid % kCand);
            any = any || ((hd & 0xFF) != 0 && (hd >> 18) <= lo[1] + kCV && (hd >> 18) + 22 >= lo[1]);
        }
        if (__syncthreads_or(any) == 0) {
            // all air (three quarters of the chunks): rows of eight bricks
            for (uint32_t i = tid; i < 2048u; i += kSlotThreads) {
                const uint32_t r = i >> 5;
                const size_t gbi = sbx + (sby + (r & 7u)) * (size_t)w.d.bx +
                                   (sbz + (r >> 3)) * (size_t)(w.d.bx * w.d.by);
                reinterpret_cast<uint4 *>(w.mat + gbi * 64u)[i & 31u] = make_uint4(0, 0, 0, 0);
            }
            for (uint32_t b = tid; b < 512u; b += kSlotThreads) {
                const size_t gbi = (sbx + (b & 7u)) + (sby + ((b >> 3) & 7u)) * (size_t)w.d.bx +
                                   (sbz + (b >> 6)) * (size_t)(w.d.bx * w.d.by);
                w.occ[gbi] = 0ull;
                w.brick_uniform[gbi] = 0;
            }
            if (tid < 8u) {
                const int64_t ti = (int64_t)(job[3] * 2 + (int32_t)(tid & 1u)) +
                                   (int64_t)(job[4] * 2 + (int32_t)((tid >> 1) & 1u)) * w.d.tx +
                                   (int64_t)(job[5] * 2 + (int32_t)(tid >> 2)) * w.d.tx * w.d.ty;
                w.tile_mask[ti] = 0ull;
                w.tile_uniform[ti] = 0;
            }
            return;
        }
    }
    uint4 *zero = reinterpret_cast<uint4 *>(s_mat);
    for (uint32_t i = tid; i < (uint32_t)(kCV * kCV * kCV / 16); i += kSlotThreads)
        zero[i] = make_uint4(0, 0, 0, 0);

    // ---- the columns (dx, dz), voxel.rs:1333-1461
    // Thread: dx = its lane, dz = its warp + 8 i.
    const int32_t y0 = lo[1];
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    const int32_t wxi = lo[0] + (int32_t)lane;
    const float wx = (float)wxi;
    // x and z lattice cells; a chunk so far out that binary32 coordinates
    // skip cells does not fit the tables and evaluates its noise directly
    const float xb = (float)lo[0], zb = (float)lo[2];
    const int32_t x1 = noise::floor_i(xb * kOreF1), x2 = noise::floor_i(xb * kOreF2);
    const int32_t z1 = noise::floor_i(zb * kOreF1), z2 = noise::floor_i(zb * kOreF2);
    const int32_t x3 = noise::floor_i(xb * kCaveF1), x4 = noise::floor_i(xb * kCaveF2);
    const int32_t z3 = noise::floor_i(zb * kCaveF1), z4 = noise::floor_i(zb * kCaveF2);
    const float xe = (float)(lo[0] + kCV - 1), ze = (float)(lo[2] + kCV - 1);
    const bool tables = noise::floor_i(xe * kOreF1) - x1 + 2 <= kN1 &&
                        noise::floor_i(ze * kOreF1) - z1 + 2 <= kN1 &&
                        noise::floor_i(xe * kOreF2) - x2 + 2 <= kN2 &&
                        noise::floor_i(ze * kOreF2) - z2 + 2 <= kN2 &&
                        noise::floor_i(xe * kCaveF1) - x3 + 2 <= kN3 &&
                        noise::floor_i(ze * kCaveF1) - z3 + 2 <= kN3 &&
                        noise::floor_i(xe * kCaveF2) - x4 + 2 <= kN4 &&
                        noise::floor_i(ze * kCaveF2) - z4 + 2 <= kN4;
    if (tid == 0) {
        sh.one[0] = sh.one[1] = 1.0f;
        sh.x0[0] = x1; sh.x0[1] = x2; sh.x0[2] = x3; sh.x0[3] = x4;
        sh.z0[0] = z1; sh.z0[1] = z2; sh.z0[2] = z3; sh.z0[3] = z4;
    }
    if (tid < 4u * kCV) {
        const uint32_t q = tid >> 5, l = tid & 31u;     // noise, level
        const float f = q == 0u ? kOreF1 : (q == 1u ? kOreF2 : (q == 2u ? kCaveY1 : kCaveY2));
        const float py = (float)(y0 + (int32_t)l) * f;
        const int32_t yi = noise::floor_i(py);
        const float yf = noise::smooth(py - (float)yi);
        sh.l[q][l] = NoiseLevel{yf, yf, 1.0f - yf, 1.0f - yf};
        sh.row[q][l] = yi;
        const int32_t below = __shfl_up_sync(0xFFFFFFFFu, yi, 1);
        const uint32_t step = __ballot_sync(0xFFFFFFFFu, l != 0u && yi != below);
        if (l == 0u) sh.step[q] = step;
    }
    for (int half = 0; half < kCV / kHalf; ++half) {
        const int32_t ylo = y0 + half * kHalf, yhi = ylo + kHalf;
        // any voxel of stone or ore (y + 4 < h) in this half?
        const bool ore = __syncthreads_or(ylo + 4 < h_max) != 0 && tables;
        const int32_t r1 = sh.row[0][half * kHalf], r2 = sh.row[1][half * kHalf];
        const int32_t r3 = sh.row[2][half * kHalf], r4 = sh.row[3][half * kHalf];
        if (ore) {
            for (uint32_t i = tid; i < (uint32_t)(kY1 * kN1 * kN1); i += kSlotThreads)
                sh.t1[i] = hash3(sh.x0[0] + (int32_t)(i % kN1), r1 + (int32_t)(i / (kN1 * kN1)),
                                 sh.z0[0] + (int32_t)((i / kN1) % kN1));
            for (uint32_t i = tid; i < (uint32_t)(kY2 * kN2 * kN2); i += kSlotThreads)
                sh.t2[i] = hash3(sh.x0[1] + (int32_t)(i % kN2), r2 + (int32_t)(i / (kN2 * kN2)),
                                 sh.z0[1] + (int32_t)((i / kN2) % kN2));
            for (uint32_t i = tid; i < (uint32_t)(kY3 * kN3 * kN3); i += kSlotThreads)
                sh.t3[i] = hash3(sh.x0[2] + (int32_t)(i % kN3), r3 + (int32_t)(i / (kN3 * kN3)),
                                 sh.z0[2] + (int32_t)((i / kN3) % kN3));
            for (uint32_t i = tid; i < (uint32_t)(kY4 * kN4 * kN4); i += kSlotThreads)
                sh.t4[i] = hash3(sh.x0[3] + (int32_t)(i % kN4), r4 + (int32_t)(i / (kN4 * kN4)),
                                 sh.z0[3] + (int32_t)((i / kN4) % kN4));
            __syncthreads();
        }
        bool caves = false;             // any in the warp's pair of rows of columns?
        for (int i = 0; i < 4; ++i) {
            const uint32_t word = __ldg(colw + tid + kSlotThreads * i);
            const int32_t h = (int32_t)(word & 0xFFu);
            const int32_t water_top = (word >> 8) & 1u ? kSea : 0;
            const int col_top = max(h, water_top);
            // caves only under water, below its seal
            const int32_t seal = water_top > h ? h - 5 : INT32_MIN;
            const uint32_t dx = lane, dz = warp + 8u * (uint32_t)i;
            const float wz = (float)(lo[2] + (int32_t)dz);
            // below the subsoil (y + 4 < h) stone and ore: without caves two
            // columns at once, dz and dz + 8
            if ((i & 1) == 0 && ore) {
                const uint32_t next = __ldg(colw + tid + kSlotThreads * (i + 1));
                const int32_t hn = (int32_t)(next & 0xFFu);
                const int32_t sn = ((next >> 8) & 1u) && kSea > hn ? hn - 5 : INT32_MIN;
                caves = __any_sync(0xFFFFFFFFu, ylo < max(seal, sn));
                const int32_t ea = min(yhi, h - 4), eb = min(yhi, hn - 4), e = max(ea, eb);
                if (!caves && ylo < e) {
                    TablePair<kN1> o1;
                    TablePair<kN2> o2;
                    const f2 one = pair(sh.one[0], sh.one[1]), third = pair(0.30f, 0.30f);
                    const float wn = (float)(lo[2] + (int32_t)dz + 8);
                    o1.init(sh.t1, wx * kOreF1, wz * kOreF1, wn * kOreF1, sh.x0[0], sh.z0[0],
                            one);
                    o2.init(sh.t2, wx * kOreF2, wz * kOreF2, wn * kOreF2, sh.x0[1], sh.z0[1],
                            one);
                    // bit 0: the next level's
                    uint32_t s1 = sh.step[0] >> (half * kHalf), s2 = sh.step[1] >> (half * kHalf);
                    uint8_t *v = s_mat + vox(dx, (uint32_t)(half * kHalf), dz);
                    for (int32_t y = ylo;;) {
                        const f2 n = add2(mul2(o2.eval(sh.l[1][y - y0], one), third),
                                          o1.eval(sh.l[0][y - y0], one), one);
                        float na, nb;
                        unpair(n, na, nb);
                        // 8 levels of z on: two brick layers
                        if (y < ea) v[0] = ore_of(na, h - y);
                        if (y < eb) v[2 * 64 * 64] = ore_of(nb, hn - y);
                        if (++y >= e) break;
                        v += (y & 3) != 0 ? 16 : 8 * 64 - 48;
                        s1 >>= 1;
                        s2 >>= 1;
                        if (s1 & 1u) o1.step(one);
                        if (s2 & 1u) o2.step(one);
                    }
                }
            }
            if (col_top < ylo) continue;
            const int biome = (int)((word >> 9) & 7u);
            const int32_t ye = min(yhi, kWorldY);
            int32_t y = ylo;
            if (ore) {
                const int32_t ore_end = min(ye, h - 4);
                if (caves) cave_column(sh, wx, wz, dx, dz, y0, half, ore_end, seal, h);
                y = max(ylo, ore_end);
            }
            if (tables) {
                // subsoil and surface (y + 4 >= h: neither ore nor caves)
                const uint8_t sub = subsoil(biome), top = top_block(biome, (uint32_t)h);
                for (; y < ye && y <= h; ++y)
                    s_mat[vox(dx, (uint32_t)(y - y0), dz)] = y >= h ? top : sub;
            } else if (y < ye && y <= h) {
                direct_column(s_mat, wx, wz, dx, dz, y0, y, ye, seal, h, biome);
            }
            if (water_top > h) {
                const int32_t fb = max(h + 1, ylo), fe = min(water_top, yhi - 1);
                for (int32_t wy = fb; wy <= fe; ++wy)
                    s_mat[vox(dx, (uint32_t)(wy - y0), dz)] = M_WATER;
            }
        }
        __syncthreads();                 // before the tables change
    }
    // surface decoration over the finished columns
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t word = __ldg(colw + tid + kSlotThreads * i);
        const uint32_t dec = (word >> 12) & 63u, dx = lane, dz = warp + 8u * (uint32_t)i;
        const int32_t dec_y = (int32_t)(word & 0xFFu) + 1;
        // a column that ends below the chunk decorates nothing in it
        if (dec != 0u && dec_y > y0 && dec_y < y0 + kCV) {
            const uint32_t dy = (uint32_t)(dec_y - y0);
            s_mat[vox(dx, dy, dz)] = (uint8_t)dec;
            if (((word >> 18) & 1u) && dec_y + 1 < y0 + kCV) s_mat[vox(dx, dy + 1u, dz)] = M_BUSH;
        }
    }
    __syncthreads();

    // ---- trees of the 3x3 source chunks in the reference's order, a slab of
    // four z levels per warp: the warp takes every primitive that can reach
    // its slab, in order, so no other thread writes its voxels
    {
        const int32_t zlo = lo[2] + 4 * (int32_t)warp, zhi = zlo + 4;
        int32_t hd[(kTrees + 31) / 32];
#pragma unroll
        for (int q = 0; q < (kTrees + 31) / 32; ++q) {
            const int c = q * 32 + (int)lane;
            hd[q] = 0;
            if (c < kTrees) hd[q] = __ldg(pl.hdr + (size_t)job[7 + c / kCand] * kCand + c % kCand);
        }
#pragma unroll
        for (int q = 0; q < (kTrees + 31) / 32; ++q) {
            const int c = q * 32 + (int)lane, k = c / kCand;
            const int32_t bx = (job[0] + k % 3 - 1) * kCV + ((hd[q] >> 8) & 31);
            const int32_t bz = (job[2] + k / 3 - 1) * kCV + ((hd[q] >> 13) & 31);
            const int32_t by = hd[q] >> 18;
            uint32_t near = __ballot_sync(
                0xFFFFFFFFu, (hd[q] & 0xFF) != 0 && by <= lo[1] + kCV && by + 22 >= lo[1] &&
                                 bx + kTreeReach >= lo[0] && bx - kTreeReach < lo[0] + kCV &&
                                 bz + kTreeReach >= zlo && bz - kTreeReach < zhi);
            while (near != 0u) {
                const int l = __ffs((int)near) - 1;
                near &= near - 1u;
                const int tc = q * 32 + l, np = __shfl_sync(0xFFFFFFFFu, hd[q], l) & 0xFF;
                // one primitive per lane; those that reach the slab, in order
                Prim mine{};
                bool meets = false;
                if ((int)lane < np) {
                    const Prim *tp = prims + ((size_t)job[7 + tc / kCand] * kCand + tc % kCand) * kPrims;
                    const int4 a = __ldg(reinterpret_cast<const int4 *>(tp + lane));
                    const int4 b = __ldg(reinterpret_cast<const int4 *>(tp + lane) + 1);
                    mine.a[0] = a.x; mine.a[1] = a.y; mine.a[2] = a.z; mine.b[0] = a.w;
                    mine.b[1] = b.x; mine.b[2] = b.y; mine.kind_mat = (uint32_t)b.z; mine.steps = b.w;
                    int32_t mn[3], mx[3];
                    prim_box(mine, mn, mx);
                    meets = mx[0] >= lo[0] && mn[0] < lo[0] + kCV && mx[1] >= lo[1] &&
                            mn[1] < lo[1] + kCV && mx[2] >= zlo && mn[2] < zhi;
                }
                uint32_t todo = __ballot_sync(0xFFFFFFFFu, meets);
                while (todo != 0u) {
                    const int o = __ffs((int)todo) - 1;
                    todo &= todo - 1u;
                    Prim pr;
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        pr.a[m] = __shfl_sync(0xFFFFFFFFu, mine.a[m], o);
                        pr.b[m] = __shfl_sync(0xFFFFFFFFu, mine.b[m], o);
                    }
                    pr.kind_mat = __shfl_sync(0xFFFFFFFFu, mine.kind_mat, o);
                    pr.steps = __shfl_sync(0xFFFFFFFFu, mine.steps, o);
                    paint_prim(s_mat, lo, zlo, zhi, pr);
                    __syncwarp();
                }
            }
        }
    }
    __syncthreads();

    // ---- bricks out: material rows, occupancy words, uniform bytes
    for (uint32_t b = tid; b < 512u; b += kSlotThreads) {
        const uint32_t gbi = (sbx + (b & 7u)) + (sby + ((b >> 3) & 7u)) * (uint32_t)w.d.bx +
                             (sbz + (b >> 6)) * (uint32_t)(w.d.bx * w.d.by);
        const uint4 *src = reinterpret_cast<const uint4 *>(s_mat + b * 64u);
        uint4 *dst = reinterpret_cast<uint4 *>(w.mat + (size_t)gbi * 64u);
        uint64_t occ = 0;
        const uint32_t m0 = s_mat[b * 64u], rep = 0x01010101u * m0;
        bool same = m0 != 0u;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
            const uint4 q = src[q4];
            dst[q4] = q;
            const uint32_t qs[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                same = same && qs[m] == rep;
                // top bit of each byte that is not 0, the four bits side by side
                const uint32_t nz = (((qs[m] & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | qs[m]) & 0x80808080u;
                occ |= (uint64_t)(((nz >> 7) * 0x10204080u) >> 28) << (16 * q4 + 4 * m);
            }
        }
        w.occ[gbi] = occ;
        const uint8_t u = (occ == ~0ull && same) ? (uint8_t)m0 : (uint8_t)0;
        w.brick_uniform[gbi] = u;
        sh.uni()[b] = u;
        sh.solid()[b] = occ != 0ull ? 1u : 0u;
    }
    __syncthreads();
    // the chunk's eight tiles, one warp each (tile word and LUT,
    // voxel.rs:253-272, :964-972): their bricks are all here
    {
        const uint32_t tx = warp & 1u, ty = (warp >> 1) & 1u, tz = warp >> 2;
        uint32_t u[2], sol[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint32_t c = lane + 32u * (uint32_t)q;   // child bit x + z*4 + y*16
            const uint32_t b = (tx * 4u + (c & 3u)) + (ty * 4u + (c >> 4)) * 8u +
                               (tz * 4u + ((c >> 2) & 3u)) * 64u;
            u[q] = sh.uni()[b];
            sol[q] = sh.solid()[b];
        }
        const uint32_t m_lo = __ballot_sync(0xFFFFFFFFu, sol[0] != 0u);
        const uint32_t m_hi = __ballot_sync(0xFFFFFFFFu, sol[1] != 0u);
        const uint32_t m0 = __shfl_sync(0xFFFFFFFFu, u[0], 0);
        const bool uni = __all_sync(0xFFFFFFFFu, m0 != 0u && u[0] == m0 && u[1] == m0);
        if (lane == 0u) {
            const int64_t ti = (int64_t)(job[3] * 2 + (int32_t)tx) +
                               (int64_t)(job[4] * 2 + (int32_t)ty) * w.d.tx +
                               (int64_t)(job[5] * 2 + (int32_t)tz) * w.d.tx * w.d.ty;
            w.tile_mask[ti] = (uint64_t)m_lo | ((uint64_t)m_hi << 32);
            w.tile_uniform[ti] = uni ? (uint8_t)m0 : (uint8_t)0;
        }
    }
}

}  // namespace

namespace {
__global__ void k_gen_math(const uint32_t *lmx, uint32_t fn, const float *__restrict__ in, size_t n,
                           float *__restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = in[i];
    float v;
    if (fn == gm::LMX_POW115) v = pow115(lmx, x);
    else if (fn == gm::LMX_POW085) v = pow085(lmx, x);
    else if (fn == gm::LMX_COS) v = cos_f(lmx, x);
    else v = sin_f(lmx, x);
    out[i] = v;
}
}  // namespace

cudaError_t launch_gen_math(const uint32_t *lmx, uint32_t fn, const float *in, size_t n, float *out,
                            cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_gen_math<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(lmx, fn, in, n, out);
    return cudaGetLastError();
}

size_t gen_prim_bytes_per_src() { return sizeof(Prim) * kCand * kPrims; }

cudaError_t launch_gen_slots(const DevWorld &w, uint64_t seed, const GenPlan &p, bool tiles_built,
                             cudaStream_t s) {
    if (p.n_jobs == 0) return cudaSuccess;
    Seed g;
    g.seed = seed;
    // seed_offset_xz, voxel.rs:1163-1167
    g.offx = (float)(int32_t)(uint32_t)(seed >> 32) * 0.01734f;
    g.offz = (float)(int32_t)(uint32_t)(seed & 0xFFFFFFFFull) * 0.02153f;
    g.lmx = p.lmx;
    if (!g.lmx) return cudaErrorInvalidValue;
    const uint32_t col_ctas = (p.n_cols * (uint32_t)(kCV * kCV) + 255u) / 256u;
    const uint32_t tree_ctas = (p.n_srcs * (uint32_t)kCand + 255u) / 256u;
    k_gen_xz<<<tree_ctas + col_ctas, 256, 0, s>>>(p, w.d, g, tree_ctas);
    cudaError_t e = cudaFuncSetAttribute(k_gen_slot, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(SlotShared));
    if (e != cudaSuccess) return e;
    k_gen_slot<<<p.n_jobs, kSlotThreads, sizeof(SlotShared), s>>>(w, p);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_rebuild_pyramid(w, !tiles_built, s);
}

}  // namespace vx
