// vx_mlp.cu -- the learned start-distance proposal: a 70->64->64->64->1 MLP
// with GELU (tanh form) that predicts log(first-hit t) of a ray from 6 ray
// values and the 64 tile bits of the chunk holding the ray origin.
//
//   inference  BF16 tensor cores (mma.sync, FP32 accumulation), in
//              vx_mlp_infer.cuh;
//   training   FP32: forward, loss and backward of a batch in one launch,
//              the partial gradients added in a fixed order, Adam.
//
// Features (80 columns, 70 used): origin mod 64 / 64 (3), direction (3), the
// 64 child bits of the origin chunk's tile mask (bit x + z*4 + y*16 of
// chunk_mask, src/voxel.rs:282-294), 10 zero columns.  The proposal only
// decides how far the exact traversal verifies before restarting; records
// never depend on its value, so this file uses ordinary float code
// generation (contraction, approximate tanh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "vx_internal.h"
#include "vx_mlp_infer.cuh"

namespace vx {

namespace {

template <bool FRAME>
__global__ void __launch_bounds__(128) k_mlp_infer(InferArgs a) {
    mlp_infer_body<FRAME>(a, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------- training
__device__ __forceinline__ float gelu_tanh(float x) {
    return tanhf(0.7978845608f * (x + 0.044715f * x * x * x));
}
// GELU (tanh form) and its derivative from th = gelu_tanh(x)
__device__ __forceinline__ float gelu_f(float x, float th) { return 0.5f * x * (1.0f + th); }
__device__ __forceinline__ float gelu_grad(float x, float th) {
    return 0.5f * (1.0f + th) +
           0.5f * x * (1.0f - th * th) * 0.7978845608f * (1.0f + 3.0f * 0.044715f * x * x);
}

// Forward, loss and backward of one batch in one launch.
//
// What bounds it: 1.1 GFLOP of FP32 FMA at a batch of 16,384 (15 us at the
// device's FMA rate); the batch itself is 5 MB.  Layer by layer the same step
// was 20 launches that carried every activation through memory, and the
// weight gradients' reductions over the batch ran on 64 CTAs: 385 us a step, now
// 91 (this kernel 54, k_train_reduce 8).
//
// One CTA per SM holds all weights in shared memory.  Its two groups of 128
// threads take tiles of 32 samples by themselves (named barriers), so one
// group's FMAs cover the other's barriers.  A tile's activations stay in
// shared memory from the forward to the backward pass, GELU's derivatives in
// the registers of the threads that need them again, and the weight
// gradients of all a group's tiles in registers (104 of them a thread):
// nothing but the batch is read and nothing but one partial gradient per CTA
// is written.  k_train_reduce adds the partials in a fixed order, so the
// gradient is the same from run to run.
//
// Thread (ty, tx) of a group, ty = 0..7, tx = 0..15:
//   activations     samples 4 ty + i, columns 4 tx + j
//   W2, W3 gradients  rows 8 ty + r, columns 4 tx + j
//   W1 gradient       rows 8 ty + r, columns tx + 16 j
// Weight rows are float4 columns, column c of row o kept at c ^ ((o >> 2) & 7):
// both the forward pass (16 rows at one column) and the backward pass (16
// columns of one row) then read without bank conflicts.
constexpr int kTs = 32;                       // samples per tile
constexpr int kXs = kIn + 4, kAs = kH + 4;    // row strides (floats) of X and activations
constexpr int kWs1 = 96, kWs = kH;            // row strides of the weights
constexpr int kGroupFloats = kTs * kXs + 4 * kTs * kAs;
constexpr int kWeightFloats = kH * kWs1 + 2 * kH * kWs + 4 * kH + 4;
constexpr int kTrainSmem = (kWeightFloats + 2 * kGroupFloats) * (int)sizeof(float);
static_assert(2 * kGroupFloats >= kMlpFloats + 16 * 4 * kH, "the epilogue's merge fits");

__device__ __forceinline__ void group_sync(int group) {
    asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");
}
__device__ __forceinline__ float at4(const float4 &v, int k) {
    return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w));
}

// z[i][j] += sum_k A[4 ty + i][k] W[4 tx + j][k], k ascending
template <int K, int AS, int WS>
__device__ __forceinline__ void tile_forward(const float *A, const float *W, int ty, int tx,
                                             float z[4][4]) {
#pragma unroll 2
    for (int c = 0; c < K / 4; ++c) {
        float4 a[4], w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            a[i] = *reinterpret_cast<const float4 *>(A + (4 * ty + i) * AS + 4 * c);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            w[j] = *reinterpret_cast<const float4 *>(W + (4 * tx + j) * WS + 4 * (c ^ (tx & 7)));
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) z[i][j] += at4(a[i], k) * at4(w[j], k);
    }
}
// d[i][j] = sum_o dZ[4 ty + i][o] W[o][4 tx + j], o ascending
__device__ __forceinline__ void tile_backward(const float *dZ, const float *W, int ty, int tx,
                                              float d[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) d[i][j] = 0.f;
#pragma unroll 2
    for (int c = 0; c < kH / 4; ++c) {
        float4 a[4], w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            a[i] = *reinterpret_cast<const float4 *>(dZ + (4 * ty + i) * kAs + 4 * c);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            w[k] = *reinterpret_cast<const float4 *>(W + (4 * c + k) * kWs + 4 * (tx ^ (c & 7)));
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) d[i][j] += at4(a[i], k) * at4(w[k], j);
    }
}
// g[r][j] += sum_b dZ[b][8 ty + r] A[b][4 tx + j], b ascending
__device__ __forceinline__ void tile_weight_grad(const float *dZ, const float *A, int ty, int tx,
                                                 float g[8][4]) {
#pragma unroll 2
    for (int b = 0; b < kTs; ++b) {
        const float4 z0 = *reinterpret_cast<const float4 *>(dZ + b * kAs + 8 * ty);
        const float4 z1 = *reinterpret_cast<const float4 *>(dZ + b * kAs + 8 * ty + 4);
        const float4 a = *reinterpret_cast<const float4 *>(A + b * kAs + 4 * tx);
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j) g[r][j] += at4(r < 4 ? z0 : z1, r & 3) * at4(a, j);
    }
}

// partial: gridDim.x x (kMlpFloats + 1) floats, each CTA's gradient and loss
__global__ void __launch_bounds__(256, 1) k_train_grad(const float *__restrict__ p,
                                                       const float *__restrict__ X,
                                                       const float *__restrict__ target, int B,
                                                       float *__restrict__ partial) {
    extern __shared__ __align__(16) float sm[];
    float *sW1 = sm, *sW2 = sW1 + kH * kWs1, *sW3 = sW2 + kH * kWs, *sV = sW3 + kH * kWs;
    const int tid = threadIdx.x, group = tid >> 7, t = tid & 127, ty = t >> 4, tx = t & 15;
    float *gs = sm + kWeightFloats + group * kGroupFloats;
    float *sX = gs, *sA1 = sX + kTs * kXs, *sA2 = sA1 + kTs * kAs, *sP = sA2 + kTs * kAs,
          *sQ = sP + kTs * kAs;
    for (int i = tid; i < kH * kIn / 4; i += 256) {
        const int o = i / (kIn / 4), c = i % (kIn / 4);
        *reinterpret_cast<float4 *>(sW1 + o * kWs1 + 4 * (c ^ ((o >> 2) & 7))) =
            *reinterpret_cast<const float4 *>(p + kW1 + 4 * i);
    }
    for (int i = tid; i < kH * kH / 4; i += 256) {
        const int o = i >> 4, c = i & 15, at = o * kWs + 4 * (c ^ ((o >> 2) & 7));
        *reinterpret_cast<float4 *>(sW2 + at) = *reinterpret_cast<const float4 *>(p + kW2 + 4 * i);
        *reinterpret_cast<float4 *>(sW3 + at) = *reinterpret_cast<const float4 *>(p + kW3 + 4 * i);
    }
    // b1, b2, b3, wo, bo
    if (tid < kH) {
        sV[tid] = p[kB1 + tid];
        sV[kH + tid] = p[kB2 + tid];
        sV[2 * kH + tid] = p[kB3 + tid];
        sV[3 * kH + tid] = p[kWo + tid];
        if (tid == 0) sV[4 * kH] = p[kBo];
    }
    __syncthreads();

    float g1[8][5] = {}, g2[8][4] = {}, g3[8][4] = {};
    float gb1[4] = {}, gb2[4] = {}, gb3[4] = {}, gwo[4] = {}, gbo = 0.f, loss = 0.f;
    const bool wide = (reinterpret_cast<uintptr_t>(X) & 15u) == 0u;
    const int tiles = (B + kTs - 1) / kTs;
    // consecutive tiles go to different SMs, then to the second groups
    for (int tile = blockIdx.x + group * gridDim.x; tile < tiles; tile += 2 * gridDim.x) {
        const int b0 = tile * kTs, rows = min(kTs, B - b0);
        // samples beyond the batch are zero rows and get a zero dY
        if (wide) {
#pragma unroll
            for (int k = 0; k < kTs * kIn / 4 / 128; ++k) {
                const int i = t + 128 * k, r = i / (kIn / 4), c = i % (kIn / 4);
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < rows) v = __ldg(reinterpret_cast<const float4 *>(X + (size_t)(b0 + r) * kIn) + c);
                *reinterpret_cast<float4 *>(sX + r * kXs + 4 * c) = v;
            }
        } else {
            for (int i = t; i < kTs * kIn; i += 128) {
                const int r = i / kIn, c = i % kIn;
                sX[r * kXs + c] = r < rows ? __ldg(X + (size_t)(b0 + r) * kIn + c) : 0.f;
            }
        }
        group_sync(group);
        float z[4][4], d1[4][4], d2[4][4];
        // layers 1 and 2: activations to shared memory, derivatives kept
#pragma unroll
        for (int layer = 0; layer < 2; ++layer) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) z[i][j] = 0.f;
            if (layer == 0) tile_forward<kIn, kXs, kWs1>(sX, sW1, ty, tx, z);
            else tile_forward<kH, kAs, kWs>(sA1, sW2, ty, tx, z);
            float *out = layer == 0 ? sA1 : sA2;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float x = z[i][j] + sV[layer * kH + 4 * tx + j], th = gelu_tanh(x);
                    v[j] = gelu_f(x, th);
                    (layer == 0 ? d1 : d2)[i][j] = gelu_grad(x, th);
                }
                *reinterpret_cast<float4 *>(out + (4 * ty + i) * kAs + 4 * tx) =
                    make_float4(v[0], v[1], v[2], v[3]);
            }
            group_sync(group);
        }
        // layer 3, the output and the loss: y = A3 . wo + bo, dY = 2 (y - target) / B
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) z[i][j] = 0.f;
        tile_forward<kH, kAs, kWs>(sA2, sW3, ty, tx, z);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 4 * ty + i;
            float a3[4], d3[4], y = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float x = z[i][j] + sV[2 * kH + 4 * tx + j], th = gelu_tanh(x);
                a3[j] = gelu_f(x, th);
                d3[j] = gelu_grad(x, th);
                y += a3[j] * sV[3 * kH + 4 * tx + j];
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) y += __shfl_xor_sync(0xFFFFFFFFu, y, o);
            float dy = 0.f;
            if (r < rows) {
                const float e = (y + sV[4 * kH]) - __ldg(target + b0 + r);
                dy = 2.0f * e / (float)B;
                if (tx == 0) {
                    loss += e * e / (float)B;
                    gbo += dy;
                }
            }
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                gwo[j] += dy * a3[j];
                v[j] = dy * sV[3 * kH + 4 * tx + j] * d3[j];
                gb3[j] += v[j];
            }
            *reinterpret_cast<float4 *>(sP + r * kAs + 4 * tx) = make_float4(v[0], v[1], v[2], v[3]);
        }
        group_sync(group);
        // backward: dZ3 in sP, dZ2 in sQ, dZ1 in sP
        tile_weight_grad(sP, sA2, ty, tx, g3);
        tile_backward(sP, sW3, ty, tx, z);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                z[i][j] *= d2[i][j];
                gb2[j] += z[i][j];
            }
            *reinterpret_cast<float4 *>(sQ + (4 * ty + i) * kAs + 4 * tx) =
                make_float4(z[i][0], z[i][1], z[i][2], z[i][3]);
        }
        group_sync(group);
        tile_weight_grad(sQ, sA1, ty, tx, g2);
        tile_backward(sQ, sW2, ty, tx, z);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                z[i][j] *= d1[i][j];
                gb1[j] += z[i][j];
            }
            *reinterpret_cast<float4 *>(sP + (4 * ty + i) * kAs + 4 * tx) =
                make_float4(z[i][0], z[i][1], z[i][2], z[i][3]);
        }
        group_sync(group);
#pragma unroll 2
        for (int b = 0; b < kTs; ++b) {
            const float4 z0 = *reinterpret_cast<const float4 *>(sP + b * kAs + 8 * ty);
            const float4 z1 = *reinterpret_cast<const float4 *>(sP + b * kAs + 8 * ty + 4);
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const float x = sX[b * kXs + tx + 16 * j];
#pragma unroll
                for (int r = 0; r < 8; ++r) g1[r][j] += at4(r < 4 ? z0 : z1, r & 3) * x;
            }
        }
        group_sync(group);
    }

    // the CTA's partial: group 1's sums through shared memory, group 0 adds
    // its own; the column sums (biases, wo) of the 16 (group, ty) rows after
    __syncthreads();
    float *mg = sm + kWeightFloats, *cols = mg + kMlpFloats;
    float *out = partial + (size_t)blockIdx.x * (kMlpFloats + 1);
#pragma unroll
    for (int phase = 0; phase < 2; ++phase) {
        if (group == 1 - phase) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
#pragma unroll
                for (int j = 0; j < 5; ++j) {
                    const int i = kW1 + (8 * ty + r) * kIn + tx + 16 * j;
                    if (phase == 0) mg[i] = g1[r][j];
                    else out[i] = g1[r][j] + mg[i];
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = (8 * ty + r) * kH + 4 * tx + j;
                    if (phase == 0) {
                        mg[kW2 + i] = g2[r][j];
                        mg[kW3 + i] = g3[r][j];
                    } else {
                        out[kW2 + i] = g2[r][j] + mg[kW2 + i];
                        out[kW3 + i] = g3[r][j] + mg[kW3 + i];
                    }
                }
            }
        }
        if (phase == 0) {
            float *c = cols + (group * 8 + ty) * 4 * kH + 4 * tx;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                c[j] = gb1[j];
                c[kH + j] = gb2[j];
                c[2 * kH + j] = gb3[j];
                c[3 * kH + j] = gwo[j];
            }
            if (tx == 0) {
                sV[group * 8 + ty] = gbo;
                sV[16 + group * 8 + ty] = loss;
            }
        }
        __syncthreads();
    }
    {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) s += cols[k * 4 * kH + tid];
        const int off[4] = {kB1, kB2, kB3, kWo};
        out[off[tid >> 6] + (tid & 63)] = s;
        if (tid < 2) {
            float v = 0.f;
#pragma unroll
            for (int k = 0; k < 16; ++k) v += sV[16 * tid + k];
            out[tid == 0 ? kBo : kMlpFloats] = v;
        }
    }
}

// grad[i] (and the loss, entry kMlpFloats) = sum of the partials in CTA order:
// 32 entries per CTA, eight threads each take every eighth partial.
__global__ void __launch_bounds__(256) k_train_reduce(const float *__restrict__ partial, int parts,
                                                      float *__restrict__ grad,
                                                      float *__restrict__ loss) {
    __shared__ float s[8][33];
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    float v = 0.f;
    if (i <= kMlpFloats) {
#pragma unroll 8
        for (int c = row; c < parts; c += 8) v += __ldg(partial + (size_t)c * (kMlpFloats + 1) + i);
    }
    s[row][lane] = v;
    __syncthreads();
    if (row == 0 && i <= kMlpFloats) {
#pragma unroll
        for (int k = 1; k < 8; ++k) v += s[k][lane];
        if (i < kMlpFloats) grad[i] = v;
        else *loss = v;
    }
}

__global__ void k_adam(float *p, const float *g, float *m, float *v, int n, float lr, float b1,
                       float b2, float eps, float bc1, float bc2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// f32 W1, W2, W3 -> padded bf16 rows
__global__ void k_to_bf16(const float *p, __nv_bfloat16 *w) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kW16) return;
    float v = 0.f;
    if (i < kH * kS1) {
        const int r = i / kS1, c = i % kS1;
        if (c < kIn) v = p[kW1 + r * kIn + c];
    } else {
        const int j = i - kH * kS1, which = j / (kH * kS2), jj = j % (kH * kS2);
        const int r = jj / kS2, c = jj % kS2;
        if (c < kH) v = p[(which == 0 ? kW2 : kW3) + r * kH + c];
    }
    w[i] = __float2bfloat16_rn(v);
}

// features of rays idx(j) = ((base + j) % n) * mult % n (f32, 80 columns)
// and their targets gathered alongside; mult coprime to n permutes the set
__global__ void k_features(DevWorld w, int32_t rox, int32_t roy, int32_t roz, const VxRay *rays,
                           unsigned long long n, unsigned long long base, unsigned long long mult,
                           unsigned long long count, float *feats, const float *tsrc,
                           float *tdst) {
    const unsigned long long j = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= count) return;
    const unsigned long long i = (((base + j) % n) * mult) % n;
    const int32_t ro[3] = {rox, roy, roz};
    const VxRay r = rays[i];
    const float o[3] = {r.org[0], r.org[1], r.org[2]};
    const float d[3] = {r.dir[0], r.dir[1], r.dir[2]};
    const uint64_t m = origin_chunk_word(w, ro, o);
    float *f = feats + j * kIn;
#pragma unroll 4
    for (int c = 0; c < kIn; ++c) f[c] = feature(o, d, m, c);
    if (tsrc) tdst[j] = tsrc[i];
}

// target: log of the plain DDA's first-hit t, or of the distance budget for a miss
__global__ void k_targets(const VxHitRecord *rec, size_t n, float max_dist, float *target) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool hit = (rec[i].flags & 1u) != 0u;
    target[i] = logf(fmaxf(hit ? rec[i].t : max_dist, 1.0f));
}

// rays of one camera through hashed random pixel positions
__global__ void k_pose_rays(VxCamera c, unsigned long long seed, size_t n, VxRay *rays,
                            float max_dist) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned long long h = seed + (i + 1) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 30; h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 27; h *= 0x94D049BB133111EBull;
    h ^= h >> 31;
    const float u = (float)(h & 0xFFFFFFull) * (1.0f / 16777216.0f);
    const float v = (float)((h >> 24) & 0xFFFFFFull) * (1.0f / 16777216.0f);
    const float ax = (u * 2.0f - 1.0f) * c.tan_half_fov * (c.res_x / c.res_y);
    const float by = (1.0f - v * 2.0f) * c.tan_half_fov;
    const float x = (c.forward[0] + c.right[0] * ax) + c.up[0] * by;
    const float y = (c.forward[1] + c.right[1] * ax) + c.up[1] * by;
    const float z = (c.forward[2] + c.right[2] * ax) + c.up[2] * by;
    const float l = sqrtf(x * x + y * y + z * z);
    VxRay r;
    r.org[0] = c.origin[0]; r.org[1] = c.origin[1]; r.org[2] = c.origin[2];
    r.dir[0] = x / l; r.dir[1] = y / l; r.dir[2] = z / l;
    r.tmax = max_dist;
    r.kind = 0;
    rays[i] = r;
}

unsigned nblk(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

cudaError_t mlp_alloc(Mlp &m) {
    cudaError_t e = cudaMalloc(&m.p, kMlpFloats * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m.g, kMlpFloats * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m.m, kMlpFloats * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m.v, kMlpFloats * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m.w16, kW16 * sizeof(uint16_t));
    if (e == cudaSuccess) e = cudaMalloc(&m.loss, sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(m.m, 0, kMlpFloats * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(m.v, 0, kMlpFloats * sizeof(float));
    return e;
}

void mlp_free(Mlp &m) {
    for (float *q : {m.p, m.g, m.m, m.v, m.partial, m.loss})
        if (q) cudaFree(q);
    if (m.w16) cudaFree(m.w16);
    m = Mlp();
}

cudaError_t mlp_sync_bf16(Mlp &m, cudaStream_t s) {
    k_to_bf16<<<nblk(kW16, 256), 256, 0, s>>>(m.p, reinterpret_cast<__nv_bfloat16 *>(m.w16));
    return cudaGetLastError();
}

cudaError_t mlp_grad(Mlp &m, const float *X, const float *target, int B, cudaStream_t s) {
    if (B <= 0) return cudaErrorInvalidValue;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess && !m.partial)
        e = cudaMalloc(&m.partial, (size_t)sms * (kMlpFloats + 1) * sizeof(float));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_train_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kTrainSmem);
    if (e != cudaSuccess) return e;
    const int grid = std::min(sms, (B + kTs - 1) / kTs);
    k_train_grad<<<grid, 256, kTrainSmem, s>>>(m.p, X, target, B, m.partial);
    k_train_reduce<<<nblk(kMlpFloats + 1, 32), 256, 0, s>>>(m.partial, grid, m.g, m.loss);
    return cudaGetLastError();
}

cudaError_t mlp_adam(Mlp &m, float lr, cudaStream_t s) {
    m.adam_t += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    k_adam<<<nblk(kMlpFloats, 256), 256, 0, s>>>(
        m.p, m.g, m.m, m.v, kMlpFloats, lr, b1, b2, 1e-8f,
        1.f - std::pow(b1, (float)m.adam_t), 1.f - std::pow(b2, (float)m.adam_t));
    return cudaGetLastError();
}

// Grid of the inference kernel: one 16-ray pass per warp (4 per CTA), at
// most eight CTAs per SM; larger batches loop.
static unsigned infer_blocks(size_t n) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t passes = (n + 15) / 16;  // 4 warps per block
    return (unsigned)std::max<size_t>(1, std::min<size_t>((passes + 3) / 4, (size_t)sms * 8));
}

cudaError_t mlp_infer_frame(const Mlp &m, const DevWorld &w, const VxCamera &cam,
                            const int32_t ro[3], uint32_t bw, uint32_t bh, float *out,
                            cudaStream_t s) {
    InferArgs a{};
    a.w = reinterpret_cast<const __nv_bfloat16 *>(m.w16);
    a.f32 = m.p;
    a.cam = cam;
    a.W = (uint32_t)cam.res_x;
    a.blk_w = bw ? bw : 1u;
    a.blk_h = bh ? bh : 1u;
    a.bw = (a.W + a.blk_w - 1u) / a.blk_w;
    a.n = a.bw * (((uint32_t)cam.res_y + a.blk_h - 1u) / a.blk_h);
    a.world = w;
    a.ro[0] = ro[0]; a.ro[1] = ro[1]; a.ro[2] = ro[2];
    a.out = out;
    if (a.n == 0) return cudaSuccess;
    k_mlp_infer<true><<<infer_blocks(a.n), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t mlp_infer_features(const Mlp &m, const float *feats, size_t n, float *out,
                               cudaStream_t s) {
    InferArgs a{};
    a.w = reinterpret_cast<const __nv_bfloat16 *>(m.w16);
    a.f32 = m.p;
    a.feats = feats;
    a.n = (uint32_t)n;
    a.out = out;
    if (n == 0) return cudaSuccess;
    k_mlp_infer<false><<<infer_blocks(n), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t mlp_features(const DevWorld &w, const int32_t ro[3], const VxRay *rays, size_t n,
                         uint64_t base, uint64_t mult, size_t count, float *feats,
                         const float *targets_src, float *targets_dst, cudaStream_t s) {
    if (count == 0 || n == 0) return cudaSuccess;
    k_features<<<nblk(count, 128), 128, 0, s>>>(w, ro[0], ro[1], ro[2], rays, n, base, mult,
                                                count, feats, targets_src, targets_dst);
    return cudaGetLastError();
}

cudaError_t mlp_targets(const VxHitRecord *rec, size_t n, float max_dist, float *target,
                        cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_targets<<<nblk(n, 256), 256, 0, s>>>(rec, n, max_dist, target);
    return cudaGetLastError();
}

cudaError_t mlp_pose_rays(const VxCamera &c, uint64_t seed, size_t n, VxRay *rays, float max_dist,
                          cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_pose_rays<<<nblk(n, 256), 256, 0, s>>>(c, seed, n, rays, max_dist);
    return cudaGetLastError();
}

}  // namespace vx
