// encoder.cu — the document encoder of the learned Metropolis-Hastings
// proposal: embedding bag -> 2 x 512 GELU MLP -> softmax over K topics, its
// backward pass and Adam, on the tensor-core GEMM of gemm.cu; and the C entry
// points of the GEMM and of the encoder.
//
// Per batch of Bp rows (the batch rounded up to 128; rows past the batch are
// zero and carry no gradient):
//   forward   X0 = embbag(E)                         [Bp x 256]  BF16 (+ X0^T)
//             P1 = X0 W1^T + b1, H1 = GELU(P1)       [Bp x 512]  FP32 / BF16 (+ H1^T)
//             P2 = H1 W2^T + b2, H2 = GELU(P2)       [Bp x 512]
//             Z  = H2 W3^T + b3, q = softmax(Z)      [Bp x K]
//   backward  dZ = (q - target) / B                  BF16 (+ dZ^T), db3 = column sums
//             dW3 = dZ^T H2                          GEMM(dZ^T, H2^T)
//             dP2 = (dZ W3) * GELU'(P2)              GEMM(dZ, W3^T), db2 = column sums
//             dW2 = dP2^T H1,  dP1 = (dP2 W2) * GELU'(P1), db1
//             dW1 = dP1^T X0,  dX0 = dP1 W1          FP32
//             dE[w] = sum of dX0[b] / L_b over the tokens of w in the batch
//                   (tokens grouped by word, one write per embedding row)
// The weight gradients split their K range (the batch) over several CTAs
// per tile.  Every GEMM is C = A B^T with both operands K-major, so each weight is kept
// in BF16 twice (W and W^T) and each activation that feeds a weight gradient
// is written transposed by the epilogue that produces it.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <vector>

#include "device_util.cuh"
#include "encoder.cuh"
#include "gemm.cuh"
#include "internal.h"
#include "philox.h"

using bf16 = __nv_bfloat16;

namespace culda {
namespace {

constexpr int kE = CULDA_ENC_EMBED, kH = CULDA_ENC_HIDDEN;
constexpr int kNumTensors = 7;

// ------------------------------------------------------------------ kernels
__global__ void init_uniform_kernel(int64_t n, float *dst, float scale, uint64_t seed, uint32_t tensor) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = scale * (2.0f * uniform_from_bits(philox_token(seed, (uint64_t)i, tensor, kPurposeWeights)) - 1.0f);
}

__global__ void to_bf16_kernel(int64_t n, const float *src, bf16 *dst) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = __float2bfloat16_rn(src[i]);
}

// out[c][r] = in[r][c] for an [R x C] matrix, through 32 x 32 shared tiles.
__global__ void transpose_bf16_kernel(int R, int C, const float *in, bf16 *out) {
    __shared__ float tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int r = r0 + i, c = c0 + threadIdx.x;
        if (r < R && c < C) tile[i][threadIdx.x] = in[(size_t)r * C + c];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int c = c0 + i, r = r0 + threadIdx.x;
        if (r < R && c < C) out[(size_t)c * R + r] = __float2bfloat16_rn(tile[threadIdx.x][i]);
    }
}

__device__ __forceinline__ void unpack8(const uint4 &v, float f[8]) {
    const bf16 *h = reinterpret_cast<const bf16 *>(&v);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __bfloat162float(h[i]);
}

// 16 bytes from global to shared memory, asynchronously (zeros when !valid).
__device__ __forceinline__ void copy16_async(void *dst, const void *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}

// One CTA per batch row: its 8 warps take contiguous eighths of the document's
// tokens, then the partial sums are added in warp order.  Lane l owns columns
// 8l .. 8l+7.  The 512-byte rows come from all over the L2, so what counts is
// how many are in flight: each warp keeps kBagRows of them on their way into a
// ring in shared memory (a lane reads only the bytes it copied itself, so the
// ring needs no barrier), 196 KB per SM.  For 4000 documents of 204 tokens (the
// longest 3200), 418 MB of rows: 134 us with 8 rows in registers at 91
// registers and 16 warps per SM, 98 us with 8 at 64 registers, 81 us with 16
// at 128 registers, 64 us in this form (71 us with 16 rows and 24 warps).  A
// grid of one CTA per row, so a long document holds back no row behind it.
// The loop over rows has one turn by that grid; without it the compiler takes
// another schedule: 67 us, 236 instead of 223 for 16384 such documents, but 495
// instead of 542 for 4000 of Pareto lengths around 300.
constexpr int kBagRows = 12, kBagGroup = 4;  // rows on their way per warp, rows per commit group
constexpr int kBagGroups = kBagRows / kBagGroup;
constexpr size_t kBagSmem = (size_t)8 * kBagRows * kE * sizeof(bf16);

__global__ void __launch_bounds__(256) embbag_fwd_kernel(int batch, int rows, const int32_t *__restrict__ docs,
                                                         const int64_t *__restrict__ doc_ptr,
                                                         const int32_t *__restrict__ words, int V,
                                                         const bf16 *__restrict__ emb, bf16 *X0, bf16 *X0t, int32_t *error) {
    extern __shared__ __align__(16) uint4 bag_ring[];
    __shared__ __align__(16) float part[8][kE];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4 *table = reinterpret_cast<const uint4 *>(emb) + lane;
    uint4 *ring = bag_ring + warp * kBagRows * 32 + lane;  // row r of the ring: ring[32 r]
    for (int b = blockIdx.x; b < rows; b += gridDim.x) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        int64_t t0 = 0, t1 = 0;
        if (b < batch) {
            const int d = docs ? docs[b] : b;
            t0 = doc_ptr[d];
            t1 = doc_ptr[d + 1];
            const int64_t per = (t1 - t0 + 7) / 8;
            const int64_t w0 = min(t1, t0 + per * warp);
            const int n = (int)(min(t1, w0 + per) - w0);
            const int32_t *ids = words + w0;
            const int groups = (n + kBagGroup - 1) / kBagGroup;
            int cur = 0, next = lane < n ? ids[lane] : 0;  // the word ids of 32 tokens, and of the 32 after them
            unsigned ok = 0u;
            for (int g = 0; g < groups + kBagGroups; ++g) {
                uint4 *slot = ring + (g % kBagGroups) * kBagGroup * 32;
                if (g >= kBagGroups) {
                    // rows are added in token order; one that was left out adds zero, which keeps a sum's bits
                    asm volatile("cp.async.wait_group %0;" ::"n"(kBagGroups - 1) : "memory");
#pragma unroll
                    for (int u = 0; u < kBagGroup; ++u) {
                        float f[8];
                        unpack8(slot[32 * u], f);
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[i] += f[i];
                    }
                }
                if (g < groups) {
                    const int j = g * kBagGroup;
                    if (j % 32 == 0) {
                        cur = next;
                        next = j + 32 + lane < n ? ids[j + 32 + lane] : 0;
                        const bool in = j + lane < n, good = in && (unsigned)cur < (unsigned)V;
                        if (in && !good) atomicOr(error, kErrWordRange);
                        ok = __ballot_sync(0xffffffffu, good);
                    }
#pragma unroll
                    for (int u = 0; u < kBagGroup; ++u) {
                        const int w = __shfl_sync(0xffffffffu, cur, (j + u) & 31);
                        const bool good = (ok >> ((j + u) & 31)) & 1u;
                        copy16_async(slot + 32 * u, table + (size_t)(good ? w : 0) * (kE / 8), good);
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
        }
        reinterpret_cast<float4 *>(part[warp])[2 * lane] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        reinterpret_cast<float4 *>(part[warp])[2 * lane + 1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        __syncthreads();
        // column threadIdx.x of the row: the partial sums in warp order
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += part[w][threadIdx.x];
        const float inv = t1 > t0 ? 1.0f / (float)(t1 - t0) : 0.f;
        const bf16 mean = __float2bfloat16_rn(sum * inv);
        X0[(size_t)b * kE + threadIdx.x] = mean;
        if (X0t) X0t[(size_t)threadIdx.x * rows + b] = mean;  // for the weight gradient
        __syncthreads();  // part is rewritten by the next row
    }
}

// The embedding gradient: the batch's (word, row) pairs are laid out in row
// order (a scan of the row lengths), sorted by word (a radix sort, stable, so
// a word's tokens stay in row order), and the sorted list is cut into chunks
// of 32 tokens.  A warp walks its chunk in order, summing dX0[b] / L_b per
// word in registers.  A word whose tokens all lie in the chunk is written with
// plain stores; a word whose run crosses the chunk's first or last token (the
// frequent ones) adds each chunk's partial sum with one vector atomic per
// lane.  gE holds zeros before the pass; words outside [0, V) sort last under
// the key V and are skipped.  So a word's terms are added in one order, and its
// row repeats bit for bit, unless it spans three chunks or more.  (Vector
// reductions straight to the words' rows need no sort, 24 us instead of 79 for
// 102k tokens, but add every word's terms in the order of arrival, rounded once
// more: at 1024 documents two runs then differ in 16% of the gradient's values
// instead of 0.3%, and by 4.5e-7 instead of 2.4e-7 in norm.)

// len[b] = L_b (for the scan of row offsets) and inv_len[b] = 1 / L_b.
__global__ void bag_rows_kernel(int batch, const int32_t *__restrict__ docs, const int64_t *__restrict__ doc_ptr,
                                int64_t *len, float *inv_len) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < batch; b += gridDim.x * blockDim.x) {
        const int d = docs ? docs[b] : b;
        const int64_t L = max((int64_t)0, (int64_t)(doc_ptr[d + 1] - doc_ptr[d]));
        len[b] = L;
        inv_len[b] = L > 0 ? 1.0f / (float)L : 0.f;
    }
}

// key[off[b] + j] = word of the j-th token of row b (V when out of range), val = b.
__global__ void __launch_bounds__(256) bag_pairs_kernel(int batch, const int32_t *__restrict__ docs,
                                                        const int64_t *__restrict__ doc_ptr,
                                                        const int32_t *__restrict__ words, int V,
                                                        const int64_t *__restrict__ off, int32_t *key, int32_t *val) {
    for (int b = blockIdx.x; b < batch; b += gridDim.x) {
        const int d = docs ? docs[b] : b;
        const int64_t t0 = doc_ptr[d], t1 = doc_ptr[d + 1];
        const int64_t o = off[b];
        for (int64_t t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
            const int w = words[t];
            key[o + (t - t0)] = (unsigned)w < (unsigned)V ? w : V;
            val[o + (t - t0)] = b;
        }
    }
}

// Warp per chunk of 32 sorted tokens; each lane holds 8 of the 256 columns.
__global__ void embbag_bwd_grouped_kernel(int64_t n, int V, const int32_t *__restrict__ wid,
                                          const int32_t *__restrict__ rows, const float *__restrict__ inv_len,
                                          const float *__restrict__ dX0, float *gE) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t c0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; c0 < n; c0 += nw * 32) {
        const int cn = (int)min((int64_t)32, n - c0);
        const int my_w = lane < cn ? wid[c0 + lane] : V;
        const int my_b = lane < cn ? rows[c0 + lane] : 0;
        const float my_s = lane < cn ? inv_len[my_b] : 0.f;
        // does the chunk's first (last) run continue from the chunk before (after) it?
        const int w_before = c0 > 0 ? wid[c0 - 1] : -1;
        const int w_after = c0 + cn < n ? wid[c0 + cn] : -1;
        const int first_w = __shfl_sync(0xffffffffu, my_w, 0), last_w = __shfl_sync(0xffffffffu, my_w, cn - 1);
        // the chunk's dX0 rows, 2 x 16 bytes per lane each, loaded 8 at a time ahead of their use
        float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
        float4 r0[8], r1[8];
        for (int j = 0; j < cn; ++j) {
            if ((j & 7) == 0) {
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int bj = __shfl_sync(0xffffffffu, my_b, (j + u) & 31);
                    const float4 *q = reinterpret_cast<const float4 *>(dX0 + (size_t)bj * kE) + 2 * lane;
                    const bool in = j + u < cn;
                    r0[u] = in ? q[0] : make_float4(0.f, 0.f, 0.f, 0.f);
                    r1[u] = in ? q[1] : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            const int w = __shfl_sync(0xffffffffu, my_w, j);
            const float sc = __shfl_sync(0xffffffffu, my_s, j);
            float4 g0 = r0[0], g1 = r1[0];
#pragma unroll
            for (int u = 1; u < 8; ++u)
                if ((j & 7) == u) {
                    g0 = r0[u];
                    g1 = r1[u];
                }
            a0.x += g0.x * sc;
            a0.y += g0.y * sc;
            a0.z += g0.z * sc;
            a0.w += g0.w * sc;
            a1.x += g1.x * sc;
            a1.y += g1.y * sc;
            a1.z += g1.z * sc;
            a1.w += g1.w * sc;
            const int wn = __shfl_sync(0xffffffffu, my_w, (j + 1) & 31);
            if (j + 1 == cn || wn != w) {  // the end of this word's run in the chunk
                if (w < V) {
                    float4 *dst = reinterpret_cast<float4 *>(gE + (size_t)w * kE) + 2 * lane;
                    const bool shared = (w == first_w && w == w_before) || (w == last_w && w == w_after);
                    if (!shared) {  // the whole word: no other chunk adds to it
                        dst[0] = a0;
                        dst[1] = a1;
                    } else {
                        atomicAdd(dst, a0);
                        atomicAdd(dst + 1, a1);
                    }
                }
                a0 = make_float4(0.f, 0.f, 0.f, 0.f);
                a1 = a0;
            }
        }
    }
}

// Softmax of each row of Z [rows x K] and, against the target, dZ = (q - t) /
// batch (BF16) with its transpose, the column sums of dZ (db3) and the summed
// cross-entropy.  A CTA takes kXentRows rows, a warp each; lane l holds columns
// l, l+32, ... of its row in registers, so Z and the target are read once.  The
// rows' gradients meet in shared memory (FP32), from where a thread per column
// adds them up in row order and writes the transpose's 16 bytes.  (With a pass
// over Z per reduction, shared atomics for the column sums and a transpose
// kernel of its own: 24.5 + 3.9 us for 1024 rows of 1024; this form 8.4 us.)
constexpr int kXentRows = 8;

template <int N>  // columns per lane: K <= 32 N
__global__ void __launch_bounds__(256) softmax_xent_kernel(int batch, int rows, int K, const float *__restrict__ Z,
                                                           EncoderTarget tg, const int32_t *__restrict__ docs,
                                                           const int64_t *__restrict__ doc_ptr, float *probs,
                                                           bf16 *dZ, bf16 *dZt, float *db3, double *loss) {
    extern __shared__ float grad[];  // [kXentRows][K], only with a target
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.x * kXentRows + warp, n = K / 32;
    float *grow = grad + (size_t)warp * K;
    if (b < batch) {
        const float *zr = Z + (size_t)b * K;
        float z[N];
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i < n) {
                z[i] = zr[lane + 32 * i];
                mx = fmaxf(mx, z[i]);
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float se = 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i < n) se += __expf(z[i] - mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
        const float lse = mx + __logf(se), inv_se = 1.0f / se;
        if (probs) {
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (i < n) probs[(size_t)b * K + lane + 32 * i] = __expf(z[i] - mx) * inv_se;
        }
        if (dZ) {
            const float inv_batch = 1.0f / (float)batch;
            const int d = docs ? docs[b] : b;
            float tscale = 0.f;
            if (!tg.dense) {
                const float L = (float)(doc_ptr[d + 1] - doc_ptr[d]);
                tscale = 1.0f / (L + (float)K * tg.alpha);
            }
            const float *tr = tg.dense ? tg.dense + (size_t)b * K : tg.acc + (size_t)d * K;
            float l = 0.f;
            // 16 targets are loaded before any gradient is stored: the stores
            // could alias them for all the compiler knows
#pragma unroll
            for (int i0 = 0; i0 < N; i0 += 16) {
                float t[16];
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    if (i0 + u < n) t[u] = tr[lane + 32 * (i0 + u)];
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    if (i0 + u < n) {
                        const int k = lane + 32 * (i0 + u);
                        if (!tg.dense) t[u] = (t[u] * tg.inv_n + tg.alpha) * tscale;
                        const float g = (__expf(z[i0 + u] - mx) * inv_se - t[u]) * inv_batch;
                        grow[k] = g;
                        dZ[(size_t)b * K + k] = __float2bfloat16_rn(g);
                        l += t[u] * (lse - z[i0 + u]);
                    }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (lane == 0 && l != 0.f) atomicAdd(loss, (double)l);
        }
    } else if (dZ) {  // padding row: no gradient (rows is a multiple of 128, so a CTA's rows are all there)
        for (int k = lane; k < K; k += 32) {
            grow[k] = 0.f;
            dZ[(size_t)b * K + k] = __float2bfloat16_rn(0.f);
        }
    }
    if (!dZ) return;
    __syncthreads();
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        float sum = 0.f;
        uint4 h;
        bf16 *hb = reinterpret_cast<bf16 *>(&h);
#pragma unroll
        for (int r = 0; r < kXentRows; ++r) {
            const float g = grad[(size_t)r * K + k];
            sum += g;
            hb[r] = __float2bfloat16_rn(g);
        }
        *reinterpret_cast<uint4 *>(dZt + (size_t)k * rows + blockIdx.x * kXentRows) = h;
        if (sum != 0.f) atomicAdd(&db3[k], sum);
    }
}

// ------------------------------------------------------------------- Adam
struct AdamStep {
    float lr, b1, b2, eps, c1, c2;

    __device__ __forceinline__ float operator()(float p, float g, float &m, float &v) const {
        m = b1 * m + (1.0f - b1) * g;
        v = b2 * v + (1.0f - b2) * g * g;
        return p - lr * (m * c1) / (sqrtf(v * c2) + eps);
    }
};

// One Adam step on every weight and the BF16 copies the next pass reads, in one
// pass over memory (30 bytes a weight).  The first flat_blocks CTAs take the
// embeddings, then the biases, 16 bytes per access; the others a 32 x 32 tile
// of W1, W2 or W3 each, whose transposed copy goes through shared memory.  (An
// Adam kernel of scalar accesses, four conversions and three transposes after
// it: 70 us and 8 launches at 6M weights; this form 32 us.)
struct AdamParams {
    float *p;
    const float *g;
    float *m, *v;
    int64_t embed;          // elements of E, the first in the blocks
    int64_t bias[3];        // offsets of b1, b2, b3
    int bias_n[3];
    bf16 *emb_bf;
    int64_t w[3];           // offsets of W1, W2, W3
    int rows[3], cols[3];   // multiples of 32
    bf16 *wb[3], *wt[3];
    int flat_blocks;
};

__global__ void __launch_bounds__(256) adam_kernel(const AdamParams a, const AdamStep step) {
    __shared__ float tile[32][33];
    const int tid = threadIdx.x;
    if ((int)blockIdx.x < a.flat_blocks) {
        const int64_t n4 = a.embed / 4, stride = (int64_t)a.flat_blocks * 256;
        for (int64_t i = (int64_t)blockIdx.x * 256 + tid; i < n4; i += stride) {
            float4 p = reinterpret_cast<const float4 *>(a.p)[i], m = reinterpret_cast<const float4 *>(a.m)[i],
                   v = reinterpret_cast<const float4 *>(a.v)[i];
            const float4 g = reinterpret_cast<const float4 *>(a.g)[i];
            p.x = step(p.x, g.x, m.x, v.x);
            p.y = step(p.y, g.y, m.y, v.y);
            p.z = step(p.z, g.z, m.z, v.z);
            p.w = step(p.w, g.w, m.w, v.w);
            reinterpret_cast<float4 *>(a.p)[i] = p;
            reinterpret_cast<float4 *>(a.m)[i] = m;
            reinterpret_cast<float4 *>(a.v)[i] = v;
            uint2 h;
            reinterpret_cast<__nv_bfloat162 *>(&h)[0] = __floats2bfloat162_rn(p.x, p.y);
            reinterpret_cast<__nv_bfloat162 *>(&h)[1] = __floats2bfloat162_rn(p.z, p.w);
            reinterpret_cast<uint2 *>(a.emb_bf)[i] = h;
        }
        for (int t = 0; t < 3; ++t)
            for (int i = blockIdx.x * 256 + tid; i < a.bias_n[t]; i += (int)stride) {
                const int64_t o = a.bias[t] + i;
                a.p[o] = step(a.p[o], a.g[o], a.m[o], a.v[o]);
            }
        return;
    }
    int x = blockIdx.x - a.flat_blocks, t = 0;
    while (x >= (a.rows[t] / 32) * (a.cols[t] / 32)) x -= (a.rows[t] / 32) * (a.cols[t] / 32), ++t;
    const int R = a.rows[t], C = a.cols[t], r0 = x / (C / 32) * 32, c0 = x % (C / 32) * 32;
    const int c = tid & 31;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = (tid >> 5) + 8 * i;
        const int64_t e = (int64_t)(r0 + r) * C + c0 + c, o = a.w[t] + e;
        const float p = step(a.p[o], a.g[o], a.m[o], a.v[o]);
        a.p[o] = p;
        a.wb[t][e] = __float2bfloat16_rn(p);
        tile[r][c] = p;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = (tid >> 5) + 8 * i;  // column of the tile
        a.wt[t][(int64_t)(c0 + r) * R + r0 + c] = __float2bfloat16_rn(tile[c][r]);
    }
}

}  // namespace
}  // namespace culda

using namespace culda;

// What an encoder's calls read back, in pinned memory.
struct EncoderReadback {
    int64_t tokens;  // of a training batch, where the caller gave none
    double loss;     // with the error word, as they lie on the device
    int32_t error;
};

// ------------------------------------------------------------------ object
struct culda_encoder {
    int device = 0;
    int V = 0, K = 0, Bmax = 0;  // Bmax: rows, a multiple of 128
    float lr = 1e-3f, b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    int64_t steps = 0;
    int64_t off[kNumTensors + 1] = {};  // offsets of the tensors in the FP32 blocks
    float *params = nullptr, *grads = nullptr, *adam_m = nullptr, *adam_v = nullptr;
    bf16 *emb_bf = nullptr, *W1 = nullptr, *W1t = nullptr, *W2 = nullptr, *W2t = nullptr, *W3 = nullptr,
         *W3t = nullptr;
    bf16 *X0 = nullptr, *X0t = nullptr, *H1 = nullptr, *H1t = nullptr, *H2 = nullptr, *H2t = nullptr;
    bf16 *dZ = nullptr, *dZt = nullptr, *dP2 = nullptr, *dP2t = nullptr, *dP1 = nullptr, *dP1t = nullptr;
    float *P1 = nullptr, *P2 = nullptr, *Z = nullptr, *dX0 = nullptr;
    double *d_loss = nullptr;
    int32_t *d_error = nullptr;
    // the batch's (word, row) pairs sorted by word, for the embedding gradient
    int64_t *bag_len = nullptr, *bag_off = nullptr;  // [Bmax + 1] row lengths and their exclusive scan
    float *bag_inv_len = nullptr;                    // [Bmax] 1 / L of every batch row
    int32_t *bag_key = nullptr, *bag_val = nullptr;  // [bag_cap] pairs in row order
    int32_t *bag_wid = nullptr, *bag_rows = nullptr; // [bag_cap] the pairs sorted by word
    int64_t bag_cap = 0;
    void *scan_tmp = nullptr, *sort_tmp = nullptr;
    size_t scan_tmp_bytes = 0, sort_tmp_bytes = 0;
    int key_bits = 1;                                // bits of the keys 0..V
    EncoderReadback *h_back = nullptr;               // pinned
    cudaEvent_t counted = nullptr;                   // h_back->tokens has arrived
    std::vector<void *> allocs;

    float *tensor(int t) { return params + off[t]; }
    float *grad(int t) { return grads + off[t]; }
};

namespace culda {
namespace {

template <class T>
cudaError_t ealloc(culda_encoder *e, T **p, size_t n) {
    const cudaError_t r =
        (cudaError_t)device_malloc(reinterpret_cast<void **>(p), std::max<size_t>(n, 1) * sizeof(T));
    if (r == cudaSuccess) e->allocs.push_back(*p);
    return r;
}

int fail_enc(int code, const char *fmt, const char *what) {
    set_global_error(fmt, what);
    return code;
}

void free_encoder(culda_encoder *e) {
    for (void *q : e->allocs) cudaFree(q);
    if (e->counted) cudaEventDestroy(e->counted);
    if (e->h_back) pinned_slot_put(e->h_back);
    delete e;
}

#define ECK(x)                                                                   \
    do {                                                                         \
        cudaError_t _e = (x);                                                    \
        if (_e != cudaSuccess) return fail_enc(CULDA_ERR_CUDA, "encoder: %s", cudaGetErrorString(_e)); \
    } while (0)

cudaError_t transpose_to_bf16(int R, int C, const float *in, bf16 *out, cudaStream_t s) {
    transpose_bf16_kernel<<<dim3((C + 31) / 32, (R + 31) / 32), dim3(32, 8), 0, s>>>(R, C, in, out);
    return cudaGetLastError();
}

// BF16 copies of the weights (and the transposes the backward pass reads).
cudaError_t refresh_bf16(culda_encoder *e, cudaStream_t s) {
    const int64_t ne = (int64_t)e->V * kE;
    to_bf16_kernel<<<grid_for(ne), 256, 0, s>>>(ne, e->tensor(CULDA_ENC_E), e->emb_bf);
    to_bf16_kernel<<<grid_for((int64_t)kH * kE), 256, 0, s>>>((int64_t)kH * kE, e->tensor(CULDA_ENC_W1), e->W1);
    to_bf16_kernel<<<grid_for((int64_t)kH * kH), 256, 0, s>>>((int64_t)kH * kH, e->tensor(CULDA_ENC_W2), e->W2);
    to_bf16_kernel<<<grid_for((int64_t)e->K * kH), 256, 0, s>>>((int64_t)e->K * kH, e->tensor(CULDA_ENC_W3), e->W3);
    cudaError_t r = transpose_to_bf16(kH, kE, e->tensor(CULDA_ENC_W1), e->W1t, s);
    if (r == cudaSuccess) r = transpose_to_bf16(kH, kH, e->tensor(CULDA_ENC_W2), e->W2t, s);
    if (r == cudaSuccess) r = transpose_to_bf16(e->K, kH, e->tensor(CULDA_ENC_W3), e->W3t, s);
    return r;
}

cudaError_t gemm(int M, int N, int K, const bf16 *A, const bf16 *B, int epi, const GemmEpilogue &ep, int32_t *err,
                 cudaStream_t s) {
    return gemm_bf16_nt(M, N, K, A, K, B, K, epi, ep, err, s);
}

template <int N>
cudaError_t softmax_xent_n(int batch, int rows, int K, const float *Z, const EncoderTarget &tg, const int32_t *docs,
                           const int64_t *doc_ptr, float *probs, bf16 *dZ, bf16 *dZt, float *db3, double *loss,
                           cudaStream_t s) {
    const size_t smem = dZ ? (size_t)kXentRows * K * sizeof(float) : 0;
    const cudaError_t e = allow_smem(reinterpret_cast<const void *>(&softmax_xent_kernel<N>), smem);
    if (e != cudaSuccess) return e;
    softmax_xent_kernel<N><<<(rows + kXentRows - 1) / kXentRows, 256, smem, s>>>(batch, rows, K, Z, tg, docs, doc_ptr,
                                                                                 probs, dZ, dZt, db3, loss);
    return cudaGetLastError();
}

// A lane's columns are in registers, so the kernel is built per power of two of K.
cudaError_t softmax_xent(int batch, int rows, int K, const float *Z, const EncoderTarget &tg, const int32_t *docs,
                         const int64_t *doc_ptr, float *probs, bf16 *dZ, bf16 *dZt, float *db3, double *loss,
                         cudaStream_t s) {
    auto run = K <= 512    ? softmax_xent_n<16>
               : K <= 1024 ? softmax_xent_n<32>
               : K <= 2048 ? softmax_xent_n<64>
                           : softmax_xent_n<128>;
    return run(batch, rows, K, Z, tg, docs, doc_ptr, probs, dZ, dZt, db3, loss, s);
}

// Weight gradients: M x N is a few tiles and K the batch, so the K range is
// cut into slices (at least 4 k-blocks each), as many as fill the two CTAs
// per SM in one wave; the slices add into the zeroed gradient.
cudaError_t gemm_wgrad(int M, int N, int K, const bf16 *A, const bf16 *B, GemmEpilogue ep, int32_t *err,
                       cudaStream_t s) {
    int sms = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int tiles = (M / 128) * (N / 128);
    const int by_k = std::max(1, (K / 64) / 4);
    ep.k_splits = std::max(1, std::min(by_k, (2 * sms) / tiles));
    return gemm_bf16_nt(M, N, K, A, K, B, K, kEpiF32, ep, err, s);
}

}  // namespace

int encoder_k(const culda_encoder *e) { return e->K; }
int encoder_num_words(const culda_encoder *e) { return e->V; }
float *encoder_tensor(culda_encoder *e, int t) { return e->tensor(t); }
int encoder_refresh(culda_encoder *e, cudaStream_t s) {
    ECK(refresh_bf16(e, s));
    return CULDA_OK;
}
int encoder_max_batch(const culda_encoder *e) { return e->Bmax; }
int32_t *encoder_error_word(culda_encoder *e) { return e->d_error; }

int encoder_pass(culda_encoder *e, int batch, const int32_t *docs, const int64_t *doc_ptr, const int32_t *words,
                 const EncoderTarget *target, bool update, float *probs, cudaStream_t s, int64_t batch_tokens) {
    if (batch <= 0 || batch > e->Bmax || !doc_ptr || !words)
        return fail_enc(CULDA_ERR_INVALID_ARG, "encoder: %s", "batch outside 1..max_batch or null CSR");
    if (target && !target->dense && !target->acc)
        return fail_enc(CULDA_ERR_INVALID_ARG, "encoder: %s", "target without data");
    ECK(cudaSetDevice(e->device));
    const int Bp = (batch + 127) & ~127, K = e->K;
    int32_t *err = e->d_error;
    if (target) {
        // where each row's (word, row) pairs go; their number is on its way to the host during the passes
        bag_rows_kernel<<<(batch + 255) / 256, 256, 0, s>>>(batch, docs, doc_ptr, e->bag_len, e->bag_inv_len);
        ECK(cudaGetLastError());
        ECK(cub::DeviceScan::ExclusiveSum(e->scan_tmp, e->scan_tmp_bytes, e->bag_len, e->bag_off, batch + 1, s));
        if (batch_tokens < 0) {
            ECK(cudaMemcpyAsync(&e->h_back->tokens, e->bag_off + batch, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
            ECK(cudaEventRecord(e->counted, s));
        }
    }
    // forward
    ECK(allow_smem(reinterpret_cast<const void *>(&embbag_fwd_kernel), kBagSmem));
    embbag_fwd_kernel<<<Bp, 256, kBagSmem, s>>>(batch, Bp, docs, doc_ptr, words, e->V, e->emb_bf,
                                                                 e->X0, target ? e->X0t : nullptr, err);
    ECK(cudaGetLastError());
    GemmEpilogue ep;
    ep.out_f32 = e->P1;
    ep.ldo = kH;
    ep.out_bf16 = e->H1;
    ep.out_bf16_t = e->H1t;
    ep.ld_t = Bp;
    ep.bias = e->tensor(CULDA_ENC_B1);
    ECK(gemm(Bp, kH, kE, e->X0, e->W1, kEpiBiasGelu, ep, err, s));
    ep.out_f32 = e->P2;
    ep.out_bf16 = e->H2;
    ep.out_bf16_t = e->H2t;
    ep.bias = e->tensor(CULDA_ENC_B2);
    ECK(gemm(Bp, kH, kH, e->H1, e->W2, kEpiBiasGelu, ep, err, s));
    GemmEpilogue ez;
    ez.out_f32 = e->Z;
    ez.ldo = K;
    ez.bias = e->tensor(CULDA_ENC_B3);
    ECK(gemm(Bp, K, kH, e->H2, e->W3, kEpiF32, ez, err, s));
    if (!target) {
        ECK(softmax_xent(batch, Bp, K, e->Z, EncoderTarget{}, docs, doc_ptr, probs, nullptr, nullptr, nullptr, nullptr,
                         s));
        return CULDA_OK;
    }
    // backward
    ECK(cudaMemsetAsync(e->grads, 0, sizeof(float) * (size_t)e->off[kNumTensors], s));
    ECK(softmax_xent(batch, Bp, K, e->Z, *target, docs, doc_ptr, probs, e->dZ, e->dZt, e->grad(CULDA_ENC_B3),
                     e->d_loss, s));
    GemmEpilogue gw;
    gw.ldo = kH;
    gw.out_f32 = e->grad(CULDA_ENC_W3);
    ECK(gemm_wgrad(K, kH, Bp, e->dZt, e->H2t, gw, err, s));  // dW3 = dZ^T H2
    GemmEpilogue gb;
    gb.ldo = kH;
    gb.ld_t = Bp;
    gb.pre = e->P2;
    gb.out_bf16 = e->dP2;
    gb.out_bf16_t = e->dP2t;
    gb.colsum = e->grad(CULDA_ENC_B2);
    ECK(gemm(Bp, kH, K, e->dZ, e->W3t, kEpiGeluBwd, gb, err, s));  // dP2 = (dZ W3) GELU'(P2)
    gw.out_f32 = e->grad(CULDA_ENC_W2);
    ECK(gemm_wgrad(kH, kH, Bp, e->dP2t, e->H1t, gw, err, s));  // dW2 = dP2^T H1
    gb.pre = e->P1;
    gb.out_bf16 = e->dP1;
    gb.out_bf16_t = e->dP1t;
    gb.colsum = e->grad(CULDA_ENC_B1);
    ECK(gemm(Bp, kH, kH, e->dP2, e->W2t, kEpiGeluBwd, gb, err, s));  // dP1 = (dP2 W2) GELU'(P1)
    GemmEpilogue g1;
    g1.ldo = kE;
    g1.out_f32 = e->grad(CULDA_ENC_W1);
    ECK(gemm_wgrad(kH, kE, Bp, e->dP1t, e->X0t, g1, err, s));  // dW1 = dP1^T X0
    g1.out_f32 = e->dX0;
    ECK(gemm(Bp, kE, kH, e->dP1, e->W1t, kEpiF32, g1, err, s));  // dX0 = dP1 W1
    // the batch's (word, row) pairs sorted by word, then one pass over them
    if (batch_tokens < 0) {
        ECK(cudaEventSynchronize(e->counted));
        batch_tokens = e->h_back->tokens;
    }
    if (batch_tokens > INT_MAX)
        return fail_enc(CULDA_ERR_UNSUPPORTED, "encoder: %s", "a training batch of more than 2^31 - 1 tokens");
    if (batch_tokens > e->bag_cap) {
        ECK(cudaStreamSynchronize(s));
        for (void **q : {(void **)&e->bag_key, (void **)&e->bag_val, (void **)&e->bag_wid, (void **)&e->bag_rows,
                         &e->sort_tmp}) {
            if (*q) {
                cudaFree(*q);
                e->allocs.erase(std::find(e->allocs.begin(), e->allocs.end(), *q));
                *q = nullptr;
            }
        }
        const int64_t cap = std::min<int64_t>(std::max<int64_t>(batch_tokens, 2 * e->bag_cap), INT_MAX);
        e->bag_cap = 0;
        ECK(ealloc(e, &e->bag_key, (size_t)cap));
        ECK(ealloc(e, &e->bag_val, (size_t)cap));
        ECK(ealloc(e, &e->bag_wid, (size_t)cap));
        ECK(ealloc(e, &e->bag_rows, (size_t)cap));
        e->sort_tmp_bytes = 0;
        ECK(cub::DeviceRadixSort::SortPairs(nullptr, e->sort_tmp_bytes, e->bag_key, e->bag_wid, e->bag_val,
                                            e->bag_rows, (int)cap, 0, e->key_bits));
        uint8_t *tmp = nullptr;
        ECK(ealloc(e, &tmp, e->sort_tmp_bytes));
        e->sort_tmp = tmp;
        e->bag_cap = cap;
    }
    if (batch_tokens > 0) {
        bag_pairs_kernel<<<std::min(batch, 148 * 16), 256, 0, s>>>(batch, docs, doc_ptr, words, e->V, e->bag_off,
                                                                   e->bag_key, e->bag_val);
        ECK(cudaGetLastError());
        ECK(cub::DeviceRadixSort::SortPairs(e->sort_tmp, e->sort_tmp_bytes, e->bag_key, e->bag_wid, e->bag_val,
                                            e->bag_rows, (int)batch_tokens, 0, e->key_bits, s));
        embbag_bwd_grouped_kernel<<<grid_for(batch_tokens), 256, 0, s>>>(batch_tokens, e->V, e->bag_wid, e->bag_rows,
                                                                         e->bag_inv_len, e->dX0,
                                                                         e->grad(CULDA_ENC_E));
        ECK(cudaGetLastError());
    }
    if (update) {
        e->steps += 1;
        const float c1 = 1.0f / (1.0f - powf(e->b1, (float)e->steps));
        const float c2 = 1.0f / (1.0f - powf(e->b2, (float)e->steps));
        AdamParams a{};
        a.p = e->params;
        a.g = e->grads;
        a.m = e->adam_m;
        a.v = e->adam_v;
        a.embed = e->off[CULDA_ENC_E + 1];
        a.emb_bf = e->emb_bf;
        const int bias[3] = {CULDA_ENC_B1, CULDA_ENC_B2, CULDA_ENC_B3};
        const int weight[3] = {CULDA_ENC_W1, CULDA_ENC_W2, CULDA_ENC_W3};
        const int rows[3] = {kH, kH, K}, cols[3] = {kE, kH, kH};
        bf16 *wb[3] = {e->W1, e->W2, e->W3}, *wt[3] = {e->W1t, e->W2t, e->W3t};
        int tiles = 0;
        for (int t = 0; t < 3; ++t) {
            a.bias[t] = e->off[bias[t]];
            a.bias_n[t] = (int)(e->off[bias[t] + 1] - e->off[bias[t]]);
            a.w[t] = e->off[weight[t]];
            a.rows[t] = rows[t];
            a.cols[t] = cols[t];
            a.wb[t] = wb[t];
            a.wt[t] = wt[t];
            tiles += (rows[t] / 32) * (cols[t] / 32);
        }
        a.flat_blocks = (int)std::min<int64_t>(148 * 8, (a.embed / 4 + 255) / 256);
        adam_kernel<<<a.flat_blocks + tiles, 256, 0, s>>>(a, AdamStep{e->lr, e->b1, e->b2, e->eps, c1, c2});
        ECK(cudaGetLastError());
    }
    return CULDA_OK;
}

int encoder_take_loss(culda_encoder *e, int batch_rows, double *loss, cudaStream_t s) {
    constexpr size_t kBytes = sizeof(double) + sizeof(int32_t);
    static_assert(offsetof(EncoderReadback, error) == offsetof(EncoderReadback, loss) + sizeof(double),
                  "the two are copied together");
    // Cleared before the call returns: the next pass may run on another stream.  Behind
    // a forward pass there is nothing to clear but its error word, if it set one (a
    // clearing behind every pass: 3 us of the 60 for one document).
    ECK(cudaMemcpyAsync(&e->h_back->loss, e->d_loss, kBytes, cudaMemcpyDeviceToHost, s));
    if (batch_rows > 0) ECK(cudaMemsetAsync(e->d_loss, 0, kBytes, s));
    ECK(cudaStreamSynchronize(s));
    const double h = e->h_back->loss;
    const int32_t err = e->h_back->error;
    if (batch_rows == 0 && (err || h != 0.0)) {
        ECK(cudaMemsetAsync(e->d_loss, 0, kBytes, s));
        ECK(cudaStreamSynchronize(s));
    }
    if (err) {
        char msg[96];
        snprintf(msg, sizeof msg, "encoder: device error 0x%x", err);
        return fail_enc(CULDA_ERR_DEVICE_STATE, "%s", msg);
    }
    if (loss) *loss = batch_rows > 0 ? h / (double)batch_rows : 0.0;
    return CULDA_OK;
}

}  // namespace culda

// ============================================================ C entry points
extern "C" int culda_gemm_bf16(const culda_gemm_args *a, void *stream) {
    if (!a) {
        set_global_error("culda_gemm_bf16: null arguments");
        return CULDA_ERR_INVALID_ARG;
    }
    GemmEpilogue ep;
    ep.out_f32 = a->out_f32;
    ep.ldo = a->ldo;
    ep.out_bf16 = reinterpret_cast<bf16 *>(a->out_bf16);
    ep.out_bf16_t = reinterpret_cast<bf16 *>(a->out_bf16_t);
    ep.ld_t = a->ld_t;
    ep.bias = a->bias;
    ep.pre = a->pre;
    ep.colsum = a->colsum;
    ep.alpha = a->alpha;
    ep.k_splits = a->k_splits > 0 ? a->k_splits : 1;
    if (const char *why = gemm_check(a->m, a->n, a->k, a->a, a->lda, a->b, a->ldb, a->epilogue, ep)) {
        set_global_error("culda_gemm_bf16: %s", why);
        return CULDA_ERR_INVALID_ARG;
    }
    const cudaError_t e = gemm_bf16_nt(a->m, a->n, a->k, a->a, a->lda, a->b, a->ldb, a->epilogue, ep, a->error,
                                       static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) {
        set_global_error("culda_gemm_bf16: %s", cudaGetErrorString(e));
        return e == cudaErrorNotSupported ? CULDA_ERR_UNSUPPORTED : CULDA_ERR_CUDA;
    }
    return CULDA_OK;
}

extern "C" int culda_encoder_create(const culda_encoder_params *p, culda_encoder **out) {
    if (!p || !out) return fail_enc(CULDA_ERR_INVALID_ARG, "culda_encoder_create: %s", "null argument");
    *out = nullptr;
    if (p->num_words <= 0 || p->k < 128 || p->k > 4096 || p->k % 128 || p->max_batch <= 0 || p->max_batch > 65536)
        return fail_enc(CULDA_ERR_INVALID_ARG, "culda_encoder_create: %s",
                        "num_words > 0, k a multiple of 128 in 128..4096, max_batch in 1..65536");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0)
        return fail_enc(CULDA_ERR_NO_DEVICE, "culda_encoder_create: %s", "no CUDA device");
    if (p->device < 0 || p->device >= ndev)
        return fail_enc(CULDA_ERR_INVALID_ARG, "culda_encoder_create: %s", "device out of range");
    culda_encoder *e = new culda_encoder;
    e->device = p->device;
    e->V = p->num_words;
    e->K = p->k;
    e->Bmax = (p->max_batch + 127) & ~127;
    if (p->lr > 0.f) e->lr = p->lr;
    if (p->beta1 > 0.f) e->b1 = p->beta1;
    if (p->beta2 > 0.f) e->b2 = p->beta2;
    if (p->eps > 0.f) e->eps = p->eps;
    const int64_t sizes[kNumTensors] = {(int64_t)e->V * kE, (int64_t)kH * kE, kH, (int64_t)kH * kH, kH,
                                        (int64_t)e->K * kH, e->K};
    for (int t = 0; t < kNumTensors; ++t) e->off[t + 1] = e->off[t] + sizes[t];
    const size_t np = (size_t)e->off[kNumTensors];
    const size_t B = (size_t)e->Bmax, K = (size_t)e->K;
    auto bail = [&](cudaError_t r) {
        free_encoder(e);
        return fail_enc(r == cudaErrorMemoryAllocation ? CULDA_ERR_OOM : CULDA_ERR_CUDA, "culda_encoder_create: %s",
                        cudaGetErrorString(r));
    };
    cudaError_t r = cudaSetDevice(e->device);
    if (r != cudaSuccess) return bail(r);
#define EALLOC(ptr, n)                 \
    r = ealloc(e, &(ptr), (size_t)(n)); \
    if (r != cudaSuccess) return bail(r)
    EALLOC(e->params, np);
    EALLOC(e->grads, np);
    EALLOC(e->adam_m, np);
    EALLOC(e->adam_v, np);
    EALLOC(e->emb_bf, (size_t)e->V * kE);
    EALLOC(e->W1, kH * kE);
    EALLOC(e->W1t, kH * kE);
    EALLOC(e->W2, kH * kH);
    EALLOC(e->W2t, kH * kH);
    EALLOC(e->W3, K * kH);
    EALLOC(e->W3t, K * kH);
    EALLOC(e->X0, B * kE);
    EALLOC(e->X0t, B * kE);
    EALLOC(e->H1, B * kH);
    EALLOC(e->H1t, B * kH);
    EALLOC(e->H2, B * kH);
    EALLOC(e->H2t, B * kH);
    EALLOC(e->dZ, B * K);
    EALLOC(e->dZt, B * K);
    EALLOC(e->dP2, B * kH);
    EALLOC(e->dP2t, B * kH);
    EALLOC(e->dP1, B * kH);
    EALLOC(e->dP1t, B * kH);
    EALLOC(e->P1, B * kH);
    EALLOC(e->P2, B * kH);
    EALLOC(e->Z, B * K);
    EALLOC(e->dX0, B * kE);
    EALLOC(e->d_loss, 2);  // the error word follows the loss, so one copy reads both
    e->d_error = reinterpret_cast<int32_t *>(e->d_loss + 1);
    EALLOC(e->bag_len, (size_t)B + 1);
    EALLOC(e->bag_off, (size_t)B + 1);
    EALLOC(e->bag_inv_len, B);
    while ((1u << e->key_bits) <= (unsigned)e->V) ++e->key_bits;  // keys 0..V
    r = cub::DeviceScan::ExclusiveSum(nullptr, e->scan_tmp_bytes, e->bag_len, e->bag_off, B + 1);
    if (r != cudaSuccess) return bail(r);
    {
        uint8_t *tmp = nullptr;
        EALLOC(tmp, e->scan_tmp_bytes);
        e->scan_tmp = tmp;
    }
    if (!(e->h_back = static_cast<EncoderReadback *>(pinned_slot_get()))) return bail(cudaErrorMemoryAllocation);
    r = cudaEventCreateWithFlags(&e->counted, cudaEventDisableTiming);
    if (r != cudaSuccess) return bail(r);
#undef EALLOC
    cudaStream_t s = nullptr;
    r = cudaMemsetAsync(e->grads, 0, sizeof(float) * np, s);
    if (r == cudaSuccess) r = cudaMemsetAsync(e->adam_m, 0, sizeof(float) * np, s);
    if (r == cudaSuccess) r = cudaMemsetAsync(e->adam_v, 0, sizeof(float) * np, s);
    if (r == cudaSuccess) r = cudaMemsetAsync(e->params, 0, sizeof(float) * np, s);
    if (r == cudaSuccess) r = cudaMemsetAsync(e->d_loss, 0, sizeof(double), s);
    if (r == cudaSuccess) r = cudaMemsetAsync(e->d_error, 0, sizeof(int32_t), s);
    if (r != cudaSuccess) return bail(r);
    // weights: uniform(-a, a) with a = sqrt(6 / (fan_in + fan_out)); embeddings
    // uniform(-0.5, 0.5); biases zero
    const struct {
        int t;
        float a;
    } init[] = {{CULDA_ENC_E, 0.5f},
                {CULDA_ENC_W1, sqrtf(6.0f / (kE + kH))},
                {CULDA_ENC_W2, sqrtf(6.0f / (kH + kH))},
                {CULDA_ENC_W3, sqrtf(6.0f / (float)(kH + e->K))}};
    for (const auto &x : init) {
        const int64_t n = sizes[x.t];
        init_uniform_kernel<<<grid_for(n), 256, 0, s>>>(n, e->tensor(x.t), x.a, p->seed, (uint32_t)x.t);
    }
    r = refresh_bf16(e, s);
    if (r == cudaSuccess) r = cudaStreamSynchronize(s);
    if (r != cudaSuccess) return bail(r);
    *out = e;
    return CULDA_OK;
}

extern "C" int culda_encoder_destroy(culda_encoder *e) {
    if (!e) return CULDA_OK;
    cudaSetDevice(e->device);
    cudaDeviceSynchronize();
    free_encoder(e);
    return CULDA_OK;
}

extern "C" int64_t culda_encoder_tensor_size(const culda_encoder *e, int32_t which) {
    if (!e) return CULDA_ERR_INVALID_ARG;
    const int t = which >= CULDA_ENC_GRAD ? which - CULDA_ENC_GRAD : which;
    if (t < 0 || t >= kNumTensors) return CULDA_ERR_INVALID_ARG;
    return e->off[t + 1] - e->off[t];
}

extern "C" int culda_encoder_get_tensor(culda_encoder *e, int32_t which, float *host) {
    const int64_t n = culda_encoder_tensor_size(e, which);
    if (n < 0 || !host) return fail_enc(CULDA_ERR_INVALID_ARG, "culda_encoder_get_tensor: %s", "bad tensor");
    ECK(cudaSetDevice(e->device));
    const float *src = which >= CULDA_ENC_GRAD ? e->grad(which - CULDA_ENC_GRAD) : e->tensor(which);
    ECK(cudaMemcpy(host, src, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost));
    return CULDA_OK;
}

extern "C" int culda_encoder_set_tensor(culda_encoder *e, int32_t which, const float *host) {
    const int64_t n = culda_encoder_tensor_size(e, which);
    if (n < 0 || !host || which >= CULDA_ENC_GRAD)
        return fail_enc(CULDA_ERR_INVALID_ARG, "culda_encoder_set_tensor: %s", "bad tensor");
    ECK(cudaSetDevice(e->device));
    ECK(cudaMemcpy(e->tensor(which), host, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice));
    ECK(refresh_bf16(e, nullptr));
    ECK(cudaDeviceSynchronize());
    return CULDA_OK;
}

extern "C" int culda_encoder_forward(culda_encoder *e, int32_t batch, const int32_t *d_docs,
                                     const int64_t *d_doc_ptr, const int32_t *d_words, float *d_probs, void *stream) {
    if (!e || !d_probs) return fail_enc(CULDA_ERR_INVALID_ARG, "culda_encoder_forward: %s", "null argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int rc = encoder_pass(e, batch, d_docs, d_doc_ptr, d_words, nullptr, false, d_probs, s);
    if (rc) return rc;
    return encoder_take_loss(e, 0, nullptr, s);
}

static int backward_call(culda_encoder *e, int32_t batch, const int32_t *d_docs, const int64_t *d_doc_ptr,
                         const int32_t *d_words, const float *d_target, double *loss, void *stream, bool update) {
    if (!e || !d_target) return fail_enc(CULDA_ERR_INVALID_ARG, "culda_encoder_backward: %s", "null argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    EncoderTarget t;
    t.dense = d_target;
    int rc = encoder_pass(e, batch, d_docs, d_doc_ptr, d_words, &t, update, nullptr, s);
    if (rc) {
        encoder_take_loss(e, 0, nullptr, s);  // what the part of the pass that ran has added
        return rc;
    }
    return encoder_take_loss(e, batch, loss, s);
}

extern "C" int culda_encoder_backward(culda_encoder *e, int32_t batch, const int32_t *d_docs,
                                      const int64_t *d_doc_ptr, const int32_t *d_words, const float *d_target,
                                      double *loss, void *stream) {
    return backward_call(e, batch, d_docs, d_doc_ptr, d_words, d_target, loss, stream, false);
}

extern "C" int culda_encoder_train_step(culda_encoder *e, int32_t batch, const int32_t *d_docs,
                                        const int64_t *d_doc_ptr, const int32_t *d_words, const float *d_target,
                                        double *loss, void *stream) {
    return backward_call(e, batch, d_docs, d_doc_ptr, d_words, d_target, loss, stream, true);
}
