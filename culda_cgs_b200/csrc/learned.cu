// learned.cu — the learned Metropolis-Hastings proposal and fold-in on a
// context: training pairs (document bag, accumulated topic distribution),
// encoder training over the context's documents, per-doc proposal tables, the
// MH iteration whose stationary target is the plain sampler's conditional on
// the frozen snapshot, p(k) ~ (n_dk + alpha) * phihat_wk, a frozen-model mode
// for new documents, and the encoder warm start of their topics.
//
// MH iteration (one launch per kernel, not graph-captured):
//   prologue -> hot_rows -> dense n_dk table from the theta CSR (when a proposal
//   is set) -> mh_kernel(z[c] -> z[1-c]) -> theta rebuild (as plain CGS).
// mh_kernel reuses the sampler's work items: per item the word's counts come
// from a histogram of the snapshot topics (or the hot row, or the frozen
// counts), then a lane per token runs `steps` steps:
//   doc step     k' ~ (n_dk + alpha): with probability L_d / (L_d + K alpha)
//                the topic of a uniformly chosen token of the doc, else a
//                uniform topic; accept with min(1, phihat_wk' / phihat_ws).
//   encoder step k' ~ q_d (two-level search of the doc's prefix table);
//                accept with min(1, (n_dk' + alpha) phihat_wk' q_d(s) /
//                ((n_ds + alpha) phihat_ws q_d(k'))).
// Steps alternate doc, encoder, doc, ... when a proposal is set; otherwise all
// are doc steps.  Each step leaves p invariant, so their sequence does too.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <numeric>
#include <vector>

#include "context.h"
#include "device_util.cuh"
#include "encoder.cuh"
#include "gemm.cuh"
#include "kernels.cuh"
#include "philox.h"

using namespace culda;

namespace {

// ------------------------------------------------------------------ kernels
// Word id of every token in doc order: doc_tok[i] is a stored (word-major)
// token index, whose word is the last w with word_ptr[w] <= doc_tok[i].
__global__ void doc_words_kernel(int64_t n, int num_words, const int64_t *__restrict__ word_ptr,
                                 const int32_t *__restrict__ doc_tok, int32_t *out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = doc_tok[i];
        int lo = 0, hi = num_words - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(word_ptr + mid) <= t)
                lo = mid;
            else
                hi = mid - 1;
        }
        out[i] = lo;
    }
}

// Warp per doc: the row's entries into a dense [D x K] table (set or added).
// A topic occurs at most once per row, so no two lanes touch one element.
template <class T>
__global__ void theta_to_dense_kernel(int D, int K, const int2 *__restrict__ rows,
                                      const ThetaEntry *__restrict__ theta, T *dense, bool add) {
    const int lane = threadIdx.x & 31;
    for (int d = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; d < D; d += (gridDim.x * blockDim.x) >> 5) {
        const int2 r = rows[d];
        for (int i = r.x + lane; i < r.y; i += 32) {
            const ThetaEntry e = theta[i];
            const uint32_t c = e & 0xFFFFu;
            if (!c) continue;
            T *p = dense + (size_t)d * K + (e >> 18);
            *p = add ? (T)(*p + (T)c) : (T)c;
        }
    }
}

// Warp per batch row: proposal (1 - mix) q + mix / K, inclusive prefix over
// the row (lane l sums topics [l*K/32, (l+1)*K/32), then a warp scan) and the
// prefix at the end of every 32 topics.
__global__ void proposal_table_kernel(int rows, int d0, int K, float mix, const float *__restrict__ probs,
                                      float *cdf, float *blk) {
    const int lane = threadIdx.x & 31;
    const int per = K >> 5, nb = K >> 5;
    const float u = mix / (float)K, a = 1.0f - mix;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < rows; b += (gridDim.x * blockDim.x) >> 5) {
        const float *q = probs + (size_t)b * K + lane * per;
        float *c = cdf + (size_t)(d0 + b) * K + lane * per;
        float s = 0.f;
        for (int i = 0; i < per; ++i) {
            s += a * q[i] + u;
            c[i] = s;
        }
        float incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const float base = incl - s;
        for (int i = 0; i < per; ++i) c[i] += base;
        __syncwarp();
        const float *row = cdf + (size_t)(d0 + b) * K;
        for (int j = lane; j < nb; j += 32) blk[(size_t)(d0 + b) * nb + j] = row[32 * j + 31];
    }
}

struct MHParams {
    int k;
    float alpha, beta, vbeta;
    int num_docs, num_items, num_hot;
    int64_t num_tokens;
    const int32_t *doc_ids;    // stored order
    const int32_t *tok_index;  // stored -> input index (Philox key), or null
    const uint16_t *topics_in;
    uint16_t *topics_out;
    const int2 *doc_span;      // {first token, length} of every doc
    const int32_t *doc_tok;
    const int32_t *nk;
    const culda_item *items;
    int num_coop;              // items [0, num_coop) take a CTA each, the others a warp
    int32_t *warp_counter;     // queue head of the others
    const int32_t *hot_phi;
    const int32_t *frozen_phi;  // [V x K] fixed counts (fold-in) or null
    int32_t *item_counter;
    const uint16_t *ndk;  // [D x K]
    const float *cdf;     // [D x K] or null
    const float *blk;     // [D x K/32]
    uint64_t seed;
    uint32_t iteration;
    int steps;
    int32_t *error;
    unsigned long long *stats;  // {accepted, proposed}
    unsigned long long *clock;  // {first start, last end} of the launch's CTAs
};

constexpr int kMHThreads = 256;

// First index in [lo, lo + n) whose value exceeds t (lo + n - 1 when none does).
__device__ __forceinline__ int first_above(const float *__restrict__ v, int lo, int n, float t) {
    int l = lo, h = lo + n - 1;
    while (l < h) {
        const int mid = (l + h) >> 1;
        if (__ldg(v + mid) > t)
            h = mid;
        else
            l = mid + 1;
    }
    return l;
}

// The phihat row of the item's word into ph[] (inv[] holds 1 / (n_k + V beta)):
// frozen counts, the hot row, or a histogram of the item's snapshot topics.
// Ends with a barrier.
__device__ __forceinline__ void item_phi_row(const MHParams &p, const culda_item &item, float *ph, const float *inv,
                                             int *hist) {
    const int K = p.k, tid = threadIdx.x;
    const int *src;
    if (p.frozen_phi) {
        src = p.frozen_phi + (size_t)item.word * K;
    } else if (item.hot < 0) {
        for (int j = tid; j < K; j += blockDim.x) hist[j] = 0;
        __syncthreads();
        for (int64_t t = item.begin + tid; t < item.begin + item.count; t += blockDim.x) {
            const uint32_t z = p.topics_in[t];
            if (z < (uint32_t)K)
                atomicAdd(&hist[z], 1);
            else
                atomicOr(p.error, kErrTopicRange);
        }
        __syncthreads();
        src = hist;
    } else {
        src = p.hot_phi + (size_t)item.hot * K;
    }
    for (int j = tid; j < K; j += blockDim.x) ph[j] = ((float)src[j] + p.beta) * inv[j];
    __syncthreads();
}

__device__ __forceinline__ bool item_ok(const MHParams &p, const culda_item &item) {
    return item.begin >= 0 && item.count >= 0 && item.begin + item.count <= p.num_tokens && item.hot < p.num_hot &&
           item.word >= 0;
}

// ------------------------------------------------- Metropolis-Hastings steps
// A token's steps are random reads behind one another (its document's span, a
// token of it, that token's topic, the proposal's tables, n_dk), so the kernel
// is bound by their latency (L1 at 36%, issue at 21% when a step followed the
// other in program order: 561 us for two steps at 6M tokens and K = 512).  No
// proposal depends on where the chain stands: the two of a pair of steps are
// formed together, their reads in flight beside one another and beside those
// of the next 32 tokens, and only the acceptances follow one another.  Words of
// fewer than kMHCoop tokens take a warp each with the counts in 16 bits (phihat
// is formed where it is read); a CTA per word left most lanes idle on them.
// 351 us.  62 registers, 32 warps per SM: 363 us at 72 registers and 24 warps,
// 413 us at 48 (spills); reading each search's 128-byte stretch with eight
// lanes and probing comparison bits instead of memory takes 32 registers more
// and was slower (497 us): the probes after the first hit the L1.
// They do while the L1 holds a warp's 32 stretches from probe to probe.  Once
// the tables are well past the L2, the reads' latency keeps so many stretches
// alive that they drive one another out, and fewer warps are faster: from
// kMHTableL2 times the L2 on an SM takes kMHTableBlocks CTAs.  Two steps at 61M
// tokens: K = 1024 (1.8 GB) 7.98 ms with 8 CTAs, 7.03 with 6, 7.05 with 5; K =
// 512 (0.9 GB) 6.84, 6.14, 6.24; but at 12M tokens, K = 1024 (0.37 GB) 1.08,
// 1.11, 1.20.  For the same room cnt lies in ph's place (8.44 -> 7.85 ms at 8
// CTAs).  With such tables a chain of more than two steps also keeps what it
// read of its topic while it stays there (kKeep; eight steps 25.7 -> 22.4 ms;
// it costs 3% at two steps and gives nothing at 12M tokens).
constexpr int kMHTableL2 = 4, kMHTableBlocks = 6;
constexpr int kMHStepThreads = 128;
constexpr int kMHWarps = kMHStepThreads / 32;

// A token before its steps: topic, document (-1: none), Philox key, the
// document's first token and length.
struct MHToken {
    int s, d;
    uint64_t key;
    int2 span;
};

__device__ __forceinline__ MHToken mh_load(const MHParams &p, bool valid, int64_t t) {
    MHToken x{0, -1, 0, make_int2(0, 1)};
    if (!valid) return x;
    x.s = p.topics_in[t];
    x.d = p.doc_ids[t];
    x.key = p.tok_index ? (uint64_t)__ldg(p.tok_index + t) : (uint64_t)t;
    if ((unsigned)x.d >= (unsigned)p.num_docs || (unsigned)x.s >= (unsigned)p.k) {
        atomicOr(p.error, kErrDocRange);
        p.topics_out[t] = (uint16_t)min(max(x.s, 0), p.k - 1);
        return MHToken{0, -1, 0, make_int2(0, 1)};
    }
    x.span = __ldg(p.doc_span + x.d);
    return x;
}

// A doc proposal: a token of the document (its index in word order, else -1)
// or, without one, the topic.
__device__ __forceinline__ int doc_proposal(const MHParams &p, const MHToken &tok, const u32x4 &x, float ka, int &kp) {
    const float L = (float)tok.span.y;
    kp = (int)bounded_from_bits(x.y, (uint32_t)p.k);
    if (tok.d >= 0 && uniform_from_bits(x.x) * (L + ka) < L)
        return __ldg(p.doc_tok + tok.span.x + (int)bounded_from_bits(x.y, (uint32_t)tok.span.y));
    return -1;
}

// The steps of up to 32 tokens, lane l's at t, against the word's phihat.  The
// whole warp takes part.
template <bool kKeep, class PhiHat>
__device__ __forceinline__ void mh_tokens(const MHParams &p, const MHToken &tok, int64_t t, const PhiHat &ph, int lane,
                                          unsigned &acc_n, unsigned &prop_n) {
    const int K = p.k, nb = K >> 5;
    const float ka = (float)K * p.alpha;
    const bool active = tok.d >= 0;
    const int d = max(tok.d, 0);
    int s = tok.s;
    // q_d and n_dk of the topic s_read, where the chain stood when they were read
    float q_s = 0.f, n_s = 0.f;
    int s_read = -1;
    for (int step = 0; step < p.steps; step += 2) {
        const bool two = step + 1 < p.steps, enc = two && p.cdf;
        const u32x4 x0 = philox_token4(p.seed, tok.key, p.iteration, kPurposeMH + (uint32_t)step);
        const u32x4 x1 = philox_token4(p.seed, tok.key, p.iteration, kPurposeMH + (uint32_t)step + 1u);
        // both proposals: first what they read first, then what that leads to
        int k0, k1 = 0, i1 = -1;
        const int i0 = doc_proposal(p, tok, x0, ka, k0);
        const float *blk = p.blk + (size_t)d * nb, *row = p.cdf + (size_t)d * K;
        float total = 0.f;
        if (enc)
            total = __ldg(blk + nb - 1);
        else if (two)
            i1 = doc_proposal(p, tok, x1, ka, k1);
        const uint16_t *nd = p.ndk + (size_t)d * K;
        auto read_s = [&] {
            if (!kKeep || s != s_read) {
                q_s = __ldg(row + s) - (s > 0 ? __ldg(row + s - 1) : 0.f);
                n_s = (float)nd[s];
                s_read = s;
            }
        };
        if (i0 >= 0) k0 = p.topics_in[i0];
        if (i1 >= 0) k1 = p.topics_in[i1];
        if (enc) {
            const float T = uniform_from_bits(x1.y) * total;
            k1 = first_above(row, 32 * first_above(blk, 0, nb, T), 32, T);
        }
        // the first acceptance
        auto accept = [&](int k, float ratio, uint32_t bits) {
            ++prop_n;
            if (k != s && uniform_from_bits(bits) < ratio) {
                s = k;
                ++acc_n;
            }
        };
        if (active) {
            if ((unsigned)k0 >= (unsigned)K) k0 = s;
            accept(k0, ph(k0) / ph(s), x0.z);
        }
        if (enc) {
            const float qk = __ldg(row + k1) - (k1 > 0 ? __ldg(row + k1 - 1) : 0.f);
            const float n_k = (float)nd[k1];
            read_s();
            if (active) {
                const float pk = (n_k + p.alpha) * ph(k1);
                const float ps = (n_s + p.alpha) * ph(s);
                accept(k1, (pk * q_s) / (ps * qk), x1.z);
                if (kKeep && s == k1) q_s = qk, n_s = n_k, s_read = k1;
            }
        } else if (two && active) {
            if ((unsigned)k1 >= (unsigned)K) k1 = s;
            accept(k1, ph(k1) / ph(s), x1.z);
        }
    }
    if (active) p.topics_out[t] = (uint16_t)s;
}

// Tokens [begin, end) of an item, 32 at a time `stride` apart, the next 32
// loaded ahead.
template <bool kKeep, class PhiHat>
__device__ __forceinline__ void mh_run(const MHParams &p, int64_t begin, int64_t end, int stride, const PhiHat &ph,
                                       int lane, unsigned &acc_n, unsigned &prop_n) {
    MHToken tok = mh_load(p, begin + lane < end, begin + lane);
    for (int64_t t0 = begin; t0 < end; t0 += stride) {
        const int64_t tn = t0 + stride + lane;
        const MHToken next = mh_load(p, tn < end, tn);
        mh_tokens<kKeep>(p, tok, t0 + lane, ph, lane, acc_n, prop_n);
        tok = next;
    }
}

template <bool kKeep>
__global__ void __launch_bounds__(kMHStepThreads, 8) mh_kernel(const MHParams p) {
    extern __shared__ float sm_mh[];
    const int K = p.k;
    float *inv = sm_mh;                              // [K] 1 / (n_k + V beta)
    float *ph = sm_mh + K;                           // [K] phihat of the CTA's word (its histogram before that)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t *cnt = reinterpret_cast<uint32_t *>(sm_mh + K) + warp * (K / 2);  // in ph's place later: the warp's word, 16-bit counts
    __shared__ int s_item;
    unsigned acc_n = 0, prop_n = 0;
    if (tid == 0) clock_start(p.clock);

    for (int j = tid; j < K; j += blockDim.x) inv[j] = 1.0f / ((float)p.nk[j] + p.vbeta);
    // the long items: a CTA each
    for (;;) {
        if (tid == 0) s_item = atomicAdd(p.item_counter, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= p.num_coop) break;
        const culda_item item = p.items[it];
        if (!item_ok(p, item)) {
            if (tid == 0) atomicOr(p.error, kErrRowRange);
            __syncthreads();
            continue;
        }
        item_phi_row(p, item, ph, inv, reinterpret_cast<int *>(ph));
        const int64_t iend = item.begin + item.count;
        mh_run<kKeep>(p, item.begin + 32 * warp, iend, kMHStepThreads, [ph](int k) { return ph[k]; }, lane, acc_n, prop_n);
        __syncthreads();  // ph is rebuilt for the next item
    }
    // the others: a warp each (behind the barrier of the loop's last turn)
    for (int j = lane; j < K / 2; j += 32) cnt[j] = 0u;
    __syncwarp();
    for (;;) {
        int it = 0;
        if (lane == 0) it = p.num_coop + atomicAdd(p.warp_counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= p.num_items) break;
        const culda_item item = p.items[it];
        if (!item_ok(p, item)) {
            if (lane == 0) atomicOr(p.error, kErrRowRange);
            continue;
        }
        const int64_t iend = item.begin + item.count;
        const int32_t *fixed = p.frozen_phi ? p.frozen_phi + (size_t)item.word * K
                               : item.hot >= 0 ? p.hot_phi + (size_t)item.hot * K : nullptr;
        if (fixed) {
            auto phihat = [&](int k) { return ((float)__ldg(fixed + k) + p.beta) * inv[k]; };
            mh_run<kKeep>(p, item.begin, iend, 32, phihat, lane, acc_n, prop_n);
            continue;
        }
        for (int64_t t = item.begin + lane; t < iend; t += 32) {
            const uint32_t z = p.topics_in[t];
            if (z < (uint32_t)K)
                atomicAdd(&cnt[z >> 1], 1u << ((z & 1u) << 4));
            else
                atomicOr(p.error, kErrTopicRange);
        }
        __syncwarp();
        auto phihat = [&](int k) {
            return ((float)((cnt[k >> 1] >> ((k & 1) << 4)) & 0xFFFFu) + p.beta) * inv[k];
        };
        mh_run<kKeep>(p, item.begin, iend, 32, phihat, lane, acc_n, prop_n);
        __syncwarp();
        for (int64_t t = item.begin + lane; t < iend; t += 32) {
            const uint32_t z = p.topics_in[t];
            if (z < (uint32_t)K) cnt[z >> 1] = 0u;
        }
        __syncwarp();
    }
    if (p.stats) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            acc_n += __shfl_xor_sync(0xffffffffu, acc_n, o);
            prop_n += __shfl_xor_sync(0xffffffffu, prop_n, o);
        }
        if (lane == 0 && prop_n) {
            atomicAdd(&p.stats[0], (unsigned long long)acc_n);
            atomicAdd(&p.stats[1], (unsigned long long)prop_n);
        }
    }
    if (tid == 0) clock_end(p.clock);
}

// {first token, length} of every document (tokens are below 2^31).
__global__ void doc_span_kernel(int D, const int64_t *__restrict__ doc_ptr, int2 *span) {
    for (int d = blockIdx.x * blockDim.x + threadIdx.x; d < D; d += gridDim.x * blockDim.x)
        span[d] = make_int2((int)doc_ptr[d], (int)(doc_ptr[d + 1] - doc_ptr[d]));
}

// Warm start: warp per token; the token's topic is drawn from
// q_d(k) * phihat_wk (q_d from the differences of the doc's proposal prefix
// table) by inverse CDF in ascending topic.  Lanes take consecutive topics,
// 32 at a time, so every table load is one coalesced line: a first pass sums
// the weights, a second runs a warp scan chunk by chunk until the running sum
// passes u * total (the last topic if rounding leaves it short).
__device__ __forceinline__ float warm_weight(const float *__restrict__ row, const float *ph, int c, int lane,
                                             float &carry) {
    const float cur = __ldg(row + c + lane);
    float prev = __shfl_up_sync(0xffffffffu, cur, 1);
    if (lane == 0) prev = carry;
    carry = __shfl_sync(0xffffffffu, cur, 31);
    return (cur - prev) * ph[c + lane];
}

__global__ void __launch_bounds__(kMHThreads) warm_start_kernel(const MHParams p) {
    extern __shared__ float sm_ws[];
    const int K = p.k;
    float *ph = sm_ws;
    float *inv = sm_ws + K;
    int *hist = reinterpret_cast<int *>(sm_ws + 2 * K);
    __shared__ int s_item;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    for (int j = tid; j < K; j += blockDim.x) inv[j] = 1.0f / ((float)p.nk[j] + p.vbeta);
    for (;;) {
        if (tid == 0) s_item = atomicAdd(p.item_counter, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= p.num_items) break;
        const culda_item item = p.items[it];
        if (!item_ok(p, item)) {
            if (tid == 0) atomicOr(p.error, kErrRowRange);
            __syncthreads();
            continue;
        }
        item_phi_row(p, item, ph, inv, hist);
        const int64_t iend = item.begin + item.count;
        for (int64_t t = item.begin + warp; t < iend; t += nwarps) {
            const int d = p.doc_ids[t];
            if ((unsigned)d >= (unsigned)p.num_docs) {
                if (lane == 0) atomicOr(p.error, kErrDocRange);
                continue;
            }
            const float *row = p.cdf + (size_t)d * K;
            float carry = 0.f, part = 0.f;
            for (int c = 0; c < K; c += 32) part += warm_weight(row, ph, c, lane, carry);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            const uint64_t key = p.tok_index ? (uint64_t)__ldg(p.tok_index + t) : (uint64_t)t;
            const float T = uniform_from_bits(philox_token(p.seed, key, 0u, kPurposeWarm)) * part;
            int pick = K - 1;
            float base = 0.f;
            carry = 0.f;
            for (int c = 0; c < K; c += 32) {
                float incl = warm_weight(row, ph, c, lane, carry);
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                incl += base;
                const unsigned hit = __ballot_sync(0xffffffffu, incl > T);
                if (hit) {
                    pick = c + __ffs(hit) - 1;
                    break;
                }
                base = __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) p.topics_out[t] = (uint16_t)pick;
        }
        __syncthreads();
    }
}

// Block per word (rows past V are zero): the word's topic profile
// (n_wk + beta) / (n_w + K beta) in BF16, from a histogram of its tokens.
__global__ void phi_profile_kernel(int V, int rows, int K, float beta, const int64_t *__restrict__ word_ptr,
                                   const uint16_t *__restrict__ topics, __nv_bfloat16 *out) {
    extern __shared__ int hist_p[];
    for (int w = blockIdx.x; w < rows; w += gridDim.x) {
        for (int j = threadIdx.x; j < K; j += blockDim.x) hist_p[j] = 0;
        __syncthreads();
        int64_t n = 0;
        if (w < V) {
            n = word_ptr[w + 1] - word_ptr[w];
            for (int64_t t = word_ptr[w] + threadIdx.x; t < word_ptr[w + 1]; t += blockDim.x) {
                const uint32_t z = topics[t];
                if (z < (uint32_t)K) atomicAdd(&hist_p[z], 1);
            }
        }
        __syncthreads();
        const float inv = 1.0f / ((float)n + (float)K * beta);
        for (int j = threadIdx.x; j < K; j += blockDim.x)
            out[(size_t)w * K + j] = __float2bfloat16_rn(w < V ? ((float)hist_p[j] + beta) * inv : 0.f);
        __syncthreads();
    }
}

// Random projection matrix R [256 x K], entries uniform with unit variance.
__global__ void projection_kernel(int n, uint64_t seed, __nv_bfloat16 *R) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        R[i] = __float2bfloat16_rn(
            1.7320508f * (2.0f * uniform_from_bits(philox_token(seed, (uint64_t)i, 0u, kPurposeWeights)) - 1.0f));
}

// Warp per word: E[w] = P[w] scaled to root-mean-square `rms`.
__global__ void rms_rows_kernel(int V, int cols, float rms, const float *__restrict__ P, float *E) {
    const int lane = threadIdx.x & 31;
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < V; w += (gridDim.x * blockDim.x) >> 5) {
        float ss = 0.f;
        for (int j = lane; j < cols; j += 32) ss += P[(size_t)w * cols + j] * P[(size_t)w * cols + j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float sc = ss > 0.f ? rms * rsqrtf(ss / (float)cols) : 0.f;
        for (int j = lane; j < cols; j += 32) E[(size_t)w * cols + j] = P[(size_t)w * cols + j] * sc;
    }
}

// ------------------------------------------------------------- host helpers
int ensure_doc_words(culda_ctx *ctx) {
    if (ctx->d_doc_words) return CULDA_OK;
    CK(dalloc(&ctx->d_doc_words, (size_t)ctx->N));
    doc_words_kernel<<<grid_for(ctx->N), 256, 0, ctx->stream>>>(ctx->N, ctx->V, ctx->d_word_ptr, ctx->d_doc_tok,
                                                                ctx->d_doc_words);
    CK(cudaGetLastError());
    return CULDA_OK;
}

int build_dense_theta(culda_ctx *ctx) {
    cudaStream_t s = ctx->stream;
    if (!ctx->d_ndk) CK(dalloc(&ctx->d_ndk, (size_t)ctx->D * ctx->K));
    CK(cudaMemsetAsync(ctx->d_ndk, 0, sizeof(uint16_t) * (size_t)ctx->D * ctx->K, s));
    theta_to_dense_kernel<uint16_t><<<grid_for((int64_t)ctx->D * 32), 256, 0, s>>>(
        ctx->D, ctx->K, ctx->d_rows, ctx->d_theta, ctx->d_ndk, false);
    CK(cudaGetLastError());
    return CULDA_OK;
}

MHParams mh_params(culda_ctx *ctx, int cur, uint32_t iteration, int steps) {
    MHParams p{};
    p.k = ctx->K;
    p.alpha = ctx->params.alpha;
    p.beta = ctx->params.beta;
    p.vbeta = ctx->params.beta * (float)ctx->V;
    p.num_docs = ctx->D;
    p.num_items = ctx->num_items;
    p.num_hot = ctx->num_hot;
    p.num_tokens = ctx->N;
    p.doc_ids = ctx->d_doc_ids;
    p.tok_index = ctx->d_tok_index;
    p.topics_in = ctx->d_z[cur];
    p.topics_out = ctx->d_z[1 - cur];
    p.doc_span = ctx->d_doc_span;
    p.num_coop = ctx->num_mh_coop;
    p.warp_counter = warp_queue(ctx);
    p.doc_tok = ctx->d_doc_tok;
    p.nk = ctx->d_frozen_phi ? ctx->d_frozen_nk : ctx->d_nk[cur];
    p.items = ctx->d_items;
    p.hot_phi = ctx->d_hot_phi;
    p.frozen_phi = ctx->d_frozen_phi;
    p.item_counter = ctx->d_counter;
    p.ndk = ctx->d_ndk;
    p.cdf = ctx->has_proposal ? ctx->d_cdf : nullptr;
    p.blk = ctx->d_cdf_blk;
    p.seed = ctx->params.seed;
    p.iteration = iteration;
    p.steps = steps;
    p.error = ctx->d_error;
    p.stats = &ctx->d_stats->mh_accepted;
    p.clock = &ctx->d_stats->sample_t0;
    return p;
}

int hot_rows_if_needed(culda_ctx *ctx, int cur) {
    cudaStream_t s = ctx->stream;
    if (ctx->num_hot > 0 && !ctx->d_frozen_phi) {
        CK(cudaMemsetAsync(ctx->d_hot_phi, 0, sizeof(int32_t) * (size_t)ctx->num_hot * ctx->K, s));
        CK(launch_hot_rows(ctx->K, ctx->d_hot_items, ctx->num_hot_items, ctx->d_z[cur], ctx->d_hot_phi, ctx->d_error,
                           s));
    }
    return CULDA_OK;
}

template <class Kernel>
int persistent_grid(culda_ctx *ctx, Kernel kernel, int threads, size_t smem, int *grid) {
    CK(allow_smem(reinterpret_cast<const void *>(kernel), smem));
    int bps = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel, threads, smem));
    *grid = std::max(1, std::min(ctx->num_items, num_sms(ctx->device) * std::max(bps, 1)));
    return CULDA_OK;
}

// Hot rows, the dense n_dk table and the MH kernel: topics d_z[cur] -> d_z[1-cur].
int launch_mh_pass(culda_ctx *ctx, int cur, uint32_t iteration, int steps) {
    cudaStream_t s = ctx->stream;
    CK(iteration_prologue(ctx, cur, false, iteration, nullptr));
    int rc = CULDA_OK;
    if (ctx->has_proposal) rc = build_dense_theta(ctx);  // the doc proposal reads no n_dk
    if (rc) return rc;
    if (!ctx->d_doc_span) {
        CK(dalloc(&ctx->d_doc_span, (size_t)ctx->D));
        doc_span_kernel<<<grid_for(ctx->D), 256, 0, s>>>(ctx->D, ctx->d_doc_ptr, ctx->d_doc_span);
        CK(cudaGetLastError());
    }
    const size_t smem = ((size_t)ctx->K + (size_t)kMHWarps * (size_t)(ctx->K / 2)) * sizeof(float);  // inv, ph or cnt
    int grid = 1, l2 = 0;
    cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, ctx->device);
    const size_t tables = ctx->has_proposal ? (sizeof(float) + sizeof(uint16_t)) * (size_t)ctx->D * ctx->K : 0;
    const bool large = tables > (size_t)kMHTableL2 * (size_t)l2;
    auto kernel = large && steps > 2 ? mh_kernel<true> : mh_kernel<false>;
    rc = persistent_grid(ctx, kernel, kMHStepThreads, smem, &grid);
    if (rc) return rc;
    if (large) grid = std::min(grid, num_sms(ctx->device) * kMHTableBlocks);
    kernel<<<grid, kMHStepThreads, smem, s>>>(mh_params(ctx, cur, iteration, steps));
    CK(cudaGetLastError());
    return CULDA_OK;
}

int check_device_error(culda_ctx *ctx, const char *what) {
    int32_t e = 0;
    CK(cudaMemcpyAsync(&e, ctx->d_error, sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    if (e) return fail(ctx, CULDA_ERR_DEVICE_STATE, "%s: device error 0x%x", what, e);
    return CULDA_OK;
}

}  // namespace

void free_learned_state(culda_ctx *ctx) {
    void *bufs[] = {ctx->d_doc_words, ctx->d_acc,    ctx->d_ndk,        ctx->d_cdf,        ctx->d_cdf_blk,
                    ctx->d_doc_span,  ctx->d_probs,     ctx->frozen_borrowed ? nullptr : ctx->d_frozen_phi,
                    ctx->frozen_borrowed ? nullptr : ctx->d_frozen_nk};
    for (void *b : bufs)
        if (b) cudaFree(b);
    ctx->frozen_borrowed = false;
    ctx->d_doc_words = nullptr;
    ctx->d_acc = nullptr;
    ctx->d_ndk = nullptr;
    ctx->d_doc_span = nullptr;
    ctx->d_cdf = nullptr;
    ctx->d_cdf_blk = nullptr;
    ctx->d_probs = nullptr;
    ctx->d_frozen_phi = nullptr;
    ctx->d_frozen_nk = nullptr;
    ctx->has_proposal = false;
}

// ============================================================ C entry points
extern "C" int culda_accumulate_theta(culda_ctx *ctx) {
    if (!ctx) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_accumulate_theta: null context");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    if (!ctx->d_acc) {
        CK(dalloc(&ctx->d_acc, (size_t)ctx->D * ctx->K));
        CK(cudaMemsetAsync(ctx->d_acc, 0, sizeof(float) * (size_t)ctx->D * ctx->K, s));
        ctx->n_acc = 0;
    }
    theta_to_dense_kernel<float><<<grid_for((int64_t)ctx->D * 32), 256, 0, s>>>(ctx->D, ctx->K, ctx->d_rows,
                                                                               ctx->d_theta, ctx->d_acc, true);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    ctx->n_acc += 1;
    return CULDA_OK;
}

extern "C" int culda_train_encoder(culda_ctx *ctx, culda_encoder *enc, int32_t epochs, uint64_t seed,
                                   double *loss) {
    if (!ctx || !enc || epochs <= 0) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_train_encoder: invalid argument");
    if (!ctx->d_acc || ctx->n_acc <= 0)
        return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_train_encoder: no accumulated states (culda_accumulate_theta)");
    if (encoder_k(enc) != ctx->K || encoder_num_words(enc) != ctx->V)
        return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_train_encoder: encoder shape does not match the context");
    CK(cudaSetDevice(ctx->device));
    int rc = ensure_doc_words(ctx);
    if (rc) return rc;
    cudaStream_t s = ctx->stream;
    const int B = std::min(encoder_max_batch(enc), ctx->D);
    int32_t *d_order = nullptr;
    CK(dalloc(&d_order, (size_t)ctx->D));
    std::vector<int32_t> order((size_t)ctx->D);
    EncoderTarget tg;
    tg.acc = ctx->d_acc;
    tg.inv_n = 1.0f / (float)ctx->n_acc;
    tg.alpha = ctx->params.alpha;
    double last = 0.0;
    for (int ep = 0; ep < epochs && rc == CULDA_OK; ++ep) {
        // Fisher-Yates with Philox draws keyed on (seed, position, epoch)
        std::iota(order.begin(), order.end(), 0);
        for (int32_t i = ctx->D - 1; i > 0; --i) {
            const uint32_t j = bounded_from_bits(philox_token(seed, (uint64_t)i, (uint32_t)ep, kPurposeShuffle),
                                                 (uint32_t)i + 1u);
            std::swap(order[(size_t)i], order[j]);
        }
        if (cudaMemcpyAsync(d_order, order.data(), sizeof(int32_t) * order.size(), cudaMemcpyHostToDevice, s) !=
            cudaSuccess) {
            rc = fail(ctx, CULDA_ERR_CUDA, "culda_train_encoder: order upload failed");
            break;
        }
        // batches of B docs; the last one holds the remainder
        const int steps = (ctx->D + B - 1) / B;
        for (int st = 0; st < steps && rc == CULDA_OK; ++st) {
            const int b0 = st * B, nb = std::min(B, ctx->D - b0);
            int64_t tokens = 0;  // the batch's tokens, known here from the host doc index
            for (int i = b0; i < b0 + nb; ++i)
                tokens += ctx->h_doc_ptr[(size_t)order[(size_t)i] + 1] - ctx->h_doc_ptr[(size_t)order[(size_t)i]];
            rc = encoder_pass(enc, nb, d_order + b0, ctx->d_doc_ptr, ctx->d_doc_words, &tg, true, nullptr, s,
                              tokens);
        }
        const int taken = encoder_take_loss(enc, ctx->D, &last, s);  // also what a failed epoch has added
        if (rc == CULDA_OK) rc = taken;
        if (rc) fail(ctx, rc, "culda_train_encoder: %s", global_error());
        // the host order buffer is rewritten by the next epoch
        if (cudaStreamSynchronize(s) != cudaSuccess && rc == CULDA_OK)
            rc = fail(ctx, CULDA_ERR_CUDA, "culda_train_encoder: sync failed");
    }
    cudaStreamSynchronize(s);
    cudaFree(d_order);
    if (rc == CULDA_OK && loss) *loss = last;
    return rc;
}

extern "C" int culda_encoder_init_from_phi(culda_ctx *ctx, culda_encoder *enc, uint64_t seed) {
    if (!ctx || !enc) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_encoder_init_from_phi: null argument");
    if (encoder_num_words(enc) != ctx->V || encoder_k(enc) != ctx->K)
        return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_encoder_init_from_phi: encoder shape does not match the context");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    const int K = ctx->K, V = ctx->V, Vp = (V + 127) & ~127, E = CULDA_ENC_EMBED;
    __nv_bfloat16 *prof = nullptr, *R = nullptr;
    float *P = nullptr;
    int rc = CULDA_OK;
    if (dalloc(&prof, (size_t)Vp * K) != cudaSuccess || dalloc(&R, (size_t)E * K) != cudaSuccess ||
        dalloc(&P, (size_t)Vp * E) != cudaSuccess) {
        rc = fail(ctx, CULDA_ERR_OOM, "culda_encoder_init_from_phi: out of device memory");
    } else {
        const size_t smem = (size_t)K * sizeof(int);
        cudaError_t e = allow_smem(reinterpret_cast<const void *>(&phi_profile_kernel), smem);
        if (e == cudaSuccess) {
            phi_profile_kernel<<<std::min(Vp, num_sms(ctx->device) * 8), 256, smem, s>>>(
                V, Vp, K, ctx->params.beta, ctx->d_word_ptr, ctx->d_z[ctx->cur], prof);
            projection_kernel<<<grid_for((int64_t)E * K), 256, 0, s>>>(E * K, seed, R);
            e = cudaGetLastError();
        }
        GemmEpilogue ep;
        ep.out_f32 = P;
        ep.ldo = E;
        if (e == cudaSuccess) e = gemm_bf16_nt(Vp, E, K, prof, K, R, K, kEpiF32, ep, ctx->d_error, s);
        if (e == cudaSuccess) {
            rms_rows_kernel<<<grid_for((int64_t)V * 32), 256, 0, s>>>(V, E, 0.3f, P,
                                                                      encoder_tensor(enc, CULDA_ENC_E));
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) rc = fail(ctx, CULDA_ERR_CUDA, "culda_encoder_init_from_phi: %s", cudaGetErrorString(e));
        if (rc == CULDA_OK && encoder_refresh(enc, s) != CULDA_OK)
            rc = fail(ctx, CULDA_ERR_CUDA, "culda_encoder_init_from_phi: %s", global_error());
        if (rc == CULDA_OK) rc = check_device_error(ctx, "culda_encoder_init_from_phi");
    }
    cudaStreamSynchronize(s);
    if (prof) cudaFree(prof);
    if (R) cudaFree(R);
    if (P) cudaFree(P);
    return rc;
}

extern "C" int culda_set_proposal(culda_ctx *ctx, culda_encoder *enc, float mix) {
    if (!ctx) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_set_proposal: null context");
    if (!enc) {
        ctx->has_proposal = false;
        return CULDA_OK;
    }
    if (!(mix >= 0.f && mix < 1.f)) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_set_proposal: mix outside [0, 1)");
    if (encoder_k(enc) != ctx->K || encoder_num_words(enc) != ctx->V)
        return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_set_proposal: encoder shape does not match the context");
    CK(cudaSetDevice(ctx->device));
    int rc = ensure_doc_words(ctx);
    if (rc) return rc;
    cudaStream_t s = ctx->stream;
    const int B = encoder_max_batch(enc), K = ctx->K;
    if (!ctx->d_cdf) CK(dalloc(&ctx->d_cdf, (size_t)ctx->D * K));
    if (!ctx->d_cdf_blk) CK(dalloc(&ctx->d_cdf_blk, (size_t)ctx->D * (K / 32)));
    if (ctx->d_probs) cudaFree(ctx->d_probs);
    ctx->d_probs = nullptr;
    CK(dalloc(&ctx->d_probs, (size_t)B * K));
    int32_t *d_docs = nullptr;
    CK(dalloc(&d_docs, (size_t)B));
    std::vector<int32_t> ids((size_t)B);
    for (int32_t d0 = 0; d0 < ctx->D && rc == CULDA_OK; d0 += B) {
        const int n = std::min(B, ctx->D - d0);
        std::iota(ids.begin(), ids.begin() + n, d0);
        if (cudaMemcpyAsync(d_docs, ids.data(), sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, s) !=
            cudaSuccess) {
            rc = fail(ctx, CULDA_ERR_CUDA, "culda_set_proposal: upload failed");
            break;
        }
        rc = encoder_pass(enc, n, d_docs, ctx->d_doc_ptr, ctx->d_doc_words, nullptr, false, ctx->d_probs, s);
        if (rc) {
            fail(ctx, rc, "culda_set_proposal: %s", global_error());
            break;
        }
        proposal_table_kernel<<<grid_for((int64_t)n * 32), 256, 0, s>>>(n, d0, K, mix, ctx->d_probs, ctx->d_cdf,
                                                                       ctx->d_cdf_blk);
        if (cudaGetLastError() != cudaSuccess) rc = fail(ctx, CULDA_ERR_CUDA, "culda_set_proposal: launch failed");
        // the host ids buffer is rewritten for the next batch
        if (cudaStreamSynchronize(s) != cudaSuccess) rc = fail(ctx, CULDA_ERR_CUDA, "culda_set_proposal: sync failed");
    }
    cudaFree(d_docs);
    if (rc) return rc;
    rc = encoder_take_loss(enc, 0, nullptr, s);
    if (rc) return fail(ctx, rc, "culda_set_proposal: %s", global_error());
    ctx->has_proposal = true;
    return CULDA_OK;
}

extern "C" int culda_get_proposal(culda_ctx *ctx, float *cdf) {
    if (!ctx || !cdf) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_get_proposal: null argument");
    if (!ctx->has_proposal) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_get_proposal: no proposal set");
    CK(cudaSetDevice(ctx->device));
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaMemcpy(cdf, ctx->d_cdf, sizeof(float) * (size_t)ctx->D * ctx->K, cudaMemcpyDeviceToHost));
    return CULDA_OK;
}

extern "C" int culda_iterate_mh(culda_ctx *ctx, int32_t n, int32_t steps, culda_iter_stats *stats) {
    if (!ctx || n < 0 || steps < 1 || steps > 64)
        return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_iterate_mh: invalid argument");
    CK(cudaSetDevice(ctx->device));
    uint32_t iteration = ctx->next_iteration;
    return run_iterations(ctx, n, stats, true, [&]() -> int {
        const int rc = launch_mh_pass(ctx, ctx->cur, iteration++, steps);
        if (rc) return rc;
        CK(iteration_rebuild(ctx, ctx->cur, 0));
        return CULDA_OK;
    });
}

extern "C" int culda_mh_snapshot(culda_ctx *ctx, uint32_t iteration, int32_t steps, uint16_t *topics_out) {
    if (!ctx || steps < 1 || steps > 64) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_mh_snapshot: invalid argument");
    CK(cudaSetDevice(ctx->device));
    int rc = launch_mh_pass(ctx, ctx->cur, iteration, steps);
    if (rc) return rc;
    rc = check_device_error(ctx, "culda_mh_snapshot");
    if (rc) return rc;
    if (!topics_out) return CULDA_OK;
    return topics_to_host(ctx, ctx->d_z[1 - ctx->cur], topics_out);
}

extern "C" int culda_set_frozen_phi(culda_ctx *ctx, const int32_t *phi, const int32_t *nk) {
    if (!ctx) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_set_frozen_phi: null context");
    CK(cudaSetDevice(ctx->device));
    CK(cudaStreamSynchronize(ctx->stream));
    if (ctx->frozen_borrowed) {  // shared counts of a chunked run: the caller's buffers
        ctx->d_frozen_phi = nullptr;
        ctx->d_frozen_nk = nullptr;
        ctx->frozen_borrowed = false;
    }
    if (!phi) {
        if (ctx->d_frozen_phi) cudaFree(ctx->d_frozen_phi);
        if (ctx->d_frozen_nk) cudaFree(ctx->d_frozen_nk);
        ctx->d_frozen_phi = nullptr;
        ctx->d_frozen_nk = nullptr;
        return build_graphs(ctx);
    }
    if (!nk) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_set_frozen_phi: phi without nk");
    const size_t n = (size_t)ctx->V * ctx->K;
    // the counts must be consistent: non-negative, and the rows summing to nk
    std::vector<int64_t> sum((size_t)ctx->K, 0);
    for (size_t i = 0; i < n; ++i) {
        if (phi[i] < 0) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_set_frozen_phi: negative count");
        sum[i % ctx->K] += phi[i];
    }
    for (int32_t k = 0; k < ctx->K; ++k)
        if (sum[(size_t)k] != nk[k])
            return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_set_frozen_phi: nk[%d] = %d but phi sums to %lld", k, nk[k],
                        (long long)sum[(size_t)k]);
    if (!ctx->d_frozen_phi) CK(dalloc(&ctx->d_frozen_phi, n));
    if (!ctx->d_frozen_nk) CK(dalloc(&ctx->d_frozen_nk, (size_t)ctx->K));
    CK(copy_to_device(ctx->d_frozen_phi, phi, sizeof(int32_t) * n, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaMemcpy(ctx->d_frozen_nk, nk, sizeof(int32_t) * (size_t)ctx->K, cudaMemcpyHostToDevice));
    return build_graphs(ctx);
}

extern "C" int culda_warm_start(culda_ctx *ctx) {
    if (!ctx) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_warm_start: null context");
    if (!ctx->has_proposal) return fail(ctx, CULDA_ERR_INVALID_ARG, "culda_warm_start: no proposal (culda_set_proposal)");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    const int cur = ctx->cur;
    CK(cudaMemsetAsync(ctx->d_counter, 0, sizeof(int32_t), s));
    int rc = hot_rows_if_needed(ctx, cur);
    if (rc) return rc;
    const size_t smem = 3 * (size_t)ctx->K * sizeof(float);
    int grid = 1;
    rc = persistent_grid(ctx, warm_start_kernel, kMHThreads, smem, &grid);
    if (rc) return rc;
    warm_start_kernel<<<grid, kMHThreads, smem, s>>>(mh_params(ctx, cur, 0u, 0));
    CK(cudaGetLastError());
    rc = check_device_error(ctx, "culda_warm_start");
    if (rc) return rc;
    ctx->cur = 1 - cur;
    return rebuild_counts(ctx);
}
