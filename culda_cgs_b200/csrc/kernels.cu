// kernels.cu — the count-rebuild and utility kernels of the one-GPU CGS
// iteration, and the kernel-level C entry points that mirror the reference's
// kernel APIs.  The sampler is in sampler.cu.
//
// Iteration data flow (all resident in HBM; tokens stored word by word, and
// inside a word ordered by their doc's length so neighbouring tokens walk
// theta rows of similar length):
//   prologue_kernel      one Philox4x32-10 uniform per token, and everything the
//                        iteration starts from zero
//   hot_rows_kernel      full phi rows of words split over several work items
//   sample_kernel<G>     the draw (sampler.cu)
//   theta_rebuild_kernel fixed-order sum of the per-item log terms; block per long doc, warp per other doc (longest
//                        first): 16-bit shared-memory histogram of the doc's
//                        new topics (docs of at most 32 tokens: match groups
//                        in registers), CSR compaction in ascending topic,
//                        zero padding, n_k as a column sum.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <numeric>

#include "device_util.cuh"
#include "kernels.cuh"
#include "philox.h"

namespace culda {

// ---------------------------------------------------------- theta rebuild
// Two bins in one persistent launch.  The longest documents (the first
// num_long of doc_order, every one at least the bin threshold long) are taken
// one at a time by a whole CTA from an atomic queue: its eight warps count
// the doc's tokens into one shared histogram.  Every other document is taken
// by one warp (static round robin over the rest of doc_order, longest first).
// Shared memory per warp: K/2 words of packed 16-bit counts (a topic can hold
// at most L_d <= 65535 tokens, so a low half never carries into the high half)
// and K/32 words of a non-zero mask; per block: K n_k partial counts.  The
// block bin uses warp 0's histogram.  The compaction walks the mask in
// ascending topic order, so each row comes out sorted as
// lda_theta_kernel.cu:58-85 leaves it, and only the touched count words are
// cleared again.

namespace {

// Counts tokens [b + first, e) with stride `step` into the packed histogram.
__device__ __forceinline__ void theta_count(int K, int64_t b, int64_t e, int first, int step,
                                            const int32_t *__restrict__ doc_tok,
                                            const uint16_t *__restrict__ topics, uint32_t *cnt, uint32_t *mask,
                                            int32_t *error) {
    // eight tokens per thread in flight: the index loads, then the topic
    // loads they address, then the histogram updates
    constexpr int kInFlight = 8;
    for (int64_t j0 = b + first; j0 < e; j0 += (int64_t)step * kInFlight) {
        int32_t idx[kInFlight];
        uint32_t zz[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) idx[u] = j0 + (int64_t)step * u < e ? doc_tok[j0 + (int64_t)step * u] : -1;
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) zz[u] = idx[u] >= 0 ? (uint32_t)topics[idx[u]] : 0u;
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
            if (idx[u] < 0) continue;
            const uint32_t z = zz[u];
            if (z >= (uint32_t)K) {
                atomicOr(error, kErrTopicRange);
                continue;
            }
            const uint32_t sh = (z & 1u) << 4;
            const uint32_t old = atomicAdd(&cnt[z >> 1], 1u << sh);
            if (((old >> sh) & 0xFFFFu) == 0u) atomicOr(&mask[z >> 5], 1u << (z & 31u));
        }
    }
}

// One warp: the doc's row from its histogram (ascending topic), zero padding
// to the row's previous end, the histogram cleared, n_k partial sums.
__device__ __forceinline__ void theta_compact(int K, int d, int64_t len, int lane, uint32_t *cnt, uint32_t *mask,
                                              uint32_t *nk_acc, int2 *rows, ThetaEntry *theta, int64_t &my_rows,
                                              int64_t &my_nnz, int64_t &my_tok_nnz) {
    const int mwords = K >> 5;
    const int2 row = rows[d];
    const int start = row.x, old_end = row.y;
    int nnz = 0;
    for (int mb = 0; mb < mwords; mb += 32) {
        const int mi = mb + lane;
        const uint32_t mw = mi < mwords ? mask[mi] : 0u;
        const int pc = __popc(mw);
        int incl = pc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        int pos = start + nnz + incl - pc;
        uint32_t bits = mw;
        while (bits) {
            const int bit = __ffs(bits) - 1;
            bits &= bits - 1u;
            const uint32_t z = ((uint32_t)mi << 5) | (uint32_t)bit;
            const uint32_t c = (cnt[z >> 1] >> ((z & 1u) << 4)) & 0xFFFFu;
            theta[pos++] = theta_entry(z, c);
            atomicAdd(&nk_acc[z], c);
        }
        __syncwarp();
        bits = mw;
        while (bits) {
            const int bit = __ffs(bits) - 1;
            bits &= bits - 1u;
            cnt[(((uint32_t)mi << 5) | (uint32_t)bit) >> 1] = 0u;
        }
        if (mi < mwords) mask[mi] = 0u;
        nnz += total;
    }
    __syncwarp();
    const int new_end = start + ((nnz + 31) & ~31);
    const int zend = max(new_end, old_end);
    for (int j = start + nnz + lane; j < zend; j += 32) theta[j] = 0u;
    if (lane == 0) {
        rows[d].y = new_end;
        my_rows += len * (int64_t)(new_end - start);
        my_nnz += nnz;
        my_tok_nnz += len * (int64_t)nnz;
    }
}

// One warp, a doc of at most 32 tokens: no histogram.  Each lane holds one
// token's topic; the lanes with equal topics form a match group whose lowest
// lane writes the entry (topic, group size) at its rank among the groups'
// topics, so the row comes out in ascending topic order as theta_compact
// leaves it.
__device__ __forceinline__ void theta_short(int K, int d, int64_t b, int len, int lane,
                                            const int32_t *__restrict__ doc_tok,
                                            const uint16_t *__restrict__ topics, uint32_t *nk_acc, int2 *rows,
                                            ThetaEntry *theta, int64_t &my_rows, int64_t &my_nnz,
                                            int64_t &my_tok_nnz, int32_t *error) {
    uint32_t z = 0xFFFFFFFFu;
    if (lane < len) {
        const uint32_t t = topics[doc_tok[b + lane]];
        if (t < (uint32_t)K)
            z = t;
        else
            atomicOr(error, kErrTopicRange);
    }
    const unsigned grp = __match_any_sync(0xffffffffu, z);
    const bool lead = z != 0xFFFFFFFFu && __ffs(grp) - 1 == lane;
    const int nnz = __popc(__ballot_sync(0xffffffffu, lead));
    const uint32_t key = lead ? z : 0xFFFFFFFFu;
    int rank = 0;
#pragma unroll 8
    for (int j = 0; j < 32; ++j) rank += __shfl_sync(0xffffffffu, key, j) < key;
    const int2 row = rows[d];
    const int start = row.x, old_end = row.y;
    if (lead) {
        const uint32_t c = (uint32_t)__popc(grp);
        theta[start + rank] = theta_entry(z, c);
        atomicAdd(&nk_acc[z], c);
    }
    const int new_end = start + ((nnz + 31) & ~31);
    const int zend = max(new_end, old_end);
    for (int j = start + nnz + lane; j < zend; j += 32) theta[j] = 0u;
    if (lane == 0) {
        rows[d].y = new_end;
        my_rows += (int64_t)len * (new_end - start);
        my_nnz += nnz;
        my_tok_nnz += (int64_t)len * nnz;
    }
}

// Sum over the CTA's threads, in a fixed order; thread 0 gets it.
__device__ __forceinline__ double theta_block_sum(double x) {
    __shared__ double red[kThetaWarps];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    __syncthreads();  // an earlier sum has been read
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < kThetaWarps; ++w) x += red[w];
    return x;
}

}  // namespace

__global__ void __launch_bounds__(kThetaWarps * 32) theta_rebuild_kernel(
    int K, int num_docs, const int64_t *__restrict__ doc_ptr, const int32_t *__restrict__ doc_tok,
    const uint16_t *__restrict__ topics, const int32_t *__restrict__ doc_order, int num_long, int32_t *long_queue,
    int2 *rows, ThetaEntry *theta, int32_t *nk, int64_t *stats, int32_t *error, const IterationEnd end) {
    extern __shared__ uint32_t sm_u32[];
    __shared__ int s_next;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cwords = K >> 1, mwords = K >> 5;
    uint32_t *nk_acc = sm_u32;
    uint32_t *cnt = sm_u32 + K + warp * (cwords + mwords);
    uint32_t *mask = cnt + cwords;
    for (int i = threadIdx.x; i < K; i += blockDim.x) nk_acc[i] = 0u;
    for (int i = lane; i < cwords + mwords; i += 32) cnt[i] = 0u;
    double ll = 0.0;  // this CTA's share of the sampler's per-item terms, added up at the end
    if (end.stats) {
        if (threadIdx.x == 0) clock_start(&end.stats->rebuild_t0);
        const int share = (end.num_items + gridDim.x - 1) / gridDim.x;
        const int i1 = min((int)(blockIdx.x + 1) * share, end.num_items);
        for (int i = blockIdx.x * share + threadIdx.x; i < i1; i += blockDim.x) ll += end.item_ll[i];
    }
    __syncthreads();

    int64_t my_rows = 0, my_nnz = 0, my_tok_nnz = 0;
    // block bin: one long document per CTA at a time
    if (num_long > 0) {
        uint32_t *bcnt = sm_u32 + K;  // warp 0's histogram
        uint32_t *bmask = bcnt + cwords;
        for (;;) {
            if (threadIdx.x == 0) s_next = atomicAdd(long_queue, 1);
            __syncthreads();
            const int i = s_next;
            __syncthreads();  // every thread has read s_next before thread 0 overwrites it
            if (i >= num_long) break;
            const int d = doc_order[i];
            const int64_t b = doc_ptr[d], e = doc_ptr[d + 1];
            if (e - b > 65535) {
                if (threadIdx.x == 0) atomicOr(error, kErrLongDoc);
                continue;
            }
            theta_count(K, b, e, threadIdx.x, kThetaWarps * 32, doc_tok, topics, bcnt, bmask, error);
            __syncthreads();
            if (warp == 0) theta_compact(K, d, e - b, lane, bcnt, bmask, nk_acc, rows, theta, my_rows, my_nnz,
                                         my_tok_nnz);
            __syncthreads();  // the histogram is clear again before the next document
        }
    }
    // warp bin: the remaining documents, one per warp
    const int nw = gridDim.x * kThetaWarps;
    for (int i = num_long + blockIdx.x * kThetaWarps + warp; i < num_docs; i += nw) {
        const int d = doc_order ? doc_order[i] : i;
        const int64_t b = doc_ptr[d], e = doc_ptr[d + 1];
        if (e - b > 65535) {
            if (lane == 0) atomicOr(error, kErrLongDoc);
            continue;
        }
        if (e - b <= 32) {
            theta_short(K, d, b, (int)(e - b), lane, doc_tok, topics, nk_acc, rows, theta, my_rows, my_nnz,
                        my_tok_nnz, error);
            continue;
        }
        theta_count(K, b, e, lane, 32, doc_tok, topics, cnt, mask, error);
        __syncwarp();
        theta_compact(K, d, e - b, lane, cnt, mask, nk_acc, rows, theta, my_rows, my_nnz, my_tok_nnz);
    }
    __syncthreads();
    if (nk)
        for (int i = threadIdx.x; i < K; i += blockDim.x)
            if (nk_acc[i]) atomicAdd(&nk[i], (int)nk_acc[i]);
    if (lane == 0 && stats) {
        atomicAdd(reinterpret_cast<unsigned long long *>(&stats[0]), (unsigned long long)my_rows);
        atomicAdd(reinterpret_cast<unsigned long long *>(&stats[1]), (unsigned long long)my_nnz);
        atomicAdd(reinterpret_cast<unsigned long long *>(&stats[2]), (unsigned long long)my_tok_nnz);
    }
    if (!end.stats) return;
    ll = theta_block_sum(ll);  // barriers inside: the CTA's atomics above are issued
    if (threadIdx.x == 0) {
        end.partials[blockIdx.x] = ll;
        clock_end(&end.stats->rebuild_t0);
        __threadfence();
        s_next = atomicAdd(end.done, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_next) return;
    // the last CTA: every other CTA's atomics and partials are visible
    __threadfence();
    ll = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) ll += __ldcg(end.partials + i);
    // the statistics word by word, one load per thread; thread 0's fields are the sums below
    constexpr int kWords = (int)(sizeof(DevStats) / sizeof(unsigned long long));
    const uint32_t iter = *end.iteration_dev;
    DevStats *out = end.ring + iter % kStatsRing;
    unsigned long long word = 0ull;
    if (threadIdx.x < kWords) word = __ldcg(reinterpret_cast<const unsigned long long *>(end.stats) + threadIdx.x);
    const int32_t err = threadIdx.x == 0 ? __ldcg(error) : 0;
    ll = theta_block_sum(ll);
    if (threadIdx.x == 0) {
        end.stats->ll_sum = ll;
        out->ll_sum = ll;
        out->error = err;
        out->iteration = iter;
        *end.iteration_dev = iter + 1u;
    } else if (threadIdx.x < kWords && threadIdx.x != offsetof(DevStats, error) / sizeof(unsigned long long)) {
        reinterpret_cast<unsigned long long *>(out)[threadIdx.x] = word;
    }
}
static_assert(sizeof(DevStats) % sizeof(unsigned long long) == 0 && offsetof(DevStats, ll_sum) == 0 &&
                  offsetof(DevStats, error) % sizeof(unsigned long long) == 0 &&
                  offsetof(DevStats, iteration) == offsetof(DevStats, error) + sizeof(int32_t),
              "the rebuild's last CTA copies the statistics as 64-bit words");

size_t theta_smem_bytes(int k) {
    return ((size_t)k + (size_t)kThetaWarps * (size_t)((k >> 1) + (k >> 5))) * sizeof(uint32_t);
}

int theta_blocks_per_sm(int k) {
    const size_t smem = theta_smem_bytes(k);
    if (allow_smem(reinterpret_cast<const void *>(&theta_rebuild_kernel), smem) != cudaSuccess) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, theta_rebuild_kernel, kThetaWarps * 32, smem) !=
        cudaSuccess)
        return 0;
    return n;
}

cudaError_t launch_theta_rebuild(int k, int num_docs, const int64_t *doc_ptr, const int32_t *doc_tok,
                                 const uint16_t *topics, const int32_t *doc_order, int2 *rows, ThetaEntry *theta,
                                 int32_t *nk, int64_t *stats, int32_t *error, int grid, cudaStream_t s,
                                 int num_long, int32_t *long_queue, const IterationEnd &end) {
    if (num_long > 0 && (!doc_order || !long_queue || num_long > num_docs)) return cudaErrorInvalidValue;
    const size_t smem = theta_smem_bytes(k);
    cudaError_t e = allow_smem(reinterpret_cast<const void *>(&theta_rebuild_kernel), smem);
    if (e != cudaSuccess) return e;
    if (num_long > 0 && !end.stats) {
        e = cudaMemsetAsync(long_queue, 0, sizeof(int32_t), s);
        if (e != cudaSuccess) return e;
    }
    theta_rebuild_kernel<<<grid, kThetaWarps * 32, smem, s>>>(k, num_docs, doc_ptr, doc_tok, topics, doc_order,
                                                              num_long > 0 ? num_long : 0, long_queue, rows, theta,
                                                              nk, stats, error, end);
    return cudaGetLastError();
}

// -------------------------------------------------------- small utilities

// z[i] = floor(x0 * K / 2^32), x0 = Philox(seed, {t, 0, 1}) with t the
// token's word-major index.
__global__ void init_topics_kernel(int64_t n, int k, uint64_t seed, const int32_t *__restrict__ tok_index,
                                   uint16_t *z) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t t = tok_index ? (uint64_t)tok_index[i] : (uint64_t)i;
        z[i] = (uint16_t)bounded_from_bits(philox_token(seed, t, 0u, kPurposeInit), (uint32_t)k);
    }
}

cudaError_t launch_init_topics(int64_t n, int k, uint64_t seed, const int32_t *tok_index, uint16_t *z,
                               cudaStream_t s) {
    init_topics_kernel<<<grid_for(n), 256, 0, s>>>(n, k, seed, tok_index, z);
    return cudaGetLastError();
}

// One Philox4x32-10 block per token, computed by all threads in parallel
// (the sampler's groups would otherwise leave most lanes idle while a
// segment's one or two tokens draw theirs), after the iteration's counters,
// totals and hot rows are cleared: one launch instead of five graph nodes.
__global__ void __launch_bounds__(256) prologue_kernel(const PrologueParams p) {
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    if (t0 == 0) {
        *p.counter = 0;
        *p.warp_counter = 0;
        *p.theta_queue = 0;
        *p.done = 0;
        DevStats *st = p.stats;
        st->row_entries = st->nnz = st->token_nnz = 0;
        st->mh_accepted = st->mh_proposed = 0ull;
        st->sample_t0 = st->rebuild_t0 = ~0ull;
        st->sample_t1 = st->rebuild_t1 = 0ull;
    }
    if (p.nk_next)
        for (int64_t i = t0; i < p.k; i += nt) p.nk_next[i] = 0;
    for (int64_t i = t0; i < p.k; i += nt) p.inv[i] = 1.0f / ((float)p.nk[i] + p.vbeta);
    for (int64_t i = t0; i < p.hot_n; i += nt) p.hot_phi[i] = 0;
    const uint32_t iter = p.iteration_dev ? *p.iteration_dev : p.iteration;
    const int32_t *__restrict__ tok_index = p.tok_index;
    float *__restrict__ u = p.u;
    const int64_t n = p.n;
    for (int64_t i = t0; i < n; i += nt) {
        const uint64_t t = tok_index ? (uint64_t)__ldg(tok_index + i) : (uint64_t)i;
        u[i] = uniform_from_bits(philox_token(p.seed, t, iter, kPurposeSample));
    }
}

cudaError_t launch_prologue(const PrologueParams &p, cudaStream_t s) {
    prologue_kernel<<<grid_for(std::max<int64_t>(std::max<int64_t>(p.n, p.hot_n), p.k)), 256, 0, s>>>(p);
    return cudaGetLastError();
}

__global__ void doc_check_kernel(int64_t n, int num_docs, const int32_t *__restrict__ doc_ids, int32_t *doc_count,
                                 int32_t *error) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int d = doc_ids[t];
        if ((unsigned)d < (unsigned)num_docs)
            atomicAdd(&doc_count[d], 1);
        else
            atomicOr(error, kErrDocRange);
    }
}

cudaError_t launch_doc_check(int64_t n, int num_docs, const int32_t *doc_ids, int32_t *doc_count, int32_t *error,
                             cudaStream_t s) {
    doc_check_kernel<<<grid_for(n), 256, 0, s>>>(n, num_docs, doc_ids, doc_count, error);
    return cudaGetLastError();
}

__global__ void check_topics_kernel(int64_t n, int k, const uint16_t *__restrict__ z, int32_t *error) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        if (z[t] >= (uint32_t)k) atomicOr(error, kErrTopicRange);
}

cudaError_t launch_check_topics(int64_t n, int k, const uint16_t *z, int32_t *error, cudaStream_t s) {
    check_topics_kernel<<<grid_for(n), 256, 0, s>>>(n, k, z, error);
    return cudaGetLastError();
}

// Thread per token: the word is found by binary search of word_ptr (V+1
// ascending offsets, L2-resident), so a Zipf-head word of millions of tokens
// is spread over the whole grid instead of one warp.
__global__ void order_keys_kernel(int num_words, int64_t num_tokens, const int64_t *__restrict__ word_ptr,
                                  const int32_t *__restrict__ doc_ids, const int64_t *__restrict__ doc_ptr,
                                  uint64_t *keys) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < num_tokens;
         t += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = num_words - 1;  // the last word w with word_ptr[w] <= t
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(word_ptr + mid) <= t)
                lo = mid;
            else
                hi = mid - 1;
        }
        const int d = doc_ids[t];
        const int64_t len = min(doc_ptr[d + 1] - doc_ptr[d], (int64_t)65535);
        keys[t] = ((uint64_t)lo << 16) | (uint64_t)(65535 - len);
    }
}

cudaError_t launch_order_keys(int num_words, int64_t num_tokens, const int64_t *word_ptr, const int32_t *doc_ids,
                              const int64_t *doc_ptr, uint64_t *keys, cudaStream_t s) {
    if (num_tokens <= 0) return cudaSuccess;
    order_keys_kernel<<<grid_for(num_tokens), 256, 0, s>>>(num_words, num_tokens, word_ptr, doc_ids, doc_ptr, keys);
    return cudaGetLastError();
}

// 32-bit keys for vocabularies of at most 2^24 words: the word above an 8-bit
// log-linear length class, 16 classes per doubling (the position of the
// length's leading one and the 4 bits after it), longest first.  Docs in one
// class keep their input order (the sort is stable), so a doc's tokens inside
// a word stay contiguous.
__global__ void order_keys32_kernel(int num_words, int64_t num_tokens, const int64_t *__restrict__ word_ptr,
                                    const int32_t *__restrict__ doc_ids, const int64_t *__restrict__ doc_ptr,
                                    uint32_t *keys) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < num_tokens;
         t += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = num_words - 1;  // the last word w with word_ptr[w] <= t
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(word_ptr + mid) <= t)
                lo = mid;
            else
                hi = mid - 1;
        }
        const int d = doc_ids[t];
        const int64_t l64 = doc_ptr[d + 1] - doc_ptr[d];
        const uint32_t len = l64 < 1 ? 1u : l64 > 65535 ? 65535u : (uint32_t)l64;
        const uint32_t msb = 31u - __clz(len);                         // 0 .. 15
        const uint32_t frac = ((len << (31u - msb)) >> 27) & 15u;      // the 4 bits after the leading one
        keys[t] = ((uint32_t)lo << 8) | (255u - (msb * 16u + frac));
    }
}

cudaError_t launch_order_keys32(int num_words, int64_t num_tokens, const int64_t *word_ptr, const int32_t *doc_ids,
                                const int64_t *doc_ptr, uint32_t *keys, cudaStream_t s) {
    if (num_tokens <= 0) return cudaSuccess;
    if (num_words > (1 << 24)) return cudaErrorInvalidValue;
    order_keys32_kernel<<<grid_for(num_tokens), 256, 0, s>>>(num_words, num_tokens, word_ptr, doc_ids, doc_ptr,
                                                             keys);
    return cudaGetLastError();
}

template <class T>
__global__ void gather_kernel(int64_t n, const int32_t *__restrict__ index, const T *__restrict__ src, T *dst) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[index[i]];
}

template <class T>
__global__ void scatter_kernel(int64_t n, const int32_t *__restrict__ index, const T *__restrict__ src, T *dst) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[index[i]] = src[i];
}

template <class T>
cudaError_t launch_gather(int64_t n, const int32_t *index, const T *src, T *dst, cudaStream_t s) {
    gather_kernel<T><<<grid_for(n), 256, 0, s>>>(n, index, src, dst);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_scatter(int64_t n, const int32_t *index, const T *src, T *dst, cudaStream_t s) {
    scatter_kernel<T><<<grid_for(n), 256, 0, s>>>(n, index, src, dst);
    return cudaGetLastError();
}

template cudaError_t launch_gather<int32_t>(int64_t, const int32_t *, const int32_t *, int32_t *, cudaStream_t);
template cudaError_t launch_gather<uint16_t>(int64_t, const int32_t *, const uint16_t *, uint16_t *, cudaStream_t);
template cudaError_t launch_scatter<uint16_t>(int64_t, const int32_t *, const uint16_t *, uint16_t *, cudaStream_t);

__global__ void iota_kernel(int64_t n, int32_t *v) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v[i] = (int32_t)i;
}

cudaError_t launch_iota(int64_t n, int32_t *v, cudaStream_t s) {
    iota_kernel<<<grid_for(n), 256, 0, s>>>(n, v);
    return cudaGetLastError();
}

// ------------------------------------------------------- dense phi (API)
// The V x K table is written once (4 V K bytes, the bound), so the kernel is
// built to keep row stores in flight: a warp takes a word, counts its topics
// in a private histogram of packed 16-bit counts and stores the row with
// 16-byte stores while clearing the histogram.  (A CTA per word with three
// barriers each took 682 us at 50k words, 4.1M tokens and K = 1024; this form
// takes 50 us and the clearing 4.5 us: 213 MB at 0.65 of the measured copy bandwidth.)
//
// The grid cuts the vocabulary into shares of equal cost, a token costing 1
// and a row K / 4.  Only words of at least kPhiSplit tokens are cut: their
// slices are added with atomics into a row that phi_zero_split_kernel has
// cleared.  Ranges of at least kPhiLong tokens are counted by the whole CTA.
constexpr int kPhiThreads = 256;
constexpr int kPhiWarps = kPhiThreads / 32;
constexpr int64_t kPhiSplit = 8192;
constexpr int64_t kPhiLong = 2048;  // below 65536: a warp's counts have 16 bits

// Where share c of `shares` begins: a word and a token offset inside it.  One
// warp: 32-way search for the last word whose cost prefix is at most the
// share's, the same in every lane.
__device__ __forceinline__ void phi_share(const int64_t *__restrict__ word_ptr, int V, int K, int c, int shares,
                                          int lane, int &word, int64_t &off) {
    const int64_t base = word_ptr[0], row = K / 4;
    const int64_t total = word_ptr[V] - base + row * V;
    const int64_t target = total / shares * c + total % shares * c / shares;
    off = 0;
    if (c >= shares) {
        word = V;
        return;
    }
    int lo = 0, n = V;  // the word lies in [lo, lo + n)
    while (n > 1) {
        const int step = (n + 31) / 32, at = lane * step;
        const bool le = at < n && word_ptr[lo + at] - base + row * (lo + at) <= target;
        const unsigned m = __ballot_sync(0xffffffffu, le);
        const int j = m ? 31 - __clz(m) : 0;
        lo += j * step;
        n = min(step, n - j * step);
    }
    word = lo;
    if (word_ptr[lo + 1] - word_ptr[lo] >= kPhiSplit)
        off = max((int64_t)0, min(target - (word_ptr[lo] - base + row * lo) - row, word_ptr[lo + 1] - word_ptr[lo]));
}

__global__ void __launch_bounds__(kPhiThreads) phi_zero_split_kernel(int K, int V, int shares,
                                                                     const int64_t *__restrict__ word_ptr,
                                                                     int32_t *phi) {
    const int lane = threadIdx.x & 31;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= shares) return;
    int w;
    int64_t off;
    phi_share(word_ptr, V, K, c, shares, lane, w, off);
    if (off > 0)
        for (int j = lane; j < K; j += 32) phi[(size_t)w * K + j] = 0;
}

__global__ void __launch_bounds__(kPhiThreads) update_phi_kernel(int K, int V, const int64_t *__restrict__ word_ptr,
                                                                 const uint16_t *__restrict__ topics, int32_t *phi,
                                                                 int32_t *nk, int32_t *error, bool wide) {
    extern __shared__ int sm_i32[];
    int *acc = sm_i32;                                        // [K] the CTA's topic totals
    int *coop = sm_i32 + K;                                   // [K] whole-CTA histogram (zero between uses)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t *hist = reinterpret_cast<uint32_t *>(sm_i32 + 2 * K) + warp * (K / 2);  // this warp's packed counts
    __shared__ int s_next, s_num_long, s_w[2];
    __shared__ int64_t s_off[2];
    __shared__ int s_long[kPhiThreads];
    for (int j = tid; j < 2 * K + kPhiWarps * (K / 2); j += kPhiThreads) sm_i32[j] = 0;
    if (warp < 2) {
        int w;
        int64_t off;
        phi_share(word_ptr, V, K, blockIdx.x + warp, gridDim.x, lane, w, off);
        if (lane == 0) {
            s_w[warp] = w;
            s_off[warp] = off;
        }
    }
    __syncthreads();
    const int w0 = s_w[0], w1 = s_w[1];
    const int64_t off0 = s_off[0], off1 = s_off[1];
    // this CTA's tokens of word w, [b, e) in all; part: other CTAs add to the row too
    auto range = [&](int w, int64_t &b, int64_t &e, bool &part) {
        b = word_ptr[w];
        e = word_ptr[w + 1];
        part = false;
        if (w == w1) {
            e = b + off1;
            part = true;
        }
        if (w == w0 && off0 > 0) {
            b += off0;
            part = true;
        }
    };
    const int w_end = w1 + (off1 > 0 ? 1 : 0);
    for (int wb = w0; wb < w_end; wb += kPhiThreads) {
        const int wn = min(wb + kPhiThreads, w_end);
        if (tid == 0) {
            s_next = wb;
            s_num_long = 0;
        }
        __syncthreads();
        if (wb + tid < wn) {
            int64_t b, e;
            bool part;
            range(wb + tid, b, e, part);
            if (part || e - b >= kPhiLong) s_long[atomicAdd(&s_num_long, 1)] = wb + tid;
        }
        __syncthreads();
        const int num_long = s_num_long;
        for (int i = 0; i < num_long; ++i) {
            const int w = s_long[i];
            int64_t b, e;
            bool part;
            range(w, b, e, part);
            for (int64_t t0 = b + tid; t0 < e; t0 += 8 * kPhiThreads) {
                uint32_t z[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) z[u] = t0 + u * kPhiThreads < e ? topics[t0 + u * kPhiThreads] : 0u;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (t0 + u * kPhiThreads >= e) continue;
                    if (z[u] < (uint32_t)K)
                        atomicAdd(&coop[z[u]], 1);
                    else if (error)
                        atomicOr(error, kErrTopicRange);
                }
            }
            __syncthreads();
            int32_t *row = phi + (size_t)w * K;
            for (int j = tid; j < K; j += kPhiThreads) {
                const int n = coop[j];
                if (!part)
                    row[j] = n;
                else if (n)
                    atomicAdd(&row[j], n);
                if (n) atomicAdd(&acc[j], n);
                coop[j] = 0;
            }
            __syncthreads();
        }
        for (;;) {
            int w = 0;
            if (lane == 0) w = atomicAdd(&s_next, 1);
            w = __shfl_sync(0xffffffffu, w, 0);
            if (w >= wn) break;
            int64_t b, e;
            bool part;
            range(w, b, e, part);
            if (part || e - b >= kPhiLong) continue;
            for (int64_t t0 = b + lane; t0 < e; t0 += 4 * 32) {
                uint32_t z[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) z[u] = t0 + 32 * u < e ? topics[t0 + 32 * u] : 0u;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (t0 + 32 * u >= e) continue;
                    if (z[u] < (uint32_t)K) {
                        atomicAdd(&hist[z[u] >> 1], 1u << ((z[u] & 1u) << 4));
                        atomicAdd(&acc[z[u]], 1);
                    } else if (error) {
                        atomicOr(error, kErrTopicRange);
                    }
                }
            }
            __syncwarp();
            int32_t *row = phi + (size_t)w * K;
            if (wide) {
                for (int j = lane; j < K / 4; j += 32) {
                    const uint2 q = reinterpret_cast<const uint2 *>(hist)[j];
                    reinterpret_cast<uint2 *>(hist)[j] = make_uint2(0u, 0u);
                    reinterpret_cast<int4 *>(row)[j] = make_int4((int)(q.x & 0xFFFFu), (int)(q.x >> 16),
                                                                 (int)(q.y & 0xFFFFu), (int)(q.y >> 16));
                }
            } else {  // phi is not 16-byte aligned
                for (int j = lane; j < K / 2; j += 32) {
                    const uint32_t q = hist[j];
                    hist[j] = 0u;
                    row[2 * j] = (int)(q & 0xFFFFu);
                    row[2 * j + 1] = (int)(q >> 16);
                }
            }
            __syncwarp();  // the histogram is clear before the next word
        }
        __syncthreads();  // every warp has left this stretch before s_next and s_long are rewritten
    }
    for (int j = tid; j < K; j += kPhiThreads)
        if (acc[j]) atomicAdd(&nk[j], acc[j]);
}

cudaError_t launch_update_phi(int k, int num_words, const int64_t *word_ptr, const uint16_t *topics, int32_t *phi,
                              int32_t *nk, int32_t *error, cudaStream_t s) {
    const size_t smem = (2 * (size_t)k + (size_t)kPhiWarps * (size_t)(k / 2)) * sizeof(int);
    cudaError_t e = allow_smem(reinterpret_cast<const void *>(&update_phi_kernel), smem);
    if (e != cudaSuccess) return e;
    int dev = 0, bps = 0;
    cudaGetDevice(&dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, update_phi_kernel, kPhiThreads, smem);
    if (e != cudaSuccess) return e;
    const int grid = std::max(1, std::min(num_words, num_sms(dev) * std::max(bps, 1)));
    phi_zero_split_kernel<<<(grid + kPhiWarps - 1) / kPhiWarps, kPhiThreads, 0, s>>>(k, num_words, grid, word_ptr,
                                                                                      phi);
    update_phi_kernel<<<grid, kPhiThreads, smem, s>>>(k, num_words, word_ptr, topics, phi, nk, error,
                                                      ((uintptr_t)phi & 15u) == 0);
    return cudaGetLastError();
}

// phi_head = (phi + beta) / (n_k + beta * V), the reference's float quotient
// (lda_phi_kernel.cu:26) kept in FP32.  Bound by its 8 V K bytes: a thread
// keeps one group of four topics (the grid's stride is a multiple of K / 4
// groups), so the four denominators are formed once and every row costs one
// 16-byte load, four divisions and one 16-byte store.  (One topic per thread
// with a 64-bit modulo each: 141 us on 410 MB; this form: 61 us, all of the
// measured copy bandwidth.)  Tables that are not 16-byte aligned take the
// scalar form.
__global__ void __launch_bounds__(256) phi_head_kernel(int K, float beta, int V, const int4 *__restrict__ phi,
                                                       const int32_t *__restrict__ nk, float4 *__restrict__ out) {
    const float vb = beta * (float)V;
    const int64_t total = (int64_t)(K / 4) * V, stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int c = 4 * (int)(i % (K / 4));
    const float d0 = (float)nk[c] + vb, d1 = (float)nk[c + 1] + vb, d2 = (float)nk[c + 2] + vb,
                d3 = (float)nk[c + 3] + vb;
    for (; i < total; i += 4 * stride) {
        int4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < total) v[u] = __ldcs(phi + i + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < total)
                __stcs(out + i + u * stride,
                       make_float4(__fdiv_rn((float)v[u].x + beta, d0), __fdiv_rn((float)v[u].y + beta, d1),
                                   __fdiv_rn((float)v[u].z + beta, d2), __fdiv_rn((float)v[u].w + beta, d3)));
    }
}

__global__ void phi_head_scalar_kernel(int K, float beta, int V, const int32_t *__restrict__ phi,
                                       const int32_t *__restrict__ nk, float *out) {
    const int64_t total = (int64_t)K * V;
    const float vb = beta * (float)V;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(i % K);
        out[i] = __fdiv_rn((float)phi[i] + beta, (float)nk[k] + vb);
    }
}

cudaError_t launch_phi_head(int k, float beta, int num_words, const int32_t *phi, const int32_t *nk, float *out,
                            cudaStream_t s) {
    int dev = 0;
    cudaGetDevice(&dev);
    if ((((uintptr_t)phi | (uintptr_t)out) & 15u) == 0) {
        // blocks whose threads together cover whole rows: a multiple of (K/4) / gcd(K/4, 256)
        const int q = (k / 4) / std::gcd(k / 4, 256);
        const int64_t need = ((int64_t)(k / 4) * num_words + 255) / 256;
        const int blocks = (int)std::min<int64_t>((int64_t)num_sms(dev) * 8, need);
        phi_head_kernel<<<(blocks + q - 1) / q * q, 256, 0, s>>>(k, beta, num_words,
                                                                 reinterpret_cast<const int4 *>(phi), nk,
                                                                 reinterpret_cast<float4 *>(out));
    } else {
        phi_head_scalar_kernel<<<num_sms(dev) * 8, 256, 0, s>>>(k, beta, num_words, phi, nk, out);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------- joint log-likelihood
// FP64 sum of  sum_{w,k: n>0} [lgamma(n_wk + beta) - lgamma(beta)]
//            + sum_{d,k: n>0} [lgamma(n_dk + alpha) - lgamma(alpha)]
//            - sum_d lgamma(L_d + K alpha) - sum_k lgamma(n_k + V beta).
// A term depends on its count alone and nearly all counts are small, so the
// kernel counts how often each count below kJointTable occurs (1, 2 and 3 in
// registers, the others in shared memory) and multiplies at the end; what
// remains is reading the topics and theta (74 MB at 12.2M tokens: 11 us at the
// measured copy bandwidth).  Words come as the sampler's work items, largest
// first: a warp counts an item's topics in packed 16-bit counts, a whole CTA the
// first num_long items (kPhiLong tokens or more), and a word split over several
// items is read from its hot row.  Items, theta, docs and topics go to fixed
// threads and the last CTA adds the CTAs' sums in order, so the result is
// reproducible.  (An lgamma per non-zero, a CTA per word, and one thread for the
// docs' terms took 1305 us at 12.2M tokens and K = 1024; a table of the terms
// and an FP64 sum per non-zero, few lanes at a time, 101 us; this form 71 us.)
constexpr int kJointTable = 256;
static_assert(kJointTable == kPhiThreads && 2 * kJointTable < kJointCounters, "a thread per tabulated count");

__global__ void __launch_bounds__(kPhiThreads) loglik_joint_kernel(const JointParams p) {
    extern __shared__ int sm_joint[];
    int *coop = sm_joint;  // [K] whole-CTA histogram
    const int K = p.k, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t *hist = reinterpret_cast<uint32_t *>(coop + K) + warp * (K / 2);  // this warp's packed counts
    __shared__ double red[kPhiThreads];
    __shared__ unsigned word_of[kJointTable], doc_of[kJointTable];  // how often a count occurs
    __shared__ bool s_last;
    double s = 0.0, c = 0.0;
    auto add = [&](double x) {
        const double t = s + x;
        if (fabs(s) >= fabs(x))
            c += (s - t) + x;
        else
            c += (x - t) + s;
        s = t;
    };
    unsigned w1 = 0, w2 = 0, w3 = 0, d1 = 0, d2 = 0, d3 = 0;
    auto word_term = [&](uint32_t n) {
        w1 += n == 1u;
        w2 += n == 2u;
        w3 += n == 3u;
        if (n > 3u) {
            if (n < kJointTable)
                atomicAdd(&word_of[n], 1u);
            else
                add(lgamma((double)n + p.beta) - p.lg_beta);
        }
    };
    auto doc_term = [&](uint32_t e) {
        const uint32_t n = e & 0xFFFFu;
        d1 += n == 1u;
        d2 += n == 2u;
        d3 += n == 3u;
        if (n > 3u) {
            if (n < kJointTable)
                atomicAdd(&doc_of[n], 1u);
            else
                add(lgamma((double)n + p.alpha) - p.lg_alpha);
        }
    };
    word_of[tid] = doc_of[tid] = 0u;
    for (int j = tid; j < K + kPhiWarps * (K / 2); j += kPhiThreads) coop[j] = 0;
    __syncthreads();
    for (int i = blockIdx.x; i < p.num_long; i += gridDim.x) {
        const culda_item it = p.items[i];
        if (it.hot >= 0) {
            if (it.first)
                for (int j = tid; j < K; j += kPhiThreads) word_term((uint32_t)p.hot_phi[(size_t)it.hot * K + j]);
            continue;  // the same branch in every thread
        }
        const int64_t e = it.begin + it.count;
        for (int64_t t0 = it.begin + tid; t0 < e; t0 += 8 * kPhiThreads) {
            uint32_t z[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) z[u] = t0 + u * kPhiThreads < e ? p.topics[t0 + u * kPhiThreads] : 0u;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (t0 + u * kPhiThreads >= e) continue;
                if (z[u] < (uint32_t)K)
                    atomicAdd(&coop[z[u]], 1);
                else
                    atomicOr(p.error, kErrTopicRange);
            }
        }
        __syncthreads();
        for (int j = tid; j < K; j += kPhiThreads) {
            word_term((uint32_t)coop[j]);
            coop[j] = 0;
        }
        __syncthreads();
    }
    // a warp's items, the topics of the next one's first 128 tokens on their way
    // while the current one is counted, and the item after it
    const int stride = gridDim.x * kPhiWarps;
    auto load_item = [&](int i) { return i < p.num_items ? p.items[i] : culda_item{0, 0, 0, -1, 0, 0, 0}; };
    auto load_topics = [&](const culda_item &it, uint32_t z[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            z[u] = it.hot < 0 && lane + 32 * u < it.count ? p.topics[it.begin + lane + 32 * u] : 0u;
    };
    const int i0 = p.num_long + blockIdx.x * kPhiWarps + warp;
    culda_item it = load_item(i0), ahead = load_item(i0 + stride);
    uint32_t z[4], next_z[4];
    load_topics(it, z);
    for (int i = i0; i < p.num_items; i += stride) {
        const culda_item after = load_item(i + 2 * stride);
        load_topics(ahead, next_z);
        if (it.hot >= 0) {
            if (it.first)
                for (int j = lane; j < K; j += 32) word_term((uint32_t)p.hot_phi[(size_t)it.hot * K + j]);
        } else if (it.count <= 128) {
            // the tokens are few: the lane whose token came first to its topic reads the
            // topic's count, instead of a pass over K counts
            bool first[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = lane + 32 * u < it.count;
                first[u] = false;
                if (in && z[u] < (uint32_t)K) {
                    const uint32_t sh = (z[u] & 1u) << 4;
                    first[u] = ((atomicAdd(&hist[z[u] >> 1], 1u << sh) >> sh) & 0xFFFFu) == 0u;
                } else if (in) {
                    atomicOr(p.error, kErrTopicRange);
                }
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (first[u]) word_term((hist[z[u] >> 1] >> ((z[u] & 1u) << 4)) & 0xFFFFu);
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (first[u]) hist[z[u] >> 1] = 0u;
            __syncwarp();
        } else {
            for (int t0 = 0; t0 < it.count; t0 += 128) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int t = t0 + lane + 32 * u;
                    if (t >= it.count) continue;
                    const uint32_t x = t0 == 0 ? z[u] : (uint32_t)p.topics[it.begin + t];
                    if (x < (uint32_t)K)
                        atomicAdd(&hist[x >> 1], 1u << ((x & 1u) << 4));
                    else
                        atomicOr(p.error, kErrTopicRange);
                }
            }
            __syncwarp();
            for (int j = lane; j < K / 4; j += 32) {
                const uint2 q = reinterpret_cast<const uint2 *>(hist)[j];
                if ((q.x | q.y) == 0u) continue;
                reinterpret_cast<uint2 *>(hist)[j] = make_uint2(0u, 0u);
                word_term(q.x & 0xFFFFu);
                word_term(q.x >> 16);
                word_term(q.y & 0xFFFFu);
                word_term(q.y >> 16);
            }
            __syncwarp();
        }
        it = ahead;
        ahead = after;
#pragma unroll
        for (int u = 0; u < 4; ++u) z[u] = next_z[u];
    }
    // theta as one array: past the end of a row it holds zeros
    const int64_t n4 = p.theta_cap / 4, threads = (int64_t)gridDim.x * kPhiThreads;  // capacity: a multiple of 32
    for (int64_t i = (int64_t)blockIdx.x * kPhiThreads + tid; i < n4; i += 4 * threads) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            v[u] = i + u * threads < n4 ? __ldg(reinterpret_cast<const uint4 *>(p.theta) + i + u * threads)
                                        : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            doc_term(v[u].x);
            doc_term(v[u].y);
            doc_term(v[u].z);
            doc_term(v[u].w);
        }
    }
    const double ka = (double)K * p.alpha, vb = (double)p.num_words * p.beta;
    for (int d = blockIdx.x * kPhiThreads + tid; d < p.num_docs; d += gridDim.x * kPhiThreads)
        add(-lgamma((double)(p.doc_ptr[d + 1] - p.doc_ptr[d]) + ka));
    for (int k = blockIdx.x * kPhiThreads + tid; k < K; k += gridDim.x * kPhiThreads)
        add(-lgamma((double)p.nk[k] + vb));
    // how often each count occurred, over all CTAs (the last one multiplies)
    if (w1 | d1) {
        atomicAdd(&word_of[1], w1);
        atomicAdd(&doc_of[1], d1);
    }
    if (w2 | d2) {
        atomicAdd(&word_of[2], w2);
        atomicAdd(&doc_of[2], d2);
    }
    if (w3 | d3) {
        atomicAdd(&word_of[3], w3);
        atomicAdd(&doc_of[3], d3);
    }
    __syncthreads();
    if (word_of[tid]) atomicAdd(&p.counts[tid], word_of[tid]);
    if (doc_of[tid]) atomicAdd(&p.counts[kJointTable + tid], doc_of[tid]);
    auto block_sum = [&](double x) {
        red[tid] = x;
        __syncthreads();
        for (int w = kPhiThreads / 2; w > 0; w >>= 1) {
            if (tid < w) red[tid] += red[tid + w];
            __syncthreads();
        }
    };
    block_sum(s + c);
    if (tid == 0) {
        p.partials[blockIdx.x] = red[0];
        __threadfence();
        s_last = atomicAdd(&p.counts[2 * kJointTable], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    s = c = 0.0;
    for (int i = tid; i < (int)gridDim.x; i += kPhiThreads) add(__ldcg(p.partials + i));
    // count tid's terms, for the words and for the docs
    const unsigned nw = __ldcg(p.counts + tid), nd = __ldcg(p.counts + kJointTable + tid);
    if (nw) add((double)nw * (lgamma((double)tid + p.beta) - p.lg_beta));
    if (nd) add((double)nd * (lgamma((double)tid + p.alpha) - p.lg_alpha));
    block_sum(s + c);
    if (tid == 0) *p.result = red[0];
}

cudaError_t launch_loglik_joint(const JointParams &p, int max_partials, cudaStream_t s) {
    const size_t smem = ((size_t)p.k + (size_t)kPhiWarps * (size_t)(p.k / 2)) * sizeof(int);
    cudaError_t e = allow_smem(reinterpret_cast<const void *>(&loglik_joint_kernel), smem);
    if (e != cudaSuccess) return e;
    int dev = 0, bps = 0;
    cudaGetDevice(&dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, loglik_joint_kernel, kPhiThreads, smem);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(p.counts, 0, kJointCounters * sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    // no more CTAs than have a warp's worth of words or docs each
    const int64_t need = ((int64_t)std::max(p.num_items, p.num_docs) + kPhiWarps - 1) / kPhiWarps;
    const int grid = (int)std::max<int64_t>(
        1, std::min<int64_t>(std::min(max_partials, num_sms(dev) * std::max(bps, 1)), need));
    loglik_joint_kernel<<<grid, kPhiThreads, smem, s>>>(p);
    return cudaGetLastError();
}

int64_t long_items(const culda_item *items, int64_t n) {
    return std::partition_point(items, items + n, [](const culda_item &x) { return x.count >= kPhiLong; }) - items;
}

int num_sms(int device) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) n = 148;
    return n;
}

}  // namespace culda

// ===================================================== kernel-level C API
using namespace culda;

static int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return CULDA_OK;
    set_global_error("CUDA error: %s", cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? CULDA_ERR_OOM : CULDA_ERR_CUDA;
}

static bool valid_k(int32_t k) { return k >= 32 && k <= 4096 && (k % 32) == 0; }

extern "C" int culda_update_phi(int32_t k, int32_t num_words, const int64_t *d_word_ptr, const uint16_t *d_topics,
                                int32_t *d_phi, int32_t *d_nk, void *stream) {
    if (!valid_k(k) || num_words <= 0 || !d_word_ptr || !d_topics || !d_phi || !d_nk) {
        set_global_error("culda_update_phi: invalid argument");
        return CULDA_ERR_INVALID_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    int rc = cuda_status(cudaMemsetAsync(d_nk, 0, sizeof(int32_t) * (size_t)k, s));
    if (rc) return rc;
    // topics outside [0, K) are skipped; the caller validates its topic array
    return cuda_status(launch_update_phi(k, num_words, d_word_ptr, d_topics, d_phi, d_nk, nullptr, s));
}

extern "C" int culda_compute_phi_head(int32_t k, float beta, int32_t num_words, const int32_t *d_phi,
                                      const int32_t *d_nk, float *d_phi_head, void *stream) {
    if (!valid_k(k) || num_words <= 0 || !d_phi || !d_nk || !d_phi_head) {
        set_global_error("culda_compute_phi_head: invalid argument");
        return CULDA_ERR_INVALID_ARG;
    }
    return cuda_status(launch_phi_head(k, beta, num_words, d_phi, d_nk, d_phi_head, (cudaStream_t)stream));
}

extern "C" size_t culda_update_theta_workspace(int32_t k, int32_t num_docs) {
    (void)k;
    (void)num_docs;
    return 256;  // the device error word
}

extern "C" int culda_update_theta(int32_t k, int32_t num_docs, const int64_t *d_doc_ptr, const int32_t *d_doc_tok,
                                  const uint16_t *d_topics, const int32_t *d_doc_order, int32_t *d_theta_rows,
                                  uint32_t *d_theta, int32_t *d_nk, int64_t *d_stats, void *d_workspace,
                                  size_t workspace_bytes, void *stream) {
    if (!valid_k(k) || num_docs <= 0 || !d_doc_ptr || !d_doc_tok || !d_topics || !d_theta_rows || !d_theta ||
        !d_workspace || workspace_bytes < culda_update_theta_workspace(k, num_docs) || ((uintptr_t)d_theta & 15u)) {
        set_global_error("culda_update_theta: invalid argument");
        return CULDA_ERR_INVALID_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    int32_t *err = (int32_t *)d_workspace;
    int rc = cuda_status(cudaMemsetAsync(err, 0, sizeof(int32_t), s));
    if (!rc && d_nk) rc = cuda_status(cudaMemsetAsync(d_nk, 0, sizeof(int32_t) * (size_t)k, s));
    if (!rc && d_stats) rc = cuda_status(cudaMemsetAsync(d_stats, 0, 3 * sizeof(int64_t), s));
    if (rc) return rc;
    int dev = 0;
    cudaGetDevice(&dev);
    int bps = theta_blocks_per_sm(k);
    if (bps <= 0) bps = 1;
    const int grid = std::max(1, std::min(num_sms(dev) * bps, (num_docs + kThetaWarps - 1) / kThetaWarps));
    return cuda_status(launch_theta_rebuild(k, num_docs, d_doc_ptr, d_doc_tok, d_topics, d_doc_order,
                                            reinterpret_cast<int2 *>(d_theta_rows),
                                            reinterpret_cast<ThetaEntry *>(d_theta), d_nk, d_stats, err, grid, s));
}

extern "C" size_t culda_sample_workspace(int32_t k, int32_t num_items, int32_t num_hot) {
    // [counter, error, stats: 256][item_ll: 8*num_items rounded][hot rows: 4*K*num_hot]
    size_t a = 256;
    a += ((size_t)num_items * sizeof(double) + 255) / 256 * 256;
    a += (size_t)num_hot * (size_t)k * sizeof(int32_t);
    return a;
}

extern "C" int culda_sample(const culda_sample_args *a, void *d_workspace, size_t workspace_bytes, void *stream) {
    if (!a || !valid_k(a->k) || a->num_docs <= 0 || a->num_words <= 0 || a->num_tokens <= 0 || !a->word_ptr ||
        !a->doc_ids || !a->topics_in || !a->topics_out || a->topics_in == a->topics_out || !a->theta ||
        !a->theta_rows || !a->nk || !a->items || a->num_items <= 0 || !a->seg_start || a->num_segs <= 0 ||
        !a->loglik_sum || !d_workspace ||
        a->num_hot < 0 || (a->num_hot > 0 && (!a->hot_items || a->num_hot_items <= 0)) || a->theta_capacity <= 0 ||
        workspace_bytes < culda_sample_workspace(a->k, a->num_items, a->num_hot) ||
        (a->group_lanes != kFlatLanes && a->group_lanes != 1 && a->group_lanes != 2 && a->group_lanes != 4 &&
         a->group_lanes != 8 && a->group_lanes != 16 && a->group_lanes != 32) ||
        ((uintptr_t)a->theta & 31u)) {
        set_global_error("culda_sample: invalid argument");
        return CULDA_ERR_INVALID_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    char *ws = (char *)d_workspace;
    int32_t *counter = (int32_t *)ws;
    double *item_ll = (double *)(ws + 256);
    int32_t *hot_phi = (int32_t *)(ws + 256 + ((size_t)a->num_items * sizeof(double) + 255) / 256 * 256);
    int rc = cuda_status(cudaMemsetAsync(counter, 0, 256, s));
    if (rc) return rc;
    int32_t first_warp = a->num_items;  // items from here on are small
    // the sampler indexes shared memory with each entry's topic: reject a
    // theta array whose rows or topics are out of range before launching it
    {
        int32_t *out = counter + 40, got[3] = {0, 0, 0};
        rc = cuda_status(launch_check_sample(a->num_docs, a->k, reinterpret_cast<const int2 *>(a->theta_rows),
                                             reinterpret_cast<const ThetaEntry *>(a->theta), a->theta_capacity,
                                             a->items, a->num_items, out, s));
        if (!rc) rc = cuda_status(cudaMemcpyAsync(got, out, sizeof got, cudaMemcpyDeviceToHost, s));
        if (!rc) rc = cuda_status(cudaStreamSynchronize(s));
        if (rc) return rc;
        if (got[0]) {
            set_global_error("culda_sample: theta rows or topics out of range (flags 0x%x)", got[0]);
            return CULDA_ERR_INVALID_ARG;
        }
        if (got[1] + got[2] <= a->num_items) first_warp = a->num_items - got[1];
    }
    if (a->num_hot > 0) {
        rc = cuda_status(cudaMemsetAsync(hot_phi, 0, (size_t)a->num_hot * a->k * sizeof(int32_t), s));
        if (!rc)
            rc = cuda_status(launch_hot_rows(a->k, a->hot_items, a->num_hot_items, a->topics_in, hot_phi,
                                             a->error ? a->error : counter + 1, s));
        if (rc) return rc;
    }
    SampleParams p{};
    p.k = a->k;
    p.kmask = pow2_ceil(a->k) - 1;
    p.alpha = a->alpha;
    p.beta = a->beta;
    p.vbeta = a->beta * (float)a->num_words;
    p.num_docs = a->num_docs;
    p.num_items = a->num_items;
    p.num_hot = a->num_hot;
    p.num_tokens = a->num_tokens;
    p.theta_cap = a->theta_capacity;
    p.doc_ids = a->doc_ids;
    p.tok_index = nullptr;
    p.topics_in = a->topics_in;
    p.topics_out = a->topics_out;
    p.theta = reinterpret_cast<const ThetaEntry *>(a->theta);
    p.rows = reinterpret_cast<const int2 *>(a->theta_rows);
    p.nk = a->nk;
    p.items = a->items;
    p.seg_start = a->seg_start;
    p.num_segs = a->num_segs;
    p.hot_phi = hot_phi;
    p.item_counter = counter;
    p.first_warp = first_warp;
    p.warp_counter = counter + 48;
    p.item_ll = item_ll;
    p.seed = a->seed;
    p.iteration = a->iteration;
    p.iteration_ptr = nullptr;
    p.error = a->error ? a->error : counter + 1;
    int dev = 0;
    cudaGetDevice(&dev);
    const int blocks = a->group_lanes == kFlatLanes ? kFlatBlocks : kSampleBlocksDefault;
    int bps = sample_blocks_per_sm(a->k, a->group_lanes, blocks);
    if (bps <= 0) bps = 1;
    const int grid = std::max(1, std::min(a->num_items, num_sms(dev) * bps));
    rc = cuda_status(launch_sample(p, a->group_lanes, blocks, grid, s));
    if (rc) return rc;
    DevStats *st = (DevStats *)(counter + 8);
    rc = cuda_status(launch_finalize_ll(item_ll, a->num_items, st, counter + 3, s));
    if (rc) return rc;
    return cuda_status(cudaMemcpyAsync(a->loglik_sum, &st->ll_sum, sizeof(double), cudaMemcpyDeviceToDevice, s));
}

extern "C" int culda_loglik(const double *d_loglik_sum, double doc_term, int64_t num_tokens, double *loglik,
                            void *stream) {
    if (!d_loglik_sum || !loglik || num_tokens <= 0) return CULDA_ERR_INVALID_ARG;
    double sum = 0;
    cudaStream_t s = (cudaStream_t)stream;
    int rc = cuda_status(cudaMemcpyAsync(&sum, d_loglik_sum, sizeof(double), cudaMemcpyDeviceToHost, s));
    if (!rc) rc = cuda_status(cudaStreamSynchronize(s));
    if (rc) return rc;
    *loglik = (sum - doc_term) / (double)num_tokens;
    return CULDA_OK;
}
