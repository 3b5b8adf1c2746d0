// kernels.cuh — launch interface of the sm_100a kernels (host side).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/culda_b200.h"
#include "internal.h"

namespace culda {

// One theta CSR entry: the count (at most 65535, the longest doc) in the low
// 16 bits and 4 * topic (the byte offset of the topic's phihat in the
// sampler's shared memory; K <= 4096) in the high 16 bits.  Four bytes per
// entry, like the reference's two int16 arrays, but read with one load.
using ThetaEntry = uint32_t;

__host__ __device__ inline uint32_t theta_entry(uint32_t topic, uint32_t count) { return (topic << 18) | count; }

// Everything the sampler reads, passed by value.
struct SampleParams {
    int32_t k;
    int32_t kmask;               // next power of two >= K, minus one (bounds every topic index)
    float alpha;
    float beta;
    float vbeta;                 // (float)V * beta, the reference's denominator term (lda_phi_kernel.cu:26)
    int32_t num_docs;
    int32_t num_items;
    int32_t num_hot;             // rows in hot_phi
    int64_t num_tokens;          // N: items must lie inside [0, N)
    int64_t theta_cap;           // entries in the theta array
    const int32_t *doc_ids;      // [N]
    const int32_t *tok_index;    // [N] word-major index of each stored token (Philox counter), or null
    const float *uniforms;       // [N] the tokens' uniforms for this iteration, or null (computed inline)
    const uint16_t *topics_in;   // [N]
    uint16_t *topics_out;        // [N]
    const ThetaEntry *theta;     // CSR rows
    const int2 *rows;            // [D] {start, end}
    const int32_t *nk;           // [K]
    const float *inv;            // [K] 1 / (n_k + V beta), or null (formed where it is used)
    const culda_item *items;     // [num_items]
    const int32_t *seg_start;    // [num_segs] first token of every segment
    const int32_t *seg_doc;      // [num_segs] its doc, or null (read at its first token)
    int32_t num_segs;
    const int32_t *hot_phi;      // [num_hot * K]
    const int32_t *frozen_phi;   // [V * K] word-topic counts held fixed (fold-in), or null; then nk
                                 // holds the matching topic totals
    int32_t *item_counter;       // work queue head, zeroed before the launch
    int32_t first_warp;          // items [first_warp, num_items) are small: the flat walk takes them a warp
                                 // each (first_warp_item)
    int32_t *warp_counter;       // their queue head, zeroed before the launch; null: all items a CTA each
    double *item_ll;             // [num_items] sum of log(S+Q) per item
    uint64_t seed;
    uint32_t iteration;          // used when iteration_ptr is null
    const uint32_t *iteration_ptr;
    int32_t *error;
    unsigned long long *clock;   // {first start, last end} of the launch's CTAs (global timer), or null
};

struct DevStats {
    double ll_sum;        // sum over tokens of log(S_t + Q_t)
    int64_t row_entries;  // sum_d L_d * rowlen_d after the theta rebuild   (stats slot 0)
    int64_t nnz;          // theta non-zeros after the rebuild              (stats slot 1)
    int64_t token_nnz;    // sum_d L_d * nnz_d after the rebuild            (stats slot 2)
    int32_t error;
    uint32_t iteration;   // Philox iteration the sampler used
    unsigned long long mh_accepted, mh_proposed;  // Metropolis-Hastings iterations
    // global timer (ns) at the first start and the last end of a CTA of the
    // sampling kernel and of the rebuild
    unsigned long long sample_t0, sample_t1, rebuild_t0, rebuild_t1;
    double joint;         // joint log-likelihood sum (written to the host copy only)
};

// What an iteration clears and forms before it samples, in one kernel.
struct PrologueParams {
    int64_t n;                       // tokens whose uniforms are formed (0: none)
    uint64_t seed;
    const uint32_t *iteration_dev;   // Philox iteration: *iteration_dev, or `iteration` when null
    uint32_t iteration;
    const int32_t *tok_index;
    float *u;
    int32_t *counter;                // the sampler's queue head, cleared
    int32_t *warp_counter;           // the queue head of the items a warp takes, cleared
    int32_t *theta_queue;            // the rebuild's queue head, cleared
    int32_t *done;                   // CTAs of the rebuild finished, cleared
    int32_t *hot_phi;                // cleared
    int64_t hot_n;
    int32_t *nk_next;                // topic totals the rebuild adds into, cleared (or null)
    int32_t k;
    const int32_t *nk;               // topic totals the iteration samples against
    float vbeta;
    float *inv;                      // [K] receives 1 / (n_k + V beta)
    DevStats *stats;                 // counts cleared, clocks set to their neutral values
};
cudaError_t launch_prologue(const PrologueParams &p, cudaStream_t s);

// What the rebuild's last CTA does at the end of an iteration: adds up the
// per-item log terms (each CTA has summed its share into partials) and
// writes the iteration's statistics to slot *iteration_dev % kStatsRing of
// the pinned ring.  stats null: nothing.
constexpr int kStatsRing = 4;
struct IterationEnd {
    DevStats *stats = nullptr;
    const double *item_ll = nullptr;
    int32_t num_items = 0;
    double *partials = nullptr;  // one per CTA
    int32_t *done = nullptr;
    uint32_t *iteration_dev = nullptr;
    DevStats *ring = nullptr;
};

inline int pow2_ceil(int k) {
    int p = 1;
    while (p < k) p <<= 1;
    return p;
}

// Sampler variants: lanes per token G and the register budget, given as the
// resident CTAs per SM the kernel is compiled for (kSampleBlocksDefault for
// every G; kSampleBlocksHigh for G = 4, 8, 16).  G = kFlatLanes is the
// warp-flattened walk, built for kSampleBlocksDefault and kFlatBlocks (56
// registers: its two-buffer walk spills at 48).
constexpr int kSampleBlocksDefault = 8;
constexpr int kSampleBlocksHigh = 10;
constexpr int kFlatBlocks = 9;
constexpr int kFlatLanes = -1;
// Items of at most this many tokens are sampled a warp each (sampler.cu says why here).
constexpr int kWarpItemTokens = 32;
size_t sample_smem_bytes(int k, int group_lanes);
bool sample_variant_exists(int group_lanes, int blocks_per_sm);
int sample_blocks_per_sm(int k, int group_lanes, int blocks_per_sm);
// The first item of a work list (largest first) that the flat walk gives to a warp.
int32_t first_warp_item(const culda_item *items, int32_t n);
cudaError_t launch_sample(const SampleParams &p, int group_lanes, int blocks_per_sm, int grid, cudaStream_t s);

size_t theta_smem_bytes(int k);
int theta_blocks_per_sm(int k);
// The first num_long docs of doc_order (which must then be given) are taken
// a whole CTA each from the queue counter long_queue (cleared by the launch,
// or by the prologue when `end` is given); the rest one warp each.
cudaError_t launch_theta_rebuild(int k, int num_docs, const int64_t *doc_ptr, const int32_t *doc_tok,
                                 const uint16_t *topics, const int32_t *doc_order, int2 *rows, ThetaEntry *theta,
                                 int32_t *nk, int64_t *stats, int32_t *error, int grid, cudaStream_t s,
                                 int num_long = 0, int32_t *long_queue = nullptr,
                                 const IterationEnd &end = IterationEnd{});

cudaError_t launch_hot_rows(int k, const culda_item *hot_items, int num_hot_items, const uint16_t *topics,
                            int32_t *hot_phi, int32_t *error, cudaStream_t s);

// Sum of item_ll (overwritten) into st->ll_sum; `done` must be zero.
cudaError_t launch_finalize_ll(double *item_ll, int num_items, DevStats *st, int32_t *done, cudaStream_t s);

// Flags theta rows outside the array or misaligned, and entries whose topic
// is not below K (the kernel-level sampler checks a caller's theta with it),
// and looks the work list over: out[0] the flags, out[1] num_items minus the
// first item of at most kWarpItemTokens tokens, out[2] one past the last larger
// one (all zero before; the list is in order when out[1] + out[2] <= num_items).
cudaError_t launch_check_sample(int num_docs, int k, const int2 *rows, const ThetaEntry *theta, int64_t cap,
                                const culda_item *items, int num_items, int32_t *out, cudaStream_t s);

cudaError_t launch_init_topics(int64_t n, int k, uint64_t seed, const int32_t *tok_index, uint16_t *z,
                               cudaStream_t s);

cudaError_t launch_update_phi(int k, int num_words, const int64_t *word_ptr, const uint16_t *topics, int32_t *phi,
                              int32_t *nk, int32_t *error, cudaStream_t s);

cudaError_t launch_phi_head(int k, float beta, int num_words, const int32_t *phi, const int32_t *nk, float *out,
                            cudaStream_t s);

cudaError_t launch_doc_check(int64_t n, int num_docs, const int32_t *doc_ids, int32_t *doc_count, int32_t *error,
                             cudaStream_t s);

// Joint log-likelihood (see kernels.cu): items are the sampler's work list,
// largest first, with the hot rows of the current topics.
constexpr int kJointCounters = 513;
struct JointParams {
    int32_t k, num_words, num_docs;
    int32_t num_items, num_long;  // num_long: long_items() of the list
    double alpha, beta, lg_alpha, lg_beta;  // and their lgamma
    const culda_item *items;
    const int32_t *hot_phi;
    const uint16_t *topics;
    const ThetaEntry *theta;
    int64_t theta_cap;  // entries; those past the end of a row are zero
    const int64_t *doc_ptr;
    const int32_t *nk;
    double *partials;  // one per CTA
    uint32_t *counts;  // [kJointCounters], cleared by the launch
    double *result;    // receives the sum; may be mapped host memory
    int32_t *error;
};
cudaError_t launch_loglik_joint(const JointParams &p, int max_partials, cudaStream_t s);
// The items of a work list (largest first) that a whole CTA counts.
int64_t long_items(const culda_item *items, int64_t n);

// Internal token order: within each word, tokens sorted by their doc's length
// (longest first, doc id breaking ties).  keys[t] = (word << 16) | (65535 - L).
cudaError_t launch_order_keys(int num_words, int64_t num_tokens, const int64_t *word_ptr, const int32_t *doc_ids,
                              const int64_t *doc_ptr, uint64_t *keys, cudaStream_t s);
// The same order with 32-bit keys (num_words <= 2^24): keys[t] = (word << 8) |
// (255 - length class), 16 classes per doubling of L.
cudaError_t launch_order_keys32(int num_words, int64_t num_tokens, const int64_t *word_ptr, const int32_t *doc_ids,
                                const int64_t *doc_ptr, uint32_t *keys, cudaStream_t s);
template <class T>
cudaError_t launch_gather(int64_t n, const int32_t *index, const T *src, T *dst, cudaStream_t s);
template <class T>
cudaError_t launch_scatter(int64_t n, const int32_t *index, const T *src, T *dst, cudaStream_t s);
cudaError_t launch_iota(int64_t n, int32_t *v, cudaStream_t s);
cudaError_t launch_check_topics(int64_t n, int k, const uint16_t *z, int32_t *error, cudaStream_t s);

int num_sms(int device);

// Copies between the host and the current device on stream s, through pinned
// staging when the host memory is pageable and the copy is large (staging.cu).
// copy_to_host returns when dst holds the bytes; copy_to_device when src has
// been read (a pinned src: when the copy is queued, as cudaMemcpyAsync).
cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t s);
cudaError_t copy_to_device(void *dst, const void *src, size_t bytes, cudaStream_t s);
// Frees the device's idle staging memory.
void release_staging(int device);

}  // namespace culda
