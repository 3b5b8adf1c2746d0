// gemm.cu — BF16 GEMM on the sm_100a tensor cores for the document encoder:
// C[M x N] = A[M x K] * B[N x K]^T, both operands K-major (row-major with K
// contiguous), FP32 accumulation in tensor memory, with the encoder's
// epilogues fused: FP32 store, bias + GELU (pre-activation kept, activation
// stored in BF16 both as is and transposed), and the GELU backward (times
// GELU'(pre), BF16 out and transposed, bias-gradient column sums).
//
// One CTA of 128 threads per output tile of 128 x 128, 64 or 32 (and per K
// slice when the K range is split), two or more CTAs resident per SM so one
// tile's epilogue runs while the other's MMAs do.  Warp 0 lane 0 streams
// tiles of A and B, 64 deep, into a 3-stage shared-memory ring with TMA
// (128-byte swizzle); warp 1 lane 0 issues tcgen05.mma (M = 128, N = the tile's,
// K = 16 per instruction) into as many TMEM columns and frees each stage with
// tcgen05.commit; when the last MMA has landed all four warps read their 32
// TMEM lanes back with tcgen05.ld into a shared-memory copy of the tile, and
// the epilogue writes it out row by row (coalesced) and, for the transposed
// BF16 copy and the column sums, column by column.  Every mbarrier wait
// is bounded: a wait that gives up sets kErrTimeout in the error word and the
// tile is not stored.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <mutex>

#include "device_util.cuh"
#include "gemm.cuh"
#include "internal.h"
#include "kernels.cuh"
#include "umma.cuh"

namespace culda {

namespace {

constexpr int kBM = 128, kBK = 64, kStages = 3;
constexpr int kGemmThreads = 128;

// The output tile is kBM x BN, BN = 128, 64 or 32.
template <int BN>
struct Tile {
    static constexpr int kA = kBM * kBK * 2, kB = BN * kBK * 2;  // bytes of a stage's operands
    // the ring (operand A's stages, then B's), which later holds the accumulator copy, + alignment slack
    static constexpr size_t kRing = (size_t)kStages * (kA + kB);
    static constexpr size_t kSmem = kRing + 1024;
    static constexpr int kSP = BN + 1;  // row stride of the accumulator copy in floats
    static_assert((size_t)kBM * kSP * sizeof(float) <= kSmem - 1023, "the accumulator copy fits the ring and the slack");
};

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_grad(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * __expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// The accumulator tile is staged in shared memory (the operand ring is free
// once the last MMA has landed) as S[128][BN + 1] floats, row = output row; the
// odd stride keeps both a lane-per-row write and a lane-per-row column read
// free of bank conflicts.  Phase 1 (rows): BN / 4 lanes take a row, 4
// consecutive columns each, so every global row store or load is one run of 4
// BN (FP32) or 2 BN (BF16) bytes.  Phase 2 (columns, BF16 epilogues): each warp
// takes columns, each lane rows l, l+32, l+64, l+96 of the column, for the
// transposed copy and the bias-gradient column sums.
template <int EPI, int BN>
__device__ __forceinline__ void epilogue_rows(const GemmEpilogue &ep, float *S, int m0, int n0, int warp, int lane) {
    constexpr int kSP = Tile<BN>::kSP;
    constexpr int kLanes = BN / 4, kRows = 32 / kLanes;  // lanes per row, rows per warp at a time
    constexpr int kRowStep = kRows * kGemmThreads / 32, kAhead = 8;
    static_assert(kBM % (kRowStep * kAhead) == 0, "whole groups of rows");
    const int c = 4 * (lane % kLanes);
    for (int r0 = warp * kRows + lane / kLanes; r0 < kBM; r0 += kRowStep * kAhead) {
        // the pre-activations of the next 8 rows are loaded before any of them
        // is stored: the stores below could alias them for all the compiler knows
        float4 pv[kAhead];
        if constexpr (EPI == kEpiGeluBwd) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                pv[u] = *reinterpret_cast<const float4 *>(ep.pre + (size_t)(m0 + r0 + kRowStep * u) * ep.ldo + n0 + c);
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
        const int r = r0 + kRowStep * u;
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = S[r * kSP + c + i];
        const size_t o = (size_t)(m0 + r) * ep.ldo + n0 + c;
        if constexpr (EPI == kEpiF32) {
            const bool with_bias = ep.bias && blockIdx.z == 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = v[i] * ep.alpha + (with_bias ? ep.bias[n0 + c + i] : 0.f);
            float4 *d = reinterpret_cast<float4 *>(ep.out_f32 + o);
            if (ep.k_splits > 1)
                atomicAdd(d, make_float4(v[0], v[1], v[2], v[3]));
            else
                *d = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            if constexpr (EPI == kEpiBiasGelu) {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] += ep.bias[n0 + c + i];
                *reinterpret_cast<float4 *>(ep.out_f32 + o) = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = gelu(v[i]);
            } else {  // kEpiGeluBwd
                const float4 pre = pv[u];
                v[0] *= gelu_grad(pre.x);
                v[1] *= gelu_grad(pre.y);
                v[2] *= gelu_grad(pre.z);
                v[3] *= gelu_grad(pre.w);
            }
            uint2 q;
            __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&q);
            h[0] = __floats2bfloat162_rn(v[0], v[1]);
            h[1] = __floats2bfloat162_rn(v[2], v[3]);
            *reinterpret_cast<uint2 *>(ep.out_bf16 + o) = q;
            // the transposed copy and the column sums take the FP32 value: both
            // copies are the same single rounding of it to BF16
#pragma unroll
            for (int i = 0; i < 4; ++i) S[r * kSP + c + i] = v[i];
        }
        }
    }
}

template <int EPI, int BN>
__device__ __forceinline__ void epilogue_cols(const GemmEpilogue &ep, const float *S, int m0, int n0, int warp,
                                              int lane) {
    constexpr int kSP = Tile<BN>::kSP;
    for (int cc = warp; cc < BN; cc += kGemmThreads / 32) {
        float s = 0.f;
        __nv_bfloat16 *dst = ep.out_bf16_t + (size_t)(n0 + cc) * ep.ld_t + m0;
#pragma unroll
        for (int k = 0; k < kBM / 32; ++k) {
            const int r = lane + 32 * k;
            const float v = S[r * kSP + cc];
            dst[r] = __float2bfloat16_rn(v);
            s += v;
        }
        if (EPI == kEpiGeluBwd && ep.colsum) {
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) s += __shfl_xor_sync(0xffffffffu, s, w);
            if (lane == 0) atomicAdd(ep.colsum + n0 + cc, s);
        }
    }
}

template <int EPI, int BN>
__global__ void __launch_bounds__(kGemmThreads, 2)
    gemm_bf16_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, int K,
                     const GemmEpilogue ep, int32_t *error) {
    extern __shared__ uint8_t gsm_raw[];
    constexpr int kA = Tile<BN>::kA, kB = Tile<BN>::kB, kSP = Tile<BN>::kSP;
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    const uint32_t raw = umma::smem_u32(gsm_raw);
    uint8_t *base = gsm_raw + ((1024u - (raw & 1023u)) & 1023u);  // 1024-byte aligned for the swizzle
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * BN;
    // this CTA's K slice: k-blocks [kb0, kb0 + nk)
    const int nk_all = K / kBK;
    const int kb0 = (int)(((int64_t)nk_all * blockIdx.z) / gridDim.z);
    const int nk = (int)(((int64_t)nk_all * (blockIdx.z + 1)) / gridDim.z) - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        umma::mbar_init(&done, 1);
        umma::mbar_fence_init();
        abort_flag = 0;
        umma::tma_prefetch_map(&tma_a);
        umma::tma_prefetch_map(&tma_b);
    }
    if (warp == 0) {
        umma::tmem_alloc(&tmem_slot, BN);
        umma::tmem_relinquish();
    }
    umma::tc_fence_before();
    __syncthreads();
    umma::tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp == 0) {
        if (lane == 0) {  // TMA producer
            for (int kb = 0; kb < nk; ++kb) {
                const int s = kb % kStages;
                if (kb >= kStages && !umma::mbar_wait(&empty[s], (uint32_t)((kb / kStages) - 1) & 1u)) {
                    if (error) atomicOr(error, kErrTimeout);
                    atomicExch(&abort_flag, 1);
                    break;
                }
                umma::mbar_arrive_expect_tx(&full[s], (uint32_t)(kA + kB));
                umma::tma_load_2d(base + (size_t)s * kA, &tma_a, (kb0 + kb) * kBK, m0, &full[s]);
                umma::tma_load_2d(base + (size_t)kStages * kA + (size_t)s * kB, &tma_b, (kb0 + kb) * kBK, n0, &full[s]);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {  // MMA issuer
            constexpr uint32_t idesc = umma::idesc_bf16_f32(kBM, BN);
            for (int kb = 0; kb < nk; ++kb) {
                const int s = kb % kStages;
                if (!umma::mbar_wait(&full[s], (uint32_t)(kb / kStages) & 1u)) {
                    if (error) atomicOr(error, kErrTimeout);
                    atomicExch(&abort_flag, 1);
                    break;
                }
                umma::tc_fence_after();
                const uint64_t ad = umma::sdesc_k_sw128(base + (size_t)s * kA);
                const uint64_t bd = umma::sdesc_k_sw128(base + (size_t)kStages * kA + (size_t)s * kB);
#pragma unroll
                for (int j = 0; j < kBK / 16; ++j)  // 16 BF16 = 32 bytes = 2 descriptor units per step
                    umma::mma_bf16(tmem, ad + 2u * j, bd + 2u * j, idesc, (kb | j) != 0 ? 1u : 0u);
                umma::mma_commit(&empty[s]);
            }
            umma::mma_commit(&done);  // arrives once every MMA issued above has completed
        }
        __syncwarp();
    }

    // epilogue: warp w owns TMEM lanes 32w .. 32w+31 = output rows m0+32w ..;
    // the decision to store is the same in every thread (barrier, then the flag)
    bool ok = umma::mbar_wait(&done, 0u);
    umma::tc_fence_after();
    if (!__all_sync(0xffffffffu, ok) && lane == 0 && error) atomicOr(error, kErrTimeout);
    const bool go = __syncthreads_and(ok) && !*(volatile int *)&abort_flag;
    if (go) {
        float *S = reinterpret_cast<float *>(base);  // the operand ring, free now: every MMA has landed
        const int r = warp * 32 + lane;
        for (int c = 0; c < BN; c += 16) {
            float v[16];
            umma::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) S[r * kSP + c + i] = v[i];
        }
        __syncthreads();
        epilogue_rows<EPI, BN>(ep, S, m0, n0, warp, lane);
        if (EPI != kEpiF32) {
            __syncthreads();
            epilogue_cols<EPI, BN>(ep, S, m0, n0, warp, lane);
        }
    }
    umma::tc_fence_before();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, BN);
}

// ------------------------------------------------------------ tensor maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// A row-major BF16 matrix [rows x cols] with row stride ld elements, read in
// boxes of box_rows rows x 64 columns with 128-byte swizzle.
cudaError_t make_map(CUtensorMap *map, const void *ptr, int rows, int cols, int ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2u};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1u, 1u};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int EPI, int BN>
cudaError_t launch(const CUtensorMap &a, const CUtensorMap &b, int M, int N, int K, const GemmEpilogue &ep,
                   int32_t *error, cudaStream_t s) {
    const cudaError_t attr = allow_smem(reinterpret_cast<const void *>(&gemm_bf16_kernel<EPI, BN>), Tile<BN>::kSmem);
    if (attr != cudaSuccess) return attr;
    gemm_bf16_kernel<EPI, BN>
        <<<dim3(N / BN, M / kBM, ep.k_splits), kGemmThreads, Tile<BN>::kSmem, s>>>(a, b, K, ep, error);
    return cudaGetLastError();
}

template <int EPI>
cudaError_t launch_tile(int bn, const CUtensorMap &a, const CUtensorMap &b, int M, int N, int K,
                        const GemmEpilogue &ep, int32_t *error, cudaStream_t s) {
    return bn == 128  ? launch<EPI, 128>(a, b, M, N, K, ep, error, s)
           : bn == 64 ? launch<EPI, 64>(a, b, M, N, K, ep, error, s)
                      : launch<EPI, 32>(a, b, M, N, K, ep, error, s);
}

// Columns per tile: the narrowest tile that needs at most two CTAs per SM.  A
// launch's time is its CTAs' fixed costs and epilogues (the MMAs of a 128 x 128
// tile take 0.5 to 2 us), so a product of few tiles is cut finer until the chip
// is full: 1024 x 512 outputs with the GELU epilogues 13.2 us (32 CTAs of 128
// columns), 9.2 (64) and 7.2 us (128 CTAs of 32); 4096 x 512 14.4, 11.7 and
// 14.3 us; 4096 x 1024 13.9, 15.3 and 18.9 us.  Every width adds an output's
// products in the same order.
int tile_columns(int M, int N, int splits) {
    int dev = 0;
    cudaGetDevice(&dev);
    const int sms = num_sms(dev);
    const int64_t wide = (int64_t)(M / kBM) * (N / 128) * splits;
    return wide * 4 <= 2 * sms ? 32 : wide * 2 <= 2 * sms ? 64 : 128;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

const char *gemm_check(int M, int N, int K, const void *A, int lda, const void *B, int ldb, int epi,
                       const GemmEpilogue &ep) {
    if (M <= 0 || N <= 0 || K <= 0 || M % kBM || N % 128 || K % kBK) return "M, N must be multiples of 128, K of 64";
    if (!A || !B || !aligned16(A) || !aligned16(B)) return "A and B must be 16-byte aligned device pointers";
    if (lda < K || ldb < K || lda % 8 || ldb % 8) return "lda, ldb must be >= K and multiples of 8";
    if (ep.ldo < N || ep.ldo % 4) return "ldo must be >= N and a multiple of 4";
    if (ep.k_splits < 1 || ep.k_splits > K / kBK) return "k_splits must be in 1..K/64";
    if (ep.k_splits > 1 && epi != kEpiF32) return "split-K needs the F32 epilogue";
    switch (epi) {
        case kEpiF32:
            if (!ep.out_f32 || !aligned16(ep.out_f32)) return "F32 epilogue needs a 16-byte aligned out_f32";
            break;
        case kEpiBiasGelu:
            if (!ep.out_f32 || !ep.out_bf16 || !ep.out_bf16_t || !ep.bias) return "bias+GELU epilogue: null output";
            if (!aligned16(ep.out_f32) || !aligned16(ep.out_bf16) || ep.ldo % 8) return "bias+GELU epilogue: alignment";
            if (ep.ld_t < M) return "ld_t must be >= M";
            break;
        case kEpiGeluBwd:
            if (!ep.pre || !ep.out_bf16 || !ep.out_bf16_t) return "GELU backward epilogue: null operand";
            if (!aligned16(ep.pre) || !aligned16(ep.out_bf16) || ep.ldo % 8) return "GELU backward epilogue: alignment";
            if (ep.ld_t < M) return "ld_t must be >= M";
            break;
        default:
            return "unknown epilogue";
    }
    return nullptr;
}

cudaError_t gemm_bf16_nt(int M, int N, int K, const void *A, int lda, const void *B, int ldb, int epi,
                         const GemmEpilogue &ep, int32_t *error, cudaStream_t s) {
    if (gemm_check(M, N, K, A, lda, B, ldb, epi, ep)) return cudaErrorInvalidValue;
    const int bn = tile_columns(M, N, ep.k_splits);
    CUtensorMap ma, mb;
    cudaError_t e = make_map(&ma, A, M, K, lda, kBM);
    if (e != cudaSuccess) return e;
    e = make_map(&mb, B, N, K, ldb, bn);
    if (e != cudaSuccess) return e;
    switch (epi) {
        case kEpiF32: return launch_tile<kEpiF32>(bn, ma, mb, M, N, K, ep, error, s);
        case kEpiBiasGelu: return launch_tile<kEpiBiasGelu>(bn, ma, mb, M, N, K, ep, error, s);
        default: return launch_tile<kEpiGeluBwd>(bn, ma, mb, M, N, K, ep, error, s);
    }
}

}  // namespace culda
