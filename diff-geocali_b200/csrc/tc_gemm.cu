// tc_gemm.cu -- BF16 x BF16 -> FP32 GEMM on the sm_100 5th-generation tensor
// cores (tcgen05.mma, accumulators in tensor memory), for the convolution
// layers of the warm-start network.  No counterpart in the reference.
//
//   C[m, n] (+)= sum_k A[m, k] * B[n, k]  (+ bias[n], optional ReLU)
//
// A (M x K) and B (N x K) are row-major bf16 ("K-major"); C is fp32 or bf16.  The
// TMA kernel also takes both operands as stored [K][M] and [K][N] ("MN-major"):
// a weight gradient reduces over the rows of activations that lie that way.
//
// Structure of a CTA (128 threads, one 128 x BN output tile):
//   * warp 0 allocates BN tensor-memory columns (a 128-lane x BN fp32
//     accumulator) and frees them at the end;
//   * all threads stage 128 x 64 tiles of A and BN x 64 tiles of B into shared
//     memory with cp.async, four stages deep, in the 128-byte-swizzled K-major
//     layout: row r of a tile is 128 contiguous bytes (its 64 K elements) at
//     r*128, its 16-byte chunk j stored at chunk j ^ (r % 8); eight
//     consecutive threads copy one row, so the global reads are 128-byte
//     coalesced and the shared-memory writes conflict-free (SBO = 1024 B
//     between 8-row groups; the K = 16 step of an MMA advances the start
//     address by 32 B inside the swizzle atom);
//   * one elected thread issues four tcgen05.mma (M=128, N=BN, K=16) per stage
//     and commits them to the stage's mbarrier, which releases the stage for
//     the next prefetch and, after the last stage, signals the epilogue;
//   * the four warps read their 32 accumulator lanes with tcgen05.ld, apply
//     bias / ReLU / accumulate and store.
// Every mbarrier wait is bounded; a timeout sets the error word, skips the
// epilogue and still frees the tensor memory.
#include <cuda.h>

#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "tc_gemm.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace dgc {

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return static_cast<EncodeTiledFn>(nullptr);
        return reinterpret_cast<EncodeTiledFn>(ptr);
    }();
    return fn;
}

namespace {

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kStages = 4;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
                 "r"(src_bytes)
                 : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

// K-major operand with 128-byte swizzle: SBO = 1024 B between 8-row groups (LBO is
// unused by swizzled K-major).
__device__ __forceinline__ uint64_t kmajor_sw128_desc(uint32_t saddr) {
    return smem_desc(saddr, 16u, 1024u, 2u);
}

// The same for MN-major operands staged as boxes of 64 (M or N) x kBK (K): a K row
// is 128 contiguous bytes; SBO = 1024 B between groups of 8 K rows, LBO = one
// box (kBK * 128 B) between groups of 64 M or N.
__device__ __forceinline__ uint64_t mnmajor_sw128_desc(uint32_t saddr) {
    return smem_desc(saddr, kBK * 128u, 1024u, 2u);
}

// Stage one K-slice: 'rows' x 64 bf16 of a K-major matrix into the 128-byte
// swizzled layout (16-byte chunk j of row r at r*128 + ((j ^ (r & 7)) * 16)).
// Out-of-range rows or K chunks are zero-filled.
template <int ROWS>
__device__ __forceinline__ void stage_tile(uint32_t sbase, const __nv_bfloat16* g, int ld,
                                           int row0, int nrows, int k0, int K) {
    constexpr int kChunks = ROWS * (kBK / 8);
#pragma unroll 4
    for (int c = threadIdx.x; c < kChunks; c += 128) {
        const int r = c >> 3, j = c & 7;
        const int row = row0 + r, k = k0 + j * 8;
        const bool ok = row < nrows && k < K;
        const __nv_bfloat16* src = ok ? g + (long long)row * ld + k : g;
        cp_async16(sbase + static_cast<uint32_t>(r * 128 + ((j ^ (r & 7)) << 4)), src, ok ? 16 : 0);
    }
}

// Epilogue: the four warps read their 32 accumulator lanes (rows) with
// tcgen05.ld, 16 columns at a time, and apply alpha / bias / ReLU /
// accumulate (or the split-K atomic sum) on the way to C.  A lane's 16 columns
// go out as 32-byte stores (whole sectors) where C's alignment allows it; one
// element at a time every lane touched another row's sector 16 times over
// (8192^3: 1087 -> 1428 TFLOP/s; the data-gradient products of the network at 180
// views, 1.1 GB of fp32 output: 1.0 -> 0.36 ms with the short-K tiles below).
template <int BN>
__device__ __forceinline__ void gemm_epilogue(const GemmArgs& p, uint32_t tmem, int m0, int n0,
                                              bool has_k, bool split) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = m0 + warp * 32 + lane;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const bool wide = (reinterpret_cast<uintptr_t>(p.C) & 31u) == 0 &&
                      p.ldc % (p.c_bf16 ? 16 : 8) == 0;
#pragma unroll 1
    for (int c0 = 0; c0 < BN && n0 + c0 < p.N; c0 += 16) {
        float v[16];
        tmem_load16(lane_addr + c0, v);
        if (row >= p.M) continue;
        const int col0 = n0 + c0;
        const bool add_bias = p.bias && (!split || blockIdx.z == 0);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            float x = has_k ? v[j] : 0.0f;
            x *= p.alpha;
            if (add_bias && col0 + j < p.N) x += p.bias[col0 + j];
            if (!split && p.relu) x = fmaxf(x, 0.0f);
            v[j] = x;
        }
        const long long off = (long long)row * p.ldc + col0;
        if (wide && col0 + 16 <= p.N) {
            if (p.c_bf16) {
                uint32_t h[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                    h[j] = *reinterpret_cast<const uint32_t*>(&b);
                }
                store32(static_cast<__nv_bfloat16*>(p.C) + off, h);
                continue;
            }
            float* C = static_cast<float*>(p.C) + off;
#pragma unroll
            for (int j = 0; j < 16; j += 8) {
                if (split) {  // partial sum of a K range; bias from split 0
                    red_add4_global(C + j, v[j], v[j + 1], v[j + 2], v[j + 3]);
                    red_add4_global(C + j + 4, v[j + 4], v[j + 5], v[j + 6], v[j + 7]);
                    continue;
                }
                uint32_t x[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    x[k] = __float_as_uint(p.accumulate ? C[j + k] + v[j + k] : v[j + k]);
                store32(C + j, x);
            }
            continue;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (col0 + j >= p.N) break;
            if (p.c_bf16) {
                static_cast<__nv_bfloat16*>(p.C)[off + j] = __float2bfloat16(v[j]);
                continue;
            }
            float* C = static_cast<float*>(p.C) + off + j;
            if (split) atomicAdd(C, v[j]);
            else *C = p.accumulate ? *C + v[j] : v[j];
        }
    }
}

template <int BN>
__global__ void __launch_bounds__(128) tc_gemm_kernel(GemmArgs p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[kStages + 1];
    __shared__ uint32_t tmem_slot;
    constexpr int kABytes = kBM * kBK * 2;
    constexpr int kBBytes = BN * kBK * 2;
    constexpr int kStageBytes = kABytes + kBBytes;
    constexpr uint32_t kIdesc = idesc_bf16(kBM, BN);

    const int warp = threadIdx.x >> 5;
    const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * BN;
    // 1024-byte aligned base (the swizzle atoms); the launch adds 1 KiB slack
    const uint32_t sbase = (smem_u32(smem) + 1023u) & ~1023u;
    // split-K: this CTA reduces K tiles [kt0, kt0 + nk)
    const int nk_total = (p.K + kBK - 1) / kBK;
    const bool split = p.k_tiles_per_split > 0;
    const int kt0 = split ? blockIdx.z * p.k_tiles_per_split : 0;
    const int nk = split ? max(0, min(p.k_tiles_per_split, nk_total - kt0)) : nk_total;
    const int k_base = kt0 * kBK;

    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), BN);
    if (threadIdx.x == 0) {
        for (int s = 0; s <= kStages; ++s) mbar_init(smem_u32(&bars[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    // prologue: stages 0 .. kStages-2
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if (s < nk) {
            const uint32_t sa = sbase + s * kStageBytes;
            stage_tile<kBM>(sa, p.A, p.lda, m0, p.M, k_base + s * kBK, p.K);
            stage_tile<BN>(sa + kABytes, p.B, p.ldb, n0, p.N, k_base + s * kBK, p.K);
        }
        cp_async_commit();
    }

    bool ok = true;
    for (int kt = 0; kt < nk; ++kt) {
        const int s = kt % kStages;
        cp_async_wait<kStages - 2>();
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        // block-uniform: a timed-out wait anywhere ends the loop for all threads
        ok = __syncthreads_and(ok);
        if (!ok) break;
        if (threadIdx.x == 0) {
            tc_fence_after();
            const uint32_t sa = sbase + s * kStageBytes;
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk) {
                // K = 16 per instruction: 32 bytes further into every 128-byte row
                const uint64_t ad = kmajor_sw128_desc(sa + kk * 32);
                const uint64_t bd = kmajor_sw128_desc(sa + kABytes + kk * 32);
                umma_bf16(tmem, ad, bd, kIdesc, (kt > 0 || kk > 0) ? 1u : 0u);
            }
            umma_commit(smem_u32(&bars[s]));
        }
        // prefetch tile kt + kStages - 1 into the stage the previous MMAs used
        const int kn = kt + kStages - 1;
        if (kn < nk) {
            const int sn = kn % kStages;
            if (kt >= 1) ok = mbar_wait(smem_u32(&bars[sn]), ((kt - 1) / kStages) & 1);
            if (ok) {
                const uint32_t sa = sbase + sn * kStageBytes;
                stage_tile<kBM>(sa, p.A, p.lda, m0, p.M, k_base + kn * kBK, p.K);
                stage_tile<BN>(sa + kABytes, p.B, p.ldb, n0, p.N, k_base + kn * kBK, p.K);
            }
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    ok = __syncthreads_and(ok);
    // the last commit completes after every MMA of the tile
    if (ok && nk > 0) ok = mbar_wait(smem_u32(&bars[(nk - 1) % kStages]), ((nk - 1) / kStages) & 1);
    ok = __syncthreads_and(ok);
    if (!ok && threadIdx.x == 0) atomicExch(p.error, 1);
    tc_fence_after();

    if (ok) gemm_epilogue<BN>(p, tmem, m0, n0, nk > 0, split);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_free(tmem, BN);
    }
}

// ---------------------------------------------------------------------------
// TMA + warp-specialised variant (the default).  Warp 0's lane 0 is the
// producer: per K tile it waits for the stage to be free (the MMAs that read
// it committed to empty[s]), posts the stage's byte count on full[s] and
// issues two cp.async.bulk.tensor loads (A 128 x 64, B BN x 64) that the
// tensor-map hardware writes in the 128-byte-swizzled layout, zero-filling
// rows and K beyond the matrix.  Warp 1's lane 0 issues the MMAs when full[s]
// completes and commits them to empty[s].  The last commit goes to `done`;
// then all four warps run the epilogue.  Every wait is bounded: on a timeout
// the error word is set, loads already issued are waited for (bounded) and
// the tensor memory is freed.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// MSUB 128-row sub-tiles of A per CTA (1 or 2): with 2, a CTA computes a
// 256 x BN tile as two M = 128 accumulators that share every staged B tile,
// which cuts the operand bytes moved per FLOP by a third at BN = 256.
template <int BN, int MSUB = 1>
struct TmaStages {
    static constexpr int kStageBytes = MSUB * kBM * kBK * 2 + BN * kBK * 2;
    // the narrow tiles' products are bound by memory: half the shared memory each,
    // so that two CTAs per SM overlap their epilogues and loads
    static constexpr int kBudget = BN <= 128 ? 98304 : 196608;
    static constexpr int value = (kBudget / kStageBytes) < 8 ? (kBudget / kStageBytes) : 8;
};

// MN: MN-major operands, staged as boxes of 64 M or N x 64 K.
template <int BN, int MSUB, bool MN>
__global__ void __launch_bounds__(128) tc_gemm_tma_kernel(const __grid_constant__ CUtensorMap tmA,
                                                          const __grid_constant__ CUtensorMap tmB,
                                                          GemmArgs p) {
    constexpr int S = TmaStages<BN, MSUB>::value;
    constexpr int kABytes = MSUB * kBM * kBK * 2;
    constexpr int kStageBytes = TmaStages<BN, MSUB>::kStageBytes;
    constexpr int kCols = MSUB * BN;  // tensor-memory columns of the accumulators
    constexpr uint32_t kIdesc = idesc_bf16(kBM, BN, MN, MN);
    constexpr uint32_t kBox = 64 * kBK * 2;  // bytes of an MN-major box
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[S];
    __shared__ __align__(8) uint64_t empty[S];
    __shared__ __align__(8) uint64_t done;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_err, s_consumed;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * kBM * MSUB, n0 = blockIdx.x * BN;
    const uint32_t sbase = (smem_u32(smem) + 1023u) & ~1023u;
    const int nk_total = (p.K + kBK - 1) / kBK;
    const bool split = p.k_tiles_per_split > 0;
    const int kt0 = split ? blockIdx.z * p.k_tiles_per_split : 0;
    const int nk = split ? max(0, min(p.k_tiles_per_split, nk_total - kt0)) : nk_total;

    if (warp == 0) tmem_alloc(smem_u32(&tmem_slot), kCols);
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(smem_u32(&full[i]), 1);
            mbar_init(smem_u32(&empty[i]), 1);
        }
        mbar_init(smem_u32(&done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        s_err = 0;
        s_consumed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    volatile int* err = &s_err;

    int issued = 0;
    if (warp == 0 && lane == 0) {
        for (int kt = 0; kt < nk; ++kt) {
            const int s = kt % S;
            if (kt >= S && !mbar_wait(smem_u32(&empty[s]), ((kt / S) - 1) & 1)) {
                *err = 1;
                break;
            }
            if (*err) break;
            const uint32_t sa = sbase + s * kStageBytes;
            const int kx = (kt0 + kt) * kBK;
            mbar_expect_tx(smem_u32(&full[s]), kStageBytes);
            if (MN) {
#pragma unroll
                for (int b = 0; b < MSUB * kBM / 64; ++b)
                    tma_load_2d(sa + b * kBox, &tmA, m0 + b * 64, kx, smem_u32(&full[s]));
#pragma unroll
                for (int b = 0; b < BN / 64; ++b)
                    tma_load_2d(sa + kABytes + b * kBox, &tmB, n0 + b * 64, kx, smem_u32(&full[s]));
            } else {
                tma_load_2d(sa, &tmA, kx, m0, smem_u32(&full[s]));
                tma_load_2d(sa + kABytes, &tmB, kx, n0, smem_u32(&full[s]));
            }
            ++issued;
        }
    } else if (warp == 1 && lane == 0) {
        int kt = 0;
        for (; kt < nk; ++kt) {
            const int s = kt % S;
            if (!mbar_wait(smem_u32(&full[s]), (kt / S) & 1)) {
                *err = 1;
                break;
            }
            tc_fence_after();
            const uint32_t sa = sbase + s * kStageBytes;
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk) {
                // K = 16 per instruction: 32 bytes further into every row (K-major)
                // or two groups of 8 K rows (MN-major)
                const uint64_t bd = MN ? mnmajor_sw128_desc(sa + kABytes + kk * 2048)
                                       : kmajor_sw128_desc(sa + kABytes + kk * 32);
#pragma unroll
                for (int m = 0; m < MSUB; ++m) {
                    // sub-tile m: rows 128m.. of the staged A (128 B per row), or its boxes
                    const uint64_t ad = MN ? mnmajor_sw128_desc(sa + m * 2 * kBox + kk * 2048)
                                           : kmajor_sw128_desc(sa + m * kBM * 128 + kk * 32);
                    umma_bf16(tmem + m * BN, ad, bd, kIdesc, (kt > 0 || kk > 0) ? 1u : 0u);
                }
            }
            umma_commit(smem_u32(&empty[s]));
        }
        s_consumed = kt;
        umma_commit(smem_u32(&done));  // arrives once every MMA issued above has completed
    }
    __syncthreads();
    bool ok = (*err == 0);
    // all MMAs (and with them every read of the staged tiles) are complete
    if (nk > 0 && !mbar_wait(smem_u32(&done), 0)) ok = false;
    ok = __syncthreads_and(ok);
    if (warp == 0 && lane == 0) {
        // loads issued but never consumed (only after a timeout) must land
        // before the CTA's shared memory is released
        for (int kt = s_consumed; kt < issued; ++kt) mbar_wait(smem_u32(&full[kt % S]), (kt / S) & 1);
    }
    __syncwarp();
    if (!ok && threadIdx.x == 0) atomicExch(p.error, 1);
    tc_fence_after();
    if (ok) {
#pragma unroll
        for (int m = 0; m < MSUB; ++m)
            gemm_epilogue<BN>(p, tmem + m * BN, m0 + m * kBM, n0, nk > 0, split);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_free(tmem, kCols);
    }
}

// 2-D bf16 map of a row-major [rows][ld] matrix with cols valid columns (K, or M
// or N of an MN-major operand): boxes of 64 columns (128 bytes) x box_rows rows,
// 128-byte swizzle, zero fill outside.
bool make_kmajor_map(CUtensorMap* map, const void* base, int rows, int cols, int ld, int box_rows) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int MSUB, bool MN>
int launch_gemm_tma(const GemmArgs& p, cudaStream_t s, bool* used) {
    *used = false;
    CUtensorMap ta, tb;
    if (MN ? !make_kmajor_map(&ta, p.A, p.K, p.M, p.lda, kBK) ||
                 !make_kmajor_map(&tb, p.B, p.K, p.N, p.ldb, kBK)
           : !make_kmajor_map(&ta, p.A, p.M, p.K, p.lda, kBM * MSUB) ||
                 !make_kmajor_map(&tb, p.B, p.N, p.K, p.ldb, BN))
        return DGC_OK;
    constexpr int kMost = TmaStages<BN, MSUB>::value * TmaStages<BN, MSUB>::kStageBytes + 1024;
    static std::atomic<unsigned long long> configured{0};
    const int rc = once_per_device(configured, []() -> int {
        DGC_CUDA(cudaFuncSetAttribute(tc_gemm_tma_kernel<BN, MSUB, MN>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
        return DGC_OK;
    });
    if (rc != DGC_OK) return rc;
    const int ktiles = ceil_div(p.K, kBK);
    const int splits = p.k_tiles_per_split > 0 ? ceil_div(ktiles, p.k_tiles_per_split) : 1;
    // only the stages that the reduction fills: a short one leaves room for
    // several CTAs per SM, whose epilogues then overlap
    const int stages = std::min(TmaStages<BN, MSUB>::value,
                                p.k_tiles_per_split > 0 ? p.k_tiles_per_split : ktiles);
    const int smem = stages * TmaStages<BN, MSUB>::kStageBytes + 1024;
    const dim3 grid(ceil_div(p.N, BN), ceil_div(p.M, kBM * MSUB), splits);
    DGC_TRACE("tc_gemm_tma_kernel", s);
    tc_gemm_tma_kernel<BN, MSUB, MN><<<grid, 128, smem, s>>>(ta, tb, p);
    DGC_LAUNCH_CHECK("tc_gemm_tma_kernel");
    *used = true;
    return DGC_OK;
}

template <int BN>
int launch_gemm(const GemmArgs& p, cudaStream_t s) {
    const int smem = kStages * (kBM * kBK * 2 + BN * kBK * 2) + 1024;
    static std::atomic<unsigned long long> configured{0};
    const int rc = once_per_device(configured, [smem]() -> int {
        DGC_CUDA(cudaFuncSetAttribute(tc_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      smem));
        return DGC_OK;
    });
    if (rc != DGC_OK) return rc;
    const int splits = p.k_tiles_per_split > 0
                           ? ceil_div(ceil_div(p.K, kBK), p.k_tiles_per_split) : 1;
    const dim3 grid(ceil_div(p.N, BN), ceil_div(p.M, kBM), splits);
    DGC_TRACE("tc_gemm_kernel", s);
    tc_gemm_kernel<BN><<<grid, 128, smem, s>>>(p);
    DGC_LAUNCH_CHECK("tc_gemm_kernel");
    return DGC_OK;
}

}  // namespace

namespace {
template <bool MN>
int launch_gemm_tma_bn(const GemmArgs& p, int bn, bool two, cudaStream_t s, bool* used) {
    return bn == 64    ? launch_gemm_tma<64, 1, MN>(p, s, used)
           : two       ? launch_gemm_tma<256, 2, MN>(p, s, used)
           : bn == 256 ? launch_gemm_tma<256, 1, MN>(p, s, used)
                       : launch_gemm_tma<128, 1, MN>(p, s, used);
}
}  // namespace

int tc_gemm(const GemmArgs& p, cudaStream_t s) {
    const int splits = p.k_tiles_per_split > 0 ? ceil_div(ceil_div(p.K, kBK), p.k_tiles_per_split) : 1;
    // Short reductions (the data gradients' K = 32..256) are bound by their
    // output: 128-column tiles leave tensor memory for four CTAs per SM.
    const bool short_k = p.K <= 4 * kBK;
    // 256-column tiles halve the B traffic per FLOP; used when they still
    // give every SM a tile
    const int bn = p.N <= 64 ? 64
                   : (!short_k && p.N > 128 && (long long)ceil_div(p.M, kBM) * ceil_div(p.N, 256) * splits >= 148)
                       ? 256
                       : 128;
    // DGC_GEMM=cpasync selects the cp.async pipeline (also the fallback when
    // the driver cannot encode tensor maps)
    const char* e = std::getenv("DGC_GEMM");
    if (!(e && std::strcmp(e, "cpasync") == 0)) {
        // 256 x 256 tiles (two accumulators) where they still give every SM a tile
        const bool two = bn == 256 &&
                         (long long)ceil_div(p.M, 2 * kBM) * ceil_div(p.N, 256) * splits >= 148;
        bool used = false;
        const int rc = p.mn_major ? launch_gemm_tma_bn<true>(p, bn, two, s, &used)
                                  : launch_gemm_tma_bn<false>(p, bn, two, s, &used);
        if (rc != DGC_OK || used) return rc;
    }
    if (p.mn_major) {
        set_error("MN-major operands need the TMA pipeline");
        return DGC_ERR_UNSUPPORTED;
    }
    if (bn == 64) return launch_gemm<64>(p, s);
    if (bn == 256) return launch_gemm<256>(p, s);
    return launch_gemm<128>(p, s);
}

}  // namespace dgc
