// fdk_tc.cu -- the FDK ramp filter's Toeplitz product on the 5th-generation tensor
// cores, with FP32 results.
//
// fdk.cu evaluates y[u,v] = sum_k h[|u-k|] w[k,v] per view as an FP32 SIMT product,
// which its shared-memory reads bound at 41 of 74 TFLOP/s.  Here both factors are
// split exactly into three bf16 parts (8 + 8 + 8 bits of the FP32 mantissa) and
// the six products down to 2^-16 of the leading one run as tcgen05.mma, whose
// bf16 products are exact.  What would lose precision is the accumulator, which
// the tensor core rounds toward zero: the leading product (hi x hi) therefore
// accumulates over 32 taps at a time only and is added into FP32 registers with
// rounding to nearest; the other five, at most 2^-8 of it, share one accumulator
// over the whole row.  (64 taps at a time: 4 % faster, but the largest errors were
// above the SIMT product's.)  Relative error against 64 bits, this / the SIMT product,
// mean of six ellipsoid phantoms: U = 96 2.6e-7 / 3.7e-7, 187 5.6e-7 / 7.0e-7, 384
// 1.2e-6 / 1.4e-6, 768 1.9e-6 / 2.3e-6, 1536 2.5e-6 / 3.5e-6; white noise at 768
// 1.5e-7 / 5.2e-7.
//
// Measured (the whole call, before -> after): 720 x 768 x 768 15.83 -> 3.79 ms, of which
// the product 2.61 ms = 1.50 PFLOP/s of bf16, near what the tensor cores sustain under
// the power limit, and the split 1.04 (its memory traffic 0.65; the rest are the
// weights' square roots and divisions); 360 x 384 x 384 1.06 -> 0.41 ms; one view of
// 768 x 768 152 -> 66 us.  The adjoint: 14.83 -> 6.42 ms, 1.13 -> 0.68 ms, 150 -> 91 us.
//
// The Toeplitz operand is never stored as a matrix.  With k reversed (k' = U-1-k)
// it is a Hankel matrix, A[u][k'] = f[u+k'] with f[j] = h[|j-(U-1)|], so in the
// unswizzled K-major layout every 8 x 8 core matrix C[q][r][c] = f[8q+r+c] serves
// all (row group, column group) pairs with the same sum q: both strides of the
// descriptor are one core matrix (128 B), and 128 rows x the whole K of the
// operand are 15 + U/8 core matrices (14 KB a part at U = 768) that a CTA loads
// once.  The other operand, the weighted rows, is MN-major as it lies (v
// contiguous) and comes by TMA.
//
// Persistent CTAs, one per SM: tiles of 128 rows u, the same for all tiles of a CTA,
// x up to 256 columns v of a view.  Warp 0 loads (32 taps of the three parts per
// stage), warp 1 issues the MMAs, warps 4-11 add the leading accumulator into their
// registers while the other five products of the same taps run, and store a tile
// while the next one's products start.  Every wait is bounded; a view on which
// one gave up, like a view whose values are outside the split's range
// (fdk_tc_holds), is recomputed by the FP32 product.
#include <cuda_bf16.h>

#include "common.cuh"
#include "fdk.cuh"
#include "fdk_product.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace dgc {

namespace {

constexpr int kTcRows = 128;     // u per CTA (M)
constexpr int kTcStageK = 32;    // taps per stage and leading accumulation
constexpr int kTcPart = 64 * kTcStageK * 2;  // bytes of a staged part: 64 v x a stage's taps
constexpr int kTcBox = 3 * kTcPart;
// Three warpgroups: producer and MMA warps (and two idle ones), and eight epilogue
// warps whose accumulators take most of the registers that the launch grants.
constexpr int kTcThreads = 384;
constexpr int kTcRegsFew = 40, kTcRegsMany = 224;
constexpr int kTcSmem = 224 * 1024;
constexpr int kTcMaxStages = 12;
constexpr int kTcTurn = 32 * 33;  // floats of an epilogue warp's turned block
constexpr size_t kTcChunkBytes = 256u << 20;  // split operands held at a time

int tc_k(int U) { return (U + kTcStageK - 1) / kTcStageK * kTcStageK; }
int tc_row_stride(int V) { return (V + 7) & ~7; }
int tc_cores(int U) {  // core matrices of the whole strip
    return ((U + kTcRows - 1) / kTcRows * kTcRows + tc_k(U)) / 8;
}
int tc_cta_cores(int U) { return kTcRows / 8 - 1 + tc_k(U) / 8; }
size_t tc_split_bytes(int U, int V) {  // of one view
    return 3 * sizeof(__nv_bfloat16) * (size_t)U * (size_t)tc_row_stride(V);
}

// max(a, b), NaN if either is.
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

struct Split3 {
    __nv_bfloat16 part[3];
};

// x as the sum of three bf16: each takes the leading 8 bits of what is left.
__device__ __forceinline__ Split3 split3(float x) {
    Split3 s;
    s.part[0] = __float2bfloat16(x);
    const float r = x - __bfloat162float(s.part[0]);
    s.part[1] = __float2bfloat16(r);
    s.part[2] = __float2bfloat16(r - __bfloat162float(s.part[1]));
    return s;
}

// split[view][part][U-1-k][v] = part of the staged value of fdk_filter_kernel: the
// cosine-weighted projection, or (ADJ) the upstream gradient; ranges[view][k / 8] =
// the range of its magnitudes.  grid: x = groups of 8 rows, y = view; the blocks
// of the row after the last view fill strip[part][q][8r + c] = part of f[8q + r + c].
// Six blocks per SM (42 registers; left to itself the compiler takes 53): 360 x 384^2
// 78.7 -> 70.4 us, 100 x 768^2 82.8 -> 74.1, of which the ranges' two instructions an
// element are 4.
template <bool ADJ>
__global__ void __launch_bounds__(256, 6) fdk_split_kernel(FdkArgs p, int stride,
                                                        __nv_bfloat16* __restrict__ split,
                                                        FdkRange* __restrict__ ranges, int cores,
                                                        __nv_bfloat16* __restrict__ strip) {
    if (blockIdx.y == p.A) {
        for (int i = blockIdx.x * 256 + threadIdx.x; i < cores * 64; i += gridDim.x * 256) {
            const int j = 8 * (i >> 6) + ((i >> 3) & 7) + (i & 7);
            const int d = j - (p.U - 1);
            const Split3 s = split3(j <= 2 * p.U - 2 ? p.taps[d < 0 ? -d : d] : 0.0f);
#pragma unroll
            for (int k = 0; k < 3; ++k) strip[(size_t)k * cores * 64 + i] = s.part[k];
        }
        return;
    }
    const int a = blockIdx.y;
    const float sid = p.sid[a];
    const float dn = p.frame_dist ? p.frame_dist[a] : sid;
    const float dn2 = __fmul_rn(dn, dn);
    const float cu = p.frame_u ? p.frame_u[a] : 0.5f * (p.U - 1);
    const float cv = p.frame_v ? p.frame_v[a] : 0.5f * (p.V - 1);
    const float* __restrict__ src =
        (ADJ ? p.grad_filtered : p.projections) + (long long)a * p.U * p.V;
    const int groups = stride / 4;
    const bool wide = (p.V & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
    // the largest magnitude (a NaN stays one) and the smallest but zero, as twice its
    // bits less one: a zero is then above all
    float high = 0.0f;
    unsigned low = 0xffffffffu;
    __shared__ int s_high;
    __shared__ unsigned s_low;
    if (threadIdx.x == 0) {
        s_high = 0;
        s_low = 0xffffffffu;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 8 * groups; i += 256) {
        const int row = i / groups, v0 = (i - row * groups) * 4;
        const int k = blockIdx.x * 8 + row;
        if (k >= p.U) break;
        float x[4];
        const float* at = src + (long long)k * p.V + v0;
        if (wide && v0 < p.V) {
            const float4 f = __ldg(reinterpret_cast<const float4*>(at));
            x[0] = f.x;
            x[1] = f.y;
            x[2] = f.z;
            x[3] = f.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = v0 + j < p.V ? __ldg(at + j) : 0.0f;
        }
        if (!ADJ) {
            const float uu = ((float)k - cu) * p.pixel_size;
            const float wk = p.uweight ? p.uweight[(long long)a * p.U + k] : 1.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float vv = ((float)(v0 + j) - cv) * p.pixel_size;
                const float dist = sqrtf(fmaf(vv, vv, fmaf(uu, uu, dn2)));
                x[j] = x[j] * (dn / dist) * wk;
            }
        }
        __align__(8) __nv_bfloat16 h[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            high = max_nan(high, fabsf(x[j]));
            low = min(low, 2u * __float_as_uint(x[j]) - 1u);
            const Split3 s = split3(x[j]);
            h[0][j] = s.part[0];
            h[1][j] = s.part[1];
            h[2][j] = s.part[2];
        }
#pragma unroll
        for (int s = 0; s < 3; ++s)
            *reinterpret_cast<uint2*>(
                split + (((size_t)a * 3 + s) * p.U + (p.U - 1 - k)) * stride + v0) =
                *reinterpret_cast<const uint2*>(h[s]);
    }
    const int top = __reduce_max_sync(0xffffffffu, __float_as_int(high));
    low = __reduce_min_sync(0xffffffffu, low);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&s_high, top);
        atomicMin(&s_low, low);
    }
    __syncthreads();
    if (threadIdx.x == 0)
        ranges[(long long)a * gridDim.x + blockIdx.x] =
            FdkRange{s_low == 0xffffffffu ? INT_MAX : (int)((s_low + 1u) >> 1), s_high};
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes,
                                          uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            dst),
        "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar)
        : "memory");
}

struct TcArgs {
    const __nv_bfloat16* strip;  // [3][cores][64]
    int cores, cta_cores;
    int U, V, n;  // n: columns per tile
    int row_tiles, col_tiles, columns, stages, k_tiles;  // columns: col_tiles * views
    float* out;        // [views][U][V]
    const float* sid;  // null: out = the plain product (the adjoint's z)
    const float* sod;
    float pixel_size;
    FdkRange* ranges;  // [views][ceil(U/8)]
    bool wide, staged;  // stores: 32 bytes a lane; rows by way of shared memory
    int polls;          // LIMIT: of the pipeline's waits (not of those for copies in flight)
};

// LIMIT: the pipeline's waits give up after p.polls polls (as an argument the limit costs
// the kernel 7-10 % of its time, so that calls without one have a constant).
template <bool LIMIT>
__global__ void __launch_bounds__(kTcThreads, 1) fdk_filter_tc_kernel(
    const __grid_constant__ CUtensorMap map, TcArgs p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[kTcMaxStages], empty[kTcMaxStages];
    __shared__ __align__(8) uint64_t strip_full, hi_full, hi_empty, low_full, low_empty, done;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_err, s_consumed;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u0 = (int)(blockIdx.x % p.row_tiles) * kTcRows;
    const int first = blockIdx.x / p.row_tiles, step = gridDim.x / p.row_tiles;
    const int boxes = (p.n + 63) / 64;
    const uint32_t stage_bytes = boxes * kTcBox;
    const uint32_t sbase = (tma_smem_u32(smem) + 1023u) & ~1023u;
    const uint32_t s_strip = sbase + p.stages * stage_bytes;
    const uint32_t strip_bytes = p.cta_cores * 128;  // of one part
    const int S = p.stages, nk = p.k_tiles;          // nk: stages of a tile

    if (warp == 0) tmem_alloc(tma_smem_u32(&tmem_slot), 512);
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) {
            tma_mbar_init(tma_smem_u32(&full[i]), 1);
            tma_mbar_init(tma_smem_u32(&empty[i]), 1);
        }
        tma_mbar_init(tma_smem_u32(&strip_full), 1);
        tma_mbar_init(tma_smem_u32(&hi_full), 1);
        tma_mbar_init(tma_smem_u32(&hi_empty), 8);
        tma_mbar_init(tma_smem_u32(&low_full), 1);
        tma_mbar_init(tma_smem_u32(&low_empty), 8);
        tma_mbar_init(tma_smem_u32(&done), 1);
        tma_fence_init();
        s_err = 0;
        s_consumed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_hi = tmem_slot, tmem_low = tmem_hi + 256;
    volatile int* err = &s_err;
    const long long polls = LIMIT ? p.polls : kTcWaitLimit;

    int issued = 0;  // stages, over all tiles (warp 0)
    bool strip_issued = false;
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kTcRegsFew));
        if (warp == 0 && lane == 0) {
            tma_expect_tx(tma_smem_u32(&strip_full), 3 * strip_bytes);
            for (int s = 0; s < 3; ++s)
                bulk_load(s_strip + s * strip_bytes,
                          p.strip + ((size_t)s * p.cores + u0 / 8) * 64, strip_bytes,
                          tma_smem_u32(&strip_full));
            strip_issued = true;
            int s = 0;
            uint32_t phase = 1;  // of the slots' empty barriers: the first round passes
            for (int tile = first; tile < p.columns && !*err; tile += step) {
                const int v0 = (tile % p.col_tiles) * p.n, a = tile / p.col_tiles;
                for (int kt = 0; kt < nk && !*err; ++kt) {
                    if (!mbar_wait(tma_smem_u32(&empty[s]), phase, polls)) {
                        *err = 1;
                        break;
                    }
                    const uint32_t bar = tma_smem_u32(&full[s]);
                    tma_expect_tx(bar, stage_bytes);
                    for (int b = 0; b < boxes; ++b)
                        tma_load_3d(sbase + s * stage_bytes + b * kTcBox, &map, v0 + 64 * b,
                                    kt * kTcStageK, 3 * a, bar);
                    ++issued;
                    if (++s == S) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
        } else if (warp == 1 && lane == 0) {
            const uint32_t idesc = idesc_bf16(kTcRows, p.n, false, true);
            // descriptors of the strip's and the stages' first parts; addresses count
            // 16-byte units, so 16 taps are 16 units of the strip and 128 of a stage
            const uint64_t a0 = smem_desc(s_strip, 128u, 128u, 0u);
            const uint64_t b0 = smem_desc(sbase, kTcBox, 1024u, 2u);
            const uint32_t a_part = strip_bytes / 16, b_stage = stage_bytes / 16;
            constexpr uint32_t b_part = kTcPart / 16;
            bool ok = mbar_wait(tma_smem_u32(&strip_full), 0, polls);
            int g = 0, s = 0;        // stages so far, this one's slot
            uint32_t phase = 0;      // of the slots' full barriers
            uint32_t done_tiles = 0;
            for (int tile = first; ok && tile < p.columns; tile += step, ++done_tiles) {
                for (int kt = 0; kt < nk; ++kt) {
                    ok = mbar_wait(tma_smem_u32(&full[s]), phase, polls);
                    // the last stage's leading product has been taken
                    if (ok && g > 0) ok = mbar_wait(tma_smem_u32(&hi_empty), (g - 1) & 1, polls);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t at = a0 + kt * kTcStageK, bt = b0 + s * b_stage;
#pragma unroll
                    for (int kk = 0; kk < kTcStageK / 16; ++kk)
                        umma_bf16(tmem_hi, at + 16 * kk, bt + 128 * kk, idesc, kk > 0);
                    umma_commit(tma_smem_u32(&hi_full));
                    // the other five, smallest first
                    if (kt == 0 && done_tiles > 0) {
                        ok = mbar_wait(tma_smem_u32(&low_empty), (done_tiles - 1) & 1, polls);
                        if (!ok) break;
                        tc_fence_after();
                    }
#pragma unroll
                    for (int kk = 0; kk < kTcStageK / 16; ++kk) {
                        const uint64_t ak = at + 16 * kk, bk = bt + 128 * kk;
                        umma_bf16(tmem_low, ak, bk + 2 * b_part, idesc, kt > 0 || kk > 0);
                        umma_bf16(tmem_low, ak + 2 * a_part, bk, idesc, 1);
                        umma_bf16(tmem_low, ak + a_part, bk + b_part, idesc, 1);
                        umma_bf16(tmem_low, ak, bk + b_part, idesc, 1);
                        umma_bf16(tmem_low, ak + a_part, bk, idesc, 1);
                    }
                    umma_commit(tma_smem_u32(&empty[s]));
                    ++g;
                    if (++s == S) {
                        s = 0;
                        phase ^= 1;
                    }
                }
                if (ok) umma_commit(tma_smem_u32(&low_full));
            }
            if (!ok) *err = 1;
            s_consumed = g;
            umma_commit(tma_smem_u32(&done));  // arrives once every MMA issued above has completed
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kTcRegsMany));
        const int half = (warp - 4) >> 2, quarter = warp & 3;  // columns, lanes
        const uint32_t at = (static_cast<uint32_t>(quarter * 32) << 16) + half * 128;
        const int u = u0 + quarter * 32 + lane;
        float* buf = reinterpret_cast<float*>(smem + (s_strip - tma_smem_u32(smem)) + 3 * strip_bytes) +
                     (warp - 4) * kTcTurn;  // staged: this warp's 32 x 32 block
        const int left = p.n - half * 128;  // columns of this half
        // acc += the accumulator at `src`, which the arrival on `bar` then releases
        const auto take = [&](uint32_t src, uint32_t bar, float (&acc)[128]) {
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (32 * i < left) {
                    float v[32];
                    tmem_load32(src + 32 * i, v);
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[32 * i + j] += v[j];
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        int chunk = 0, done_tiles = 0;
        bool ok = true;
        for (int tile = first; ok && tile < p.columns; tile += step, ++done_tiles) {
            float acc[128];
#pragma unroll
            for (int i = 0; i < 128; ++i) acc[i] = 0.0f;
            for (int c = 0; c < nk; ++c, ++chunk) {
                ok = __all_sync(0xffffffffu, mbar_wait(tma_smem_u32(&hi_full), chunk & 1, polls));
                if (!ok) break;
                take(tmem_hi + at, tma_smem_u32(&hi_empty), acc);
            }
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(tma_smem_u32(&low_full), done_tiles & 1, polls));
            if (!ok) break;
            take(tmem_low + at, tma_smem_u32(&low_empty), acc);
            // the next tile's products run while this one is stored
            const int v0 = (tile % p.col_tiles) * p.n + half * 128, a = tile / p.col_tiles;
            if (p.sid) {  // filtering.py:104: filtered * pixel_size * (sid / sod)
                const float ratio = p.sid[a] / p.sod[a];
#pragma unroll
                for (int i = 0; i < 128; ++i) acc[i] = (acc[i] * p.pixel_size) * ratio;
            }
            if (p.staged) {
                // a lane holds a row: turned, a warp stores rows of 32 columns
#pragma unroll
                for (int cb = 0; cb < 128; cb += 32) {
                    if (cb >= left) break;
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 32; ++i) buf[lane * 33 + i] = acc[cb + i];
                    __syncwarp();
                    const int rows = min(32, p.U - (u - lane)), col = v0 + cb + lane;
                    if (cb + lane < left && col < p.V) {
                        float* __restrict__ to = p.out + ((long long)a * p.U + (u - lane)) * p.V + col;
#pragma unroll 8
                        for (int r = 0; r < rows; ++r, to += p.V) *to = buf[r * 33 + lane];
                    }
                }
            } else {
                float* __restrict__ row = p.out + ((long long)a * p.U + u) * p.V;
#pragma unroll
                for (int i = 0; i < 128; i += 8) {
                    const int col = v0 + i;
                    if (u < p.U && i < left) {
                        if (p.wide && col + 8 <= p.V) {
                            uint32_t x[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) x[k] = __float_as_uint(acc[i + k]);
                            store32(row + col, x);
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                if (col + k < p.V) row[col + k] = acc[i + k];
                        }
                    }
                }
            }
            __syncwarp();
        }
        if (!ok) *err = 1;
    }
    __syncthreads();
    bool ok = *err == 0;
    // every MMA, and with them every read of the staged tiles, is complete
    if (!mbar_wait(tma_smem_u32(&done), 0)) ok = false;
    ok = __syncthreads_and(ok);
    if (!ok && threadIdx.x == 0) {
        // copies that nothing waited for must land before the shared memory is
        // released; every view of this CTA is left to the FP32 product
        if (strip_issued) mbar_wait(tma_smem_u32(&strip_full), 0);
        for (int g = s_consumed; g < issued; ++g)
            mbar_wait(tma_smem_u32(&full[g % S]), (g / S) & 1);
        for (int tile = first; tile < p.columns; tile += step)
            p.ranges[(long long)(tile / p.col_tiles) * ((p.U + 7) / 8)].high = INT_MAX;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_free(tmem_hi, 512);
    }
}

// Polls after which this thread's launches give a wait up, or -1: the constant.
thread_local int tc_polls = -1;

// 3-D map of the split rows: V columns, U rows, 3 parts a view; boxes of 64 columns x
// kTcStageK rows x the parts, 128-byte swizzle, zero fill outside.
bool split_map(CUtensorMap* map, const __nv_bfloat16* split, int views, int U, int V) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    const size_t row = sizeof(__nv_bfloat16) * (size_t)tc_row_stride(V);
    const cuuint64_t dims[3] = {(cuuint64_t)V, (cuuint64_t)U, (cuuint64_t)(3 * (long long)views)};
    const cuuint64_t strides[2] = {(cuuint64_t)row, (cuuint64_t)(row * (size_t)U)};
    const cuuint32_t box[3] = {64, kTcStageK, 3};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(split), dims,
              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The product of `views` split views into out (scaled where f is given).
int launch_tc(const FdkArgs* f, const __nv_bfloat16* strip, const __nv_bfloat16* split, int views,
              int U, int V, float* out, FdkRange* ranges, cudaStream_t s, bool* used) {
    *used = false;
    CUtensorMap map;
    if (!split_map(&map, split, views, U, V)) return DGC_OK;
    TcArgs p;
    p.strip = strip;
    p.cores = tc_cores(U);
    p.cta_cores = tc_cta_cores(U);
    p.U = U;
    p.V = V;
    p.col_tiles = ceil_div(V, 256);
    p.n = (ceil_div(V, p.col_tiles) + 15) & ~15;
    p.row_tiles = ceil_div(U, kTcRows);
    p.k_tiles = tc_k(U) / kTcStageK;
    const int stage_bytes = ceil_div(p.n, 64) * kTcBox;
    const int strip_bytes = 3 * p.cta_cores * 128;
    // Rows that do not start on 32 bytes are turned in shared memory where two stages
    // are left beside it: stores of 4 bytes a lane, one row each, take 32 sectors an
    // instruction (filter of 200 x 187 x 161 104 -> 73 us, of 100 x 384 x 381 201 -> 141).
    constexpr int kTurnBytes = 8 * kTcTurn * (int)sizeof(float);
    p.wide = (V & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 31u) == 0;
    p.staged = !p.wide && (kTcSmem - strip_bytes - kTurnBytes) / stage_bytes >= 2;
    const int turn_bytes = p.staged ? kTurnBytes : 0;
    p.stages = std::min(kTcMaxStages, (kTcSmem - strip_bytes - turn_bytes) / stage_bytes);
    p.out = out;
    p.sid = f ? f->sid : nullptr;
    p.sod = f ? f->sod : nullptr;
    p.pixel_size = f ? f->pixel_size : 1.0f;
    p.ranges = ranges;
    p.polls = tc_polls;
    static std::atomic<unsigned long long> configured{0}, unfit{0};
    const int rc = once_per_device(configured, []() -> int {
        for (const auto kernel : {fdk_filter_tc_kernel<false>, fdk_filter_tc_kernel<true>}) {
            DGC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kTcSmem + 1024));
            // the register split must fit what a launch grants, or it would wait for good
            cudaFuncAttributes attr;
            DGC_CUDA(cudaFuncGetAttributes(&attr, kernel));
            if (attr.numRegs * kTcThreads < 128 * kTcRegsFew + 256 * kTcRegsMany) unfit.store(1);
        }
        return DGC_OK;
    });
    if (rc != DGC_OK) return rc;
    if (unfit.load()) return DGC_OK;  // the FP32 product takes the call
    DGC_TRACE("fdk_filter_tc_kernel", s);
    // a CTA keeps its rows (and their strip), so the grid is whole sets of row tiles
    p.columns = p.col_tiles * views;
    int dev = 0, sms = 0;
    DGC_CUDA(cudaGetDevice(&dev));
    DGC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const unsigned grid =
        (unsigned)(p.row_tiles * std::min(p.columns, std::max(1, sms / p.row_tiles)));
    const size_t smem = p.stages * stage_bytes + strip_bytes + turn_bytes + 1024;
    if (p.polls < 0) fdk_filter_tc_kernel<false><<<grid, kTcThreads, smem, s>>>(map, p);
    else fdk_filter_tc_kernel<true><<<grid, kTcThreads, smem, s>>>(map, p);
    DGC_LAUNCH_CHECK("fdk_filter_tc_kernel");
    *used = true;
    return DGC_OK;
}

template <bool ADJ>
int launch_split(const FdkArgs& p, __nv_bfloat16* split, FdkRange* ranges, __nv_bfloat16* strip,
                 cudaStream_t s) {
    DGC_TRACE("fdk_split_kernel", s);
    const dim3 grid((unsigned)ceil_div(p.U, 8), (unsigned)p.A + (strip ? 1 : 0));
    fdk_split_kernel<ADJ><<<grid, 256, 0, s>>>(p, tc_row_stride(p.V), split, ranges, tc_cores(p.U),
                                               strip);
    DGC_LAUNCH_CHECK("fdk_split_kernel");
    return DGC_OK;
}

// The epilogue of the FP32 adjoint from a stored z = H(g) (the tensor cores'
// product), with its tiles and sums, for the views that these hold.  1024 threads, so
// that a thread's chain of FP64 divisions is 16 elements long and a warp reads whole
// rows: 4.12 -> 2.38 ms at 720 x 768 x 768 against 64 elements a thread in the product's
// layout; with an element's four loads ahead of its branch 100 x 768 x 768 takes 0.283 ms
// for 0.341 (all gradients), 0.251 for 0.275 (the distances' alone).
constexpr int kEpilogueThreads = 1024;

template <bool CG>
__global__ void __launch_bounds__(kEpilogueThreads, 2) fdk_adjoint_epilogue_kernel(
    FdkLeft p, const float* __restrict__ z) {
    constexpr int kWarps = kEpilogueThreads / 32, kRows = kEpilogueThreads / kFdkTileColumns;
    __shared__ double s_part[kWarps][kFdkPartials];
    const int a = blockIdx.z;
    if (!fdk_tc_holds(p, a)) return;
    const float ratio = p.sid[a] / p.sod[a];
    const float dn = p.frame_dist ? p.frame_dist[a] : p.sid[a];
    const float dn2 = dn * dn;
    const float cu = p.frame_u ? p.frame_u[a] : 0.5f * (p.U - 1);
    const float cv = p.frame_v ? p.frame_v[a] : 0.5f * (p.V - 1);
    const long long base = (long long)a * p.U * p.V;
    const bool sums = p.partials != nullptr;
    const int u0 = blockIdx.y * kFdkTileRows + threadIdx.x / kFdkTileColumns;
    const int v = blockIdx.x * kFdkTileColumns + threadIdx.x % kFdkTileColumns;
    const float vv = ((float)v - cv) * p.pixel_size;
    double s_gy = 0.0, s_zpw = 0.0, s_zpu = 0.0, s_zpv = 0.0;
#pragma unroll 4
    for (int i = 0; i < kFdkTileRows; i += kRows) {
        const int u = u0 + i;
        const bool in = u < p.U && v < p.V;
        const long long idx = base + (long long)u * p.V + v;
        // the loads together, ahead of the branch
        const float zv = in ? z[idx] : 0.0f;
        const float pv = in && sums ? p.projections[idx] : 0.0f;
        const float gv = in && sums ? p.grad_filtered[idx] : 0.0f;
        const float yv = in && sums ? p.forward_out[idx] : 0.0f;
        if (!in) continue;
        const float uu = ((float)u - cu) * p.pixel_size;
        const float r2 = uu * uu + vv * vv;
        const float dist = sqrtf(dn2 + r2);
        if (p.grad_projections) p.grad_projections[idx] = (zv * p.pixel_size) * ratio * (dn / dist);
        if (sums) {
            const double zp = (double)zv * (double)pv;
            const double d3 = (double)dist * dist * dist;
            s_gy += (double)gv * (double)yv;
            s_zpw += zp * ((double)r2 / d3);
            if (CG) {
                s_zpu += zp * ((double)uu / d3);
                s_zpv += zp * ((double)vv / d3);
            }
        }
    }
    if (!sums) return;
    // the CTA's sums in a fixed order, as the FP32 adjoint's
    constexpr int kSums = CG ? 4 : 2;
    s_gy = warp_sum(s_gy);
    s_zpw = warp_sum(s_zpw);
    if (CG) {
        s_zpu = warp_sum(s_zpu);
        s_zpv = warp_sum(s_zpv);
    }
    const int tid = threadIdx.x;
    if ((tid & 31) == 0) {
        double* part = s_part[tid >> 5];
        part[0] = s_gy;
        part[1] = s_zpw;
        if (CG) {
            part[2] = s_zpu;
            part[3] = s_zpv;
        }
    }
    __syncthreads();
    if (tid < kFdkPartials) {
        double t = 0.0;
        if (tid < kSums)
            for (int w = 0; w < kWarps; ++w) t += s_part[w][tid];
        const long long tiles = (long long)gridDim.x * gridDim.y;
        const long long tile = (long long)blockIdx.y * gridDim.x + blockIdx.x;
        p.partials[((long long)a * tiles + tile) * kFdkPartials + tid] = t;
    }
}

int launch_epilogue(const FdkLeft& p, const float* z, cudaStream_t s) {
    DGC_TRACE("fdk_adjoint_epilogue", s);
    const dim3 grid(ceil_div(p.V, kFdkTileColumns), ceil_div(p.U, kFdkTileRows), p.A);
    if (p.frame_grads)
        fdk_adjoint_epilogue_kernel<true><<<grid, kEpilogueThreads, 0, s>>>(p, z);
    else
        fdk_adjoint_epilogue_kernel<false><<<grid, kEpilogueThreads, 0, s>>>(p, z);
    DGC_LAUNCH_CHECK("fdk_adjoint_epilogue");
    return DGC_OK;
}

// The FP32 product of the views that the tensor cores' does not hold.
int launch_left(const FdkLeft& p, bool adjoint, cudaStream_t s) {
    DGC_TRACE("fdk_filter_left", s);
    const dim3 grid(ceil_div(p.V, FBN), ceil_div(p.U, FBM), p.A);
    if (!adjoint)
        fdk_filter_kernel<false, false, FdkLeft><<<grid, 256, 0, s>>>(p);
    else if (p.frame_grads)
        fdk_filter_kernel<true, true, FdkLeft><<<grid, 256, 0, s>>>(p);
    else
        fdk_filter_kernel<true, false, FdkLeft><<<grid, 256, 0, s>>>(p);
    DGC_LAUNCH_CHECK("fdk_filter_left");
    return DGC_OK;
}

// Views a0 .. a0+n-1 of the arguments.
FdkArgs views_of(const FdkArgs& p, int a0, int n) {
    FdkArgs q = p;
    const long long skip = (long long)a0 * p.U * p.V;
    const auto shift = [](auto*& ptr, long long by) {
        if (ptr) ptr += by;
    };
    shift(q.projections, skip);
    shift(q.filtered, skip);
    shift(q.grad_filtered, skip);
    shift(q.forward_out, skip);
    shift(q.grad_projections, skip);
    shift(q.sod, a0);
    shift(q.sid, a0);
    shift(q.frame_dist, a0);
    shift(q.frame_u, a0);
    shift(q.frame_v, a0);
    shift(q.uweight, (long long)a0 * p.U);
    shift(q.partials, (long long)a0 * fdk_filter_tiles(p.U, p.V) * kFdkPartials);
    q.A = n;
    return q;
}

}  // namespace

void fdk_tc_limit_waits(int polls) { tc_polls = std::max(polls, -1); }

int fdk_tc_views(int A, int U, int V, bool adjoint) {
    // Below, the FP32 product's time is that of its chain over U, the tensor cores' that of
    // their launches and of rows that the tile of 128 pads.  Tensor cores / FP32, over
    // 1 to 512 views of 16 to 600 columns: the filter 0.68-1.14 at U = 96 (0.79-1.04 to 64
    // columns), 0.66-1.09 at 112 (0.79-1.05 to 128), 0.63-0.98 at 128, 0.40-0.66 at 256; the adjoint, whose epilogue is a launch of
    // its own, 0.77-1.25 at 96, 0.82-1.20 at 128, 0.56-1.16 at 129 to 160 (0.56-1.08
    // from 96 columns), 0.56-1.07 at 192, 0.54-0.94 at 256.  To 2048: the strip and two stages
    // fill the shared memory.  The rule has no number of views in it, so that a view's
    // result does not depend on its neighbours.
    const bool rows = adjoint ? U >= 192 || (U >= 129 && V >= 96)
                              : U >= (V <= 64 ? 96 : V <= 128 ? 112 : 128);
    if (A < 1 || !rows || U > 2048 || V < 16 || tc_split_bytes(U, V) > kTcChunkBytes) return 0;
    const int most = (int)std::min<long long>(16384, (long long)(kTcChunkBytes / tc_split_bytes(U, V)));
    return ceil_div(A, ceil_div(A, most));  // equal chunks
}

size_t fdk_tc_scratch(int U, int V, bool adjoint, int views) {
    return Workspace::align(3 * 128 * (size_t)tc_cores(U)) +
           Workspace::align(sizeof(FdkRange) * (size_t)views * (size_t)ceil_div(U, 8)) +
           Workspace::align(tc_split_bytes(U, V) * (size_t)views) +
           (adjoint ? Workspace::align(sizeof(float) * (size_t)U * V * (size_t)views) : 0);
}

size_t fdk_tc_bytes(int A, int U, int V, bool adjoint) {
    const int views = fdk_tc_views(A, U, V, adjoint);
    return views ? fdk_tc_scratch(U, V, adjoint, views) : 0;
}

// Views at a time: those of the rule or, in less room, as many as it holds (a view's
// result is the same whatever their number).
static int views_that_fit(const FdkArgs& p, bool adjoint, const Workspace& ws) {
    const size_t room = ws.base ? ws.size - ws.used : 0;
    int low = 0, high = fdk_tc_views(p.A, p.U, p.V, adjoint);
    if (!high || fdk_tc_scratch(p.U, p.V, adjoint, high) <= room) return high;
    while (low + 1 < high) {
        const int mid = (low + high) / 2;
        (fdk_tc_scratch(p.U, p.V, adjoint, mid) <= room ? low : high) = mid;
    }
    return low;
}

int fdk_tc_filter(const FdkArgs& p, bool adjoint, Workspace ws, cudaStream_t s, bool* used) {
    *used = false;
    const int views = views_that_fit(p, adjoint, ws);
    if (!views) return DGC_OK;
    __nv_bfloat16* strip = ws.take<__nv_bfloat16>((size_t)3 * 64 * (size_t)tc_cores(p.U));
    FdkRange* ranges = ws.take<FdkRange>((size_t)views * (size_t)ceil_div(p.U, 8));
    __nv_bfloat16* split = reinterpret_cast<__nv_bfloat16*>(
        ws.take<char>(tc_split_bytes(p.U, p.V) * (size_t)views));
    float* z = adjoint ? ws.take<float>((size_t)p.U * p.V * (size_t)views) : nullptr;
    if (!strip || !ranges || !split || (adjoint && !z)) return DGC_OK;
    for (int a0 = 0; a0 < p.A; a0 += views) {
        FdkArgs q = views_of(p, a0, std::min(views, p.A - a0));
        __nv_bfloat16* fill = a0 == 0 ? strip : nullptr;  // the taps serve every chunk
        int rc = adjoint ? launch_split<true>(q, split, ranges, fill, s)
                         : launch_split<false>(q, split, ranges, fill, s);
        if (rc != DGC_OK) return rc;
        bool launched = false;
        rc = launch_tc(adjoint ? nullptr : &q, strip, split, q.A, q.U, q.V,
                       adjoint ? z : q.filtered, ranges, s, &launched);
        if (rc != DGC_OK) return rc;
        if (!launched) {
            if (a0 == 0) return DGC_OK;  // nothing written yet: the SIMT product takes the call
            set_error("fdk filter: no tensor map for a later chunk of views");
            return DGC_ERR_CUDA;
        }
        const FdkLeft left(q, ranges);
        if (adjoint) {
            if ((rc = launch_epilogue(left, z, s)) != DGC_OK) return rc;
        }
        if ((rc = launch_left(left, adjoint, s)) != DGC_OK) return rc;
    }
    *used = true;
    return DGC_OK;
}

}  // namespace dgc
