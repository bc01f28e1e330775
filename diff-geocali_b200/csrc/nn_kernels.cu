// nn_kernels.cu -- data movement around the tensor-core GEMM for the
// convolution layers of the warm-start network (NHWC activations).
// No counterpart in the reference.
//
//   im2col:  col[(b*Ho + oy)*Wo + ox][(ky*kw + kx)*C + c] = x[b][oy*s - p + ky][ox*s - p + kx][c]
//            (zero outside the image and for k >= kh*kw*C up to the padded width Kp)
//   col2im:  the adjoint, as a gather per input element (no atomics), to fp32 or
//            rounded to bf16.
//   relu_grad: g = gy * (y > 0) and its column sums (the bias gradient).
//
// All are bound by memory traffic, so they move 16 bytes a thread and keep the
// index arithmetic to 32 bits with one division by a launch-wide size per step.
#include <cuda_bf16.h>

#include "common.cuh"

namespace dgc {
namespace {

__global__ void im2col_nhwc_kernel(const __nv_bfloat16* __restrict__ x, int B, int H, int W, int C,
                                   int kh, int kw, int stride, int pad, int Ho, int Wo,
                                   __nv_bfloat16* __restrict__ col, int Kp, bool vec8) {
    const long long rows = (long long)B * Ho * Wo;
    const int kchunks = vec8 ? Kp / 8 : Kp;
    const long long total = rows * kchunks;
    const int Kreal = kh * kw * C;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long m = i / kchunks;
        const int kc = (int)(i - m * kchunks);
        const int k = vec8 ? kc * 8 : kc;
        const int ox = (int)(m % Wo);
        const long long t = m / Wo;
        const int oy = (int)(t % Ho);
        const int b = (int)(t / Ho);
        const int tap = k / C, c = k - tap * C;
        const int ky = tap / kw, kx = tap - ky * kw;
        const int iy = oy * stride - pad + ky, ix = ox * stride - pad + kx;
        const bool inside = k < Kreal && iy >= 0 && iy < H && ix >= 0 && ix < W;
        const long long src = (((long long)b * H + iy) * W + ix) * C + c;
        if (vec8) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (inside) v = *reinterpret_cast<const uint4*>(x + src);
            *reinterpret_cast<uint4*>(col + m * Kp + k) = v;
        } else {
            col[m * Kp + k] = inside ? x[src] : __float2bfloat16(0.0f);
        }
    }
}

// Eight channels (16 bytes) of one tap a thread; a block walks the chunks of one
// output row (b, oy).
__global__ void __launch_bounds__(256) im2col_row_kernel(const __nv_bfloat16* __restrict__ x, int H,
                                                         int W, int C, int kh, int kw, int stride,
                                                         int pad, int Ho, int Wo,
                                                         __nv_bfloat16* __restrict__ col, int Kp) {
    const int b = blockIdx.x / Ho, oy = blockIdx.x - b * Ho;
    const int chunks = Kp / 8, c8 = C / 8, taps = kh * kw;
    uint4* __restrict__ out =
        reinterpret_cast<uint4*>(col + (long long)blockIdx.x * Wo * Kp);
    for (int i = threadIdx.x; i < Wo * chunks; i += 256) {
        const int ox = i / chunks, kc = i - ox * chunks;
        const int tap = kc / c8, c = kc - tap * c8;
        const int ky = tap / kw, kx = tap - ky * kw;
        const int iy = oy * stride - pad + ky, ix = ox * stride - pad + kx;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (tap < taps && iy >= 0 && iy < H && ix >= 0 && ix < W)
            v = *reinterpret_cast<const uint4*>(x + (((long long)b * H + iy) * W + ix) * C + c * 8);
        out[i] = v;
    }
}

// The same for few channels (the network's input): a thread gathers the 8 values
// of its chunk one by one.
__global__ void __launch_bounds__(256) im2col_row_few_kernel(const __nv_bfloat16* __restrict__ x,
                                                             int H, int W, int C, int kh, int kw,
                                                             int stride, int pad, int Ho, int Wo,
                                                             __nv_bfloat16* __restrict__ col,
                                                             int Kp) {
    const int b = blockIdx.x / Ho, oy = blockIdx.x - b * Ho;
    const int chunks = Kp / 8, real = kh * kw * C;
    uint4* __restrict__ out =
        reinterpret_cast<uint4*>(col + (long long)blockIdx.x * Wo * Kp);
    for (int i = threadIdx.x; i < Wo * chunks; i += 256) {
        const int ox = i / chunks, kc = i - ox * chunks;
        __align__(16) __nv_bfloat16 h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = kc * 8 + j;
            const int tap = k / C, c = k - tap * C;
            const int ky = tap / kw, kx = tap - ky * kw;
            const int iy = oy * stride - pad + ky, ix = ox * stride - pad + kx;
            const bool inside = k < real && iy >= 0 && iy < H && ix >= 0 && ix < W;
            h[j] = inside ? x[(((long long)b * H + iy) * W + ix) * C + c] : __float2bfloat16(0.0f);
        }
        out[i] = *reinterpret_cast<const uint4*>(h);
    }
}

// Input element i of [B][H][W][C] as a sum over its taps, VEC channels a thread,
// in the order ky, kx whatever VEC and the output type; a block walks one input
// row (b, iy).  1.30 -> 0.40 ms over the network at 180 views (1.1 GB of columns).
template <int VEC, typename Out>
__global__ void __launch_bounds__(256) col2im_nhwc_kernel(const float* __restrict__ col, int H, int W,
                                                          int C, int kh, int kw, int stride,
                                                          int pad, int Ho, int Wo, int Kp,
                                                          Out* __restrict__ dx) {
    const int b = blockIdx.x / H, iy = blockIdx.x - b * H;
    const int cv = C / VEC;
    Out* __restrict__ out = dx + (long long)blockIdx.x * W * C;
    for (int i = threadIdx.x; i < W * cv; i += 256) {
        const int ix = i / cv, c = (i - ix * cv) * VEC;
        float acc[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) acc[j] = 0.0f;
        for (int ky = 0; ky < kh; ++ky) {
            const int ny = iy + pad - ky;
            const int oy = ny / stride;
            if (ny < 0 || oy * stride != ny || oy >= Ho) continue;
            for (int kx = 0; kx < kw; ++kx) {
                const int nx = ix + pad - kx;
                const int ox = nx / stride;
                if (nx < 0 || ox * stride != nx || ox >= Wo) continue;
                const float* __restrict__ src =
                    col + (((long long)b * Ho + oy) * Wo + ox) * Kp + (ky * kw + kx) * C + c;
                if constexpr (VEC == 4) {
                    const float4 v = __ldg(reinterpret_cast<const float4*>(src));
                    acc[0] += v.x;
                    acc[1] += v.y;
                    acc[2] += v.z;
                    acc[3] += v.w;
                } else {
                    acc[0] += __ldg(src);
                }
            }
        }
        if constexpr (VEC == 4 && sizeof(Out) == 4) {
            *reinterpret_cast<float4*>(out + i * 4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        } else if constexpr (VEC == 4) {
            __align__(8) __nv_bfloat16 h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) h[j] = __float2bfloat16(acc[j]);
            *reinterpret_cast<uint2*>(out + i * 4) = *reinterpret_cast<const uint2*>(h);
        } else if constexpr (sizeof(Out) == 4) {
            out[i] = acc[0];
        } else {
            out[i] = __float2bfloat16(acc[0]);
        }
    }
}

// g = gy * (y > 0) (y null: g = gy) for [M][C] bf16, C a multiple of 8, and each
// block's FP32 column sums of g: a thread owns 8 channels and every
// (256 / (C/8))-th row of its block's rows.  partial: [blocks][C].
__global__ void __launch_bounds__(256) relu_grad_kernel(const __nv_bfloat16* __restrict__ gy,
                                                        const __nv_bfloat16* __restrict__ y, int M,
                                                        int C, int rows_per_block,
                                                        __nv_bfloat16* __restrict__ g,
                                                        float* __restrict__ partial) {
    __shared__ float s_sum[256][9];
    const int c8 = C / 8, lanes = 256 / c8;  // threads per row, rows at a time
    const int r = threadIdx.x / c8, c = threadIdx.x - r * c8;
    const int m0 = blockIdx.x * rows_per_block, m1 = min(m0 + rows_per_block, M);
    float sum[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) sum[j] = 0.0f;
    if (r < lanes) {
        for (int m = m0 + r; m < m1; m += lanes) {
            const long long at = (long long)m * c8 + c;
            uint4 v = reinterpret_cast<const uint4*>(gy)[at];
            __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(&v);
            if (y) {
                const uint4 w = reinterpret_cast<const uint4*>(y)[at];
                const __nv_bfloat16* k = reinterpret_cast<const __nv_bfloat16*>(&w);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    h[j] = __float2bfloat16(__bfloat162float(h[j]) *
                                            (__bfloat162float(k[j]) > 0.0f ? 1.0f : 0.0f));
                reinterpret_cast<uint4*>(g)[at] = v;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) sum[j] += __bfloat162float(h[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s_sum[threadIdx.x][j] = sum[j];
    __syncthreads();
    for (int i = threadIdx.x; i < C; i += 256) {
        float t = 0.0f;
        for (int k = 0; k < lanes; ++k) t += s_sum[k * c8 + i / 8][i % 8];
        partial[(long long)blockIdx.x * C + i] = t;
    }
}

// db[c] = sum of the blocks' partials, in order, in FP64: one warp per channel.
__global__ void __launch_bounds__(256) bias_grad_kernel(const float* __restrict__ partial, int blocks,
                                                        int C, float* __restrict__ db) {
    const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= C) return;
    double t = 0.0;
    for (int b = lane; b < blocks; b += 32) t += (double)partial[(long long)b * C + c];
    t = warp_sum(t);
    if (lane == 0) db[c] = (float)t;
}

// Blocks of relu_grad_kernel: up to eight per SM, 64 rows each at least.
int relu_grad_blocks(int M) { return std::max(1, std::min(148 * 8, ceil_div(M, 64))); }

int conv_out(int n, int k, int stride, int pad) { return (n + 2 * pad - k) / stride + 1; }

}  // namespace
}  // namespace dgc

using namespace dgc;

extern "C" int dgc_im2col_nhwc_bf16(const void* x, int B, int H, int W, int C, int kh, int kw,
                                    int stride, int pad, void* col, int Kp, void* stream) {
    clear_error();
    DGC_REQUIRE(x && col, "x and col must be non-null");
    DGC_REQUIRE(B > 0 && H > 0 && W > 0 && C > 0 && kh > 0 && kw > 0 && stride > 0 && pad >= 0,
                "invalid convolution shape");
    DGC_REQUIRE(Kp >= kh * kw * C, "Kp must be >= kh*kw*C");
    const int Ho = conv_out(H, kh, stride, pad), Wo = conv_out(W, kw, stride, pad);
    DGC_REQUIRE(Ho > 0 && Wo > 0, "empty convolution output");
    cudaStream_t s = (cudaStream_t)stream;
    DGC_TRACE("im2col_nhwc", s);
    const bool vec8 = (C % 8 == 0) && (Kp % 8 == 0) && ((uintptr_t)x % 16 == 0) &&
                      ((uintptr_t)col % 16 == 0);
    const bool rows = Kp % 8 == 0 && ((uintptr_t)col % 16 == 0) && (long long)B * Ho < (1LL << 31) &&
                      (long long)Wo * Kp < (1LL << 31);
    if (rows && !vec8) {
        im2col_row_few_kernel<<<(unsigned)(B * Ho), 256, 0, s>>>(
            static_cast<const __nv_bfloat16*>(x), H, W, C, kh, kw, stride, pad, Ho, Wo,
            static_cast<__nv_bfloat16*>(col), Kp);
        DGC_LAUNCH_CHECK("im2col_nhwc");
        return DGC_OK;
    }
    if (rows) {
        im2col_row_kernel<<<(unsigned)(B * Ho), 256, 0, s>>>(
            static_cast<const __nv_bfloat16*>(x), H, W, C, kh, kw, stride, pad, Ho, Wo,
            static_cast<__nv_bfloat16*>(col), Kp);
        DGC_LAUNCH_CHECK("im2col_nhwc");
        return DGC_OK;
    }
    const long long total = (long long)B * Ho * Wo * (vec8 ? Kp / 8 : Kp);
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148LL * 32);
    im2col_nhwc_kernel<<<blocks, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(x), B, H, W, C, kh,
                                              kw, stride, pad, Ho, Wo,
                                              static_cast<__nv_bfloat16*>(col), Kp, vec8);
    DGC_LAUNCH_CHECK("im2col_nhwc");
    return DGC_OK;
}

namespace {

template <typename Out>
int col2im(const float* col, int B, int H, int W, int C, int kh, int kw, int stride, int pad, int Kp,
           Out* dx, cudaStream_t s) {
    DGC_REQUIRE(col && dx, "col and dx must be non-null");
    DGC_REQUIRE(B > 0 && H > 0 && W > 0 && C > 0 && kh > 0 && kw > 0 && stride > 0 && pad >= 0,
                "invalid convolution shape");
    DGC_REQUIRE(Kp >= kh * kw * C, "Kp must be >= kh*kw*C");
    const int Ho = conv_out(H, kh, stride, pad), Wo = conv_out(W, kw, stride, pad);
    DGC_REQUIRE(Ho > 0 && Wo > 0, "empty convolution output");
    DGC_REQUIRE((long long)B * H < (1LL << 31) && (long long)W * C < (1LL << 31),
                "convolution too large for one launch");
    DGC_TRACE("col2im_nhwc", s);
    const bool vec4 = C % 4 == 0 && Kp % 4 == 0 && ((uintptr_t)col % 16 == 0) &&
                      ((uintptr_t)dx % (4 * sizeof(Out)) == 0);
    const unsigned blocks = (unsigned)((long long)B * H);
    if (vec4)
        col2im_nhwc_kernel<4, Out><<<blocks, 256, 0, s>>>(col, H, W, C, kh, kw, stride, pad, Ho, Wo,
                                                          Kp, dx);
    else
        col2im_nhwc_kernel<1, Out><<<blocks, 256, 0, s>>>(col, H, W, C, kh, kw, stride, pad, Ho, Wo,
                                                          Kp, dx);
    DGC_LAUNCH_CHECK("col2im_nhwc");
    return DGC_OK;
}

}  // namespace

extern "C" int dgc_col2im_nhwc_f32(const float* col, int B, int H, int W, int C, int kh, int kw,
                                   int stride, int pad, int Kp, float* dx, void* stream) {
    clear_error();
    return col2im(col, B, H, W, C, kh, kw, stride, pad, Kp, dx, (cudaStream_t)stream);
}

extern "C" int dgc_col2im_nhwc_bf16(const float* col, int B, int H, int W, int C, int kh, int kw,
                                    int stride, int pad, int Kp, void* dx, void* stream) {
    clear_error();
    return col2im(col, B, H, W, C, kh, kw, stride, pad, Kp, static_cast<__nv_bfloat16*>(dx),
                  (cudaStream_t)stream);
}

extern "C" size_t dgc_relu_grad_workspace_bytes(int M, int C) {
    if (M <= 0 || C <= 0) return 0;
    return Workspace::align(sizeof(float) * (size_t)relu_grad_blocks(M) * (size_t)C);
}

extern "C" int dgc_relu_grad_bf16(const void* gy, const void* y, int M, int C, void* g, float* db,
                                  void* workspace, size_t workspace_bytes, void* stream) {
    clear_error();
    cudaStream_t s = (cudaStream_t)stream;
    DGC_REQUIRE(gy && db && (!y || g), "gy, db and (with y) g must be non-null");
    DGC_REQUIRE(M > 0 && C > 0 && C % 8 == 0 && C <= 2048, "C must be a multiple of 8 up to 2048");
    DGC_REQUIRE((((uintptr_t)gy | (uintptr_t)y | (uintptr_t)g) & 15u) == 0,
                "gy, y and g must be 16-byte aligned");
    Workspace ws(workspace, workspace_bytes);
    const int blocks = relu_grad_blocks(M);
    float* partial = ws.take<float>((size_t)blocks * C);
    if (!partial) {
        set_error("workspace too small: dgc_relu_grad_bf16 needs " +
                  std::to_string(dgc_relu_grad_workspace_bytes(M, C)) + " bytes");
        return DGC_ERR_WORKSPACE;
    }
    DGC_TRACE("relu_grad", s);
    relu_grad_kernel<<<blocks, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(gy),
                                            static_cast<const __nv_bfloat16*>(y), M, C,
                                            ceil_div(M, blocks), static_cast<__nv_bfloat16*>(g),
                                            partial);
    DGC_LAUNCH_CHECK("relu_grad");
    bias_grad_kernel<<<ceil_div(C, 8), 256, 0, s>>>(partial, blocks, C, db);
    DGC_LAUNCH_CHECK("bias_grad");
    return DGC_OK;
}
