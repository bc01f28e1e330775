// fdk_product.cuh -- the FP32 product of the FDK filter and its adjoint, a template that
// fdk.cu instantiates for whole calls and fdk_tc.cu for the views that the tensor
// cores leave.
#pragma once

#include <climits>
#include <type_traits>

#include "fdk.cuh"

namespace dgc {

// The smallest magnitude but zero and the largest (their bits; INT_MAX and 0 without
// any) of what the tensor cores' product was given of eight rows of a view.
struct FdkRange {
    int low, high;
};

// The tensor cores' views, with their values' `ranges`.  They leave views outside
// their range to the FP32 product, which then computes these alone.  (A type of its
// own: one more member in FdkArgs made the compiler unroll fdk_filter_kernel's epilogue
// into half as much code again, the adjoint of 64 x 64 views 37 -> 44 us.)
struct FdkLeft : FdkArgs {
    const FdkRange* ranges = nullptr;  // [A][ceil(U/8)]
    explicit FdkLeft(const FdkArgs& p, const FdkRange* ranges_) : FdkArgs(p), ranges(ranges_) {}
};

// Whether the tensor cores' product of view a stands (all threads of the
// block ask).  A bf16 split holds FP32's range, but its lower parts and the products
// must stay clear of overflow and of the subnormals: of every value but zero, since a
// detector column whose values are all small has no larger one to hide its errors.
// Measured, white noise: columns of 2^-108 and more lose nothing (h[0] = 0.05), one of
// 2^-117 has 6 to 23 times the FP32 product's error, one of 2^-123 89 to 345 times (U
// = 2048 to 96).  A view with a NaN or an infinity, or that a wait gave up on,
// is out of range too.
__device__ __forceinline__ bool fdk_tc_holds(const FdkLeft& p, int a) {
    const int groups = (p.U + 7) >> 3;
    const float h = fabsf(p.taps[0]);
    bool out = !(h >= 1e-25f && h <= 1e35f);
    for (int i = threadIdx.x; i < groups; i += blockDim.x) {
        const FdkRange r = p.ranges[(long long)a * groups + i];
        const float high = __int_as_float(r.high);
        out = out || !(high <= 1e35f && high * h <= 1e35f);
        if (r.low != INT_MAX) {
            const float low = __int_as_float(r.low);
            out = out || !(low >= 1e-31f && low * h >= 1e-32f);
        }
    }
    return !__syncthreads_or(out);
}

constexpr int FBM = kFdkTileRows;     // output rows (U) per CTA
constexpr int FBN = kFdkTileColumns;  // output columns (V) per CTA
constexpr int FBK = 16;   // reduction slice

// ADJ = false: y = c H(w P) (the filter).  ADJ = true: its adjoint, z = H(g)
// for the upstream gradient g (H is symmetric), grad P = c w z, and per CTA
// the FP64 sums of g*y, z*P*dw/dD and (CG, the frame centre's gradients
// asked for) z*P*u_c/dist^3, z*P*v_c/dist^3 -- zeros without CG -- for the
// distance and centre gradients; c = pixel*sid/sod,
// w = D/dist the cosine weight with D the source's distance to the detector
// plane (sid unless a frame is given), u_c, v_c the pixel's offsets from the
// frame centre in length units, dist^2 = D^2 + u_c^2 + v_c^2, and
// dw/dD = (u_c^2 + v_c^2)/dist^3.
// Args = FdkLeft: only the views that the tensor cores' product does not hold.
template <bool ADJ, bool CG = false, class Args = FdkArgs>
__global__ void __launch_bounds__(256, 2) fdk_filter_kernel(Args p) {
    __shared__ __align__(16) float ws[FBK][FBN];
    __shared__ f32x2 gw2[FBM + FBK];  // taps, each duplicated into a packed pair
    __shared__ double s_part[8][kFdkPartials];
    const int a = blockIdx.z;
    if constexpr (std::is_same<Args, FdkLeft>::value) {
        if (fdk_tc_holds(p, a)) return;
    }
    const int m0 = blockIdx.y * FBM;
    const int n0 = blockIdx.x * FBN;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const float sid = p.sid[a], sod = p.sod[a];
    const float dn = p.frame_dist ? p.frame_dist[a] : sid;  // preweight distance D
    const float dn2 = dn * dn;
    const float* __restrict__ Pa = p.projections + (long long)a * p.U * p.V;
    const float* __restrict__ Ga = ADJ ? p.grad_filtered + (long long)a * p.U * p.V : nullptr;
    const float cu = p.frame_u ? p.frame_u[a] : 0.5f * (p.U - 1);
    const float cv = p.frame_v ? p.frame_v[a] : 0.5f * (p.V - 1);

    // 8 x 8 outputs per thread as packed pairs along v: one fma.rn.f32x2 per
    // two outputs (lane by lane the scalar FMA, in the same order)
    f32x2 acc2[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc2[i][j] = pack2(0.0f, 0.0f);

    for (int k0 = 0; k0 < p.U; k0 += FBK) {
        {   // stage the cosine-weighted input slice w[k0..k0+FBK) x [n0..n0+FBN)
            const int r = tid >> 4;
            const int k = k0 + r;
            const int c0 = (tid & 15) * 8;
            const float uu = ((float)k - cu) * p.pixel_size;
            const float wk = (p.uweight && k < p.U) ? p.uweight[(long long)a * p.U + k] : 1.0f;
            float vals[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int v = n0 + c0 + j;
                float val = 0.0f;
                if (k < p.U && v < p.V) {
                    if (ADJ) {
                        val = Ga[(long long)k * p.V + v];
                    } else {
                        const float vv = ((float)v - cv) * p.pixel_size;
                        const float dist = sqrtf(dn2 + uu * uu + vv * vv);
                        val = Pa[(long long)k * p.V + v] * (dn / dist) * wk;
                    }
                }
                vals[j] = val;
            }
            *reinterpret_cast<float4*>(&ws[r][c0]) = make_float4(vals[0], vals[1], vals[2], vals[3]);
            *reinterpret_cast<float4*>(&ws[r][c0 + 4]) = make_float4(vals[4], vals[5], vals[6], vals[7]);
        }
        // Toeplitz window: gw[i] = h[|m0 - k0 - (FBK-1) + i|]
        for (int i = tid; i < FBM + FBK - 1; i += 256) {
            int d = m0 - k0 - (FBK - 1) + i;
            d = d < 0 ? -d : d;
            const float h = p.taps[min(d, p.U - 1)];
            gw2[i] = pack2(h, h);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < FBK; ++kk) {
            // a thread's columns: tx*4..+3 and FBN/2 + tx*4..+3, so the 16 lanes of
            // a load read contiguous 16-byte chunks (no bank conflicts)
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&ws[kk][tx * 4]);
            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&ws[kk][FBN / 2 + tx * 4]);
            const f32x2 b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const f32x2 av = gw2[ty * 8 + i - kk + FBK - 1];
#pragma unroll
                for (int j = 0; j < 4; ++j) acc2[i][j] = fma2(av, b[j], acc2[i][j]);
            }
        }
        __syncthreads();
    }
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 e = unpack2(acc2[i][j]);
            acc[i][2 * j] = e.x;
            acc[i][2 * j + 1] = e.y;
        }
    // filtering.py:104: filtered * pixel_size * (sid / sod)
    const float ratio = sid / sod;
    if (!ADJ) {
        float* __restrict__ Oa = p.filtered + (long long)a * p.U * p.V;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int u = m0 + ty * 8 + i;
            if (u >= p.U) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int v = n0 + (j < 4 ? tx * 4 + j : FBN / 2 + tx * 4 + j - 4);
                if (v < p.V) Oa[(long long)u * p.V + v] = (acc[i][j] * p.pixel_size) * ratio;
            }
        }
        return;
    }
    // adjoint epilogue: acc = z = H(g) at (u, v)
    const long long base = (long long)a * p.U * p.V;
    double s_gy = 0.0, s_zpw = 0.0, s_zpu = 0.0, s_zpv = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int u = m0 + ty * 8 + i;
        if (u >= p.U) continue;
        const float uu = ((float)u - cu) * p.pixel_size;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int v = n0 + (j < 4 ? tx * 4 + j : FBN / 2 + tx * 4 + j - 4);
            if (v >= p.V) continue;
            const long long idx = (long long)u * p.V + v;
            const float vv = ((float)v - cv) * p.pixel_size;
            const float r2 = uu * uu + vv * vv;
            const float dist = sqrtf(dn2 + r2);
            const float z = acc[i][j];
            if (p.grad_projections)
                p.grad_projections[base + idx] = (z * p.pixel_size) * ratio * (dn / dist);
            if (p.partials) {
                const double zp = (double)z * (double)Pa[idx];
                const double d3 = (double)dist * dist * dist;
                s_gy += (double)Ga[idx] * (double)p.forward_out[base + idx];
                s_zpw += zp * ((double)r2 / d3);
                if (CG) {
                    s_zpu += zp * ((double)uu / d3);
                    s_zpv += zp * ((double)vv / d3);
                }
            }
        }
    }
    if (!p.partials) return;
    // CTA sums in a fixed order: warp shuffles, then the eight warps in turn
    constexpr int kSums = CG ? 4 : 2;  // sums this variant accumulates
    s_gy = warp_sum(s_gy);
    s_zpw = warp_sum(s_zpw);
    if (CG) {
        s_zpu = warp_sum(s_zpu);
        s_zpv = warp_sum(s_zpv);
    }
    const int lane = tid & 31, warp = tid >> 5;
    if (lane == 0) {
        s_part[warp][0] = s_gy;
        s_part[warp][1] = s_zpw;
        if (CG) {
            s_part[warp][2] = s_zpu;
            s_part[warp][3] = s_zpv;
        }
    }
    __syncthreads();
    if (tid < kFdkPartials) {
        double t = 0.0;
        if (tid < kSums)
            for (int w8 = 0; w8 < 8; ++w8) t += s_part[w8][tid];
        const long long tiles = (long long)gridDim.x * gridDim.y;
        const long long tile = (long long)blockIdx.y * gridDim.x + blockIdx.x;
        p.partials[((long long)a * tiles + tile) * kFdkPartials + tid] = t;
    }
}

}  // namespace dgc
