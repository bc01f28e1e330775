// backprojector.cu -- voxel-driven, FDK-weighted cone-beam backprojector and
// its hand-written backward, for sm_100a.
//
// Semantics follow the reference kernels of TomSHINING/diff-geoCali,
// csrc/src_cbct_backprojector_cuda.cu:
//   forward   15-98  : vol[z,y,x] = sum_a mask * ((sod+ds_n)/q)^2 * bilerp(P_a, u_idx, v_idx)
//   backward 101-295 : grad_proj (bilinear scatter) + d/d(sid, sod, beta, u0, v0, src_xyz)
//
// B200 design (not the reference's):
//   * A warp owns one (x, y) voxel column; its lanes walk Z (lane + 32k).  For a
//     fixed column and view, u_idx, the magnification t and the FDK weight do
//     not depend on z, and the lanes read one detector row pair at nearby V
//     positions (coalesced).
//   * Per-view trig and source terms are tabulated once per call; within a
//     warp, lane j evaluates the column geometry of view a0+j and the warp
//     broadcasts it (the forward through shared memory, the backward with
//     shuffles), so no lane recomputes it.
//   * Projections are re-laid out as quads PQ[a][u][v] = float4(P[u][v],
//     P[u+1][v], P[u][v+1], P[u+1][v+1]) -- two column pairs, so the lerp
//     along v runs as one packed f32x2 lerp over rows u and u+1: one 16-byte
//     load per voxel-view.
//   * Outputs go through a shared-memory transpose so the volume is written
//     along X (coalesced).
//   * The backward sums the per-voxel terms over Z in four accumulators and
//     applies the (column, view) chain-rule coefficients once per warp; the
//     eight per-view gradients are reduced in FP64 in a fixed order.
#include <climits>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "backprojector.cuh"

namespace dgc {

// ---------------------------------------------------------------------------
// Per-view table and projection re-layout
// ---------------------------------------------------------------------------

__device__ __forceinline__ ViewRow view_row(const Geometry& g, int a) {
    const float beta = g.angles[a];
    const float c = cosf(beta);
    const float s = sinf(beta);
    ViewRow r;
    r.c = c;
    r.s = s;
    // World-coordinate source offset in the rotating system (bp.cu:53-56).
    r.ds_u = g.src_x[a] * c + g.src_y[a] * s;
    r.ds_n = -g.src_x[a] * s + g.src_y[a] * c;
    r.ds_v = g.src_z[a];
    r.sod = g.sod[a];
    r.sid = g.sid[a];
    r.u0 = g.det_u0[a];
    r.v0 = g.det_v0[a];
    r.gather = 0;
    r.pad1 = r.pad2 = 0.0f;
    return r;
}

__global__ void bp_view_table_kernel(Geometry g, int A, ViewRow* __restrict__ vt) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a < A) vt[a] = view_row(g, a);
}

int bp_view_table(const Geometry& g, int A, ViewRow* vt, cudaStream_t s) {
    DGC_TRACE("bp_view_table", s);
    bp_view_table_kernel<<<ceil_div(A, 128), 128, 0, s>>>(g, A, vt);
    DGC_LAUNCH_CHECK("bp_view_table");
    return DGC_OK;
}

// Bound by the quads' stores.  A block (32, 8) fills 32 columns x 32 rows of a view,
// kQuadRows rows a thread with the row shared by two quads read once and all loads
// issued first; the only divisions are the block's.  720 x 768^2 1.77 -> 1.29 ms (1.31
// at the copy bandwidth), 360 x 384^2 220 -> 163 us, 200 x 187 x 161 26 -> 17 us against
// one quad a thread with 64-bit divisions for its place.
constexpr int kQuadRows = 4;

__global__ void __launch_bounds__(256) build_proj_quads_kernel(const float* __restrict__ P, int U,
                                                               int V, int tiles_v, int tiles_u,
                                                               float4* __restrict__ PQ) {
    const int QU = U - 1, QV = V - 1;
    int b = (int)blockIdx.x;
    const int v = (b % tiles_v) * 32 + (int)threadIdx.x;
    b /= tiles_v;
    const int u = (b % tiles_u) * 8 * kQuadRows + (int)threadIdx.y * kQuadRows;
    const int a = b / tiles_u;
    if (v >= QV || u >= QU) return;
    const float* __restrict__ row = P + ((long long)a * U + u) * V + v;
    float4* __restrict__ to = PQ + ((long long)a * QU + u) * QV + v;
    const int n = min(kQuadRows, QU - u);
    float x[kQuadRows + 1], y[kQuadRows + 1];
#pragma unroll
    for (int r = 0; r <= kQuadRows; ++r) {
        x[r] = r <= n ? __ldg(row + (long long)r * V) : 0.0f;
        y[r] = r <= n ? __ldg(row + (long long)r * V + 1) : 0.0f;
    }
#pragma unroll
    for (int r = 0; r < kQuadRows; ++r)
        if (r < n) to[(long long)r * QV] = make_float4(x[r], x[r + 1], y[r], y[r + 1]);
}

int build_proj_quads(const float* P, int A, int U, int V, float4* PQ, cudaStream_t s) {
    DGC_TRACE("build_proj_quads", s);
    const int tiles_v = ceil_div(V - 1, 32), tiles_u = ceil_div(U - 1, 8 * kQuadRows);
    const unsigned blocks = (unsigned)((long long)tiles_v * tiles_u * A);
    build_proj_quads_kernel<<<blocks, dim3(32, 8), 0, s>>>(P, U, V, tiles_v, tiles_u, PQ);
    DGC_LAUNCH_CHECK("build_proj_quads");
    return DGC_OK;
}

// ---------------------------------------------------------------------------
// Column geometry of one (x, y, view) (bp.cu:48-79)
// ---------------------------------------------------------------------------

struct ColumnView {
    bool valid;   // q, sid+ds_n > 1e-6 and 0 <= u_idx < U-1
    int row;      // quad-row index (a*(U-1) + u0)*(V-1)
    float t;      // magnification (sid+ds_n)/q
    float w;      // ((sod+ds_n)/q)^2
    float fu;     // u_idx - u0
    float ds_v;
    float v0;
};

template <bool PIXDIV>
__device__ __forceinline__ ColumnView column_view(const ViewRow& r, int a, float vx, float vy,
                                                  const BpArgs& p) {
    ColumnView cv;
    cv.valid = false;
    cv.row = 0;
    cv.t = cv.w = cv.fu = cv.ds_v = cv.v0 = 0.0f;
    const float px = vx * r.c + vy * r.s;
    const float py = -vx * r.s + vy * r.c;
    const float denom = r.sod + r.ds_n - py;
    const float sdn = r.sid + r.ds_n;
    if (!(denom > 1e-6f && sdn > 1e-6f)) return cv;
    const float t = sdn / denom;
    const float u_phys = r.ds_u + t * (px - r.ds_u);
    const float sw = (r.sod + r.ds_n) / denom;
    const float u_idx = PIXDIV ? div_by(u_phys, p.pixel_size, p.inv_pixel) + r.u0
                               : fmaf(u_phys, p.inv_pixel, r.u0);
    if (!(u_idx >= 0.0f && u_idx < (p.U - 1.0f))) return cv;
    const int ui = (int)floorf(u_idx);
    cv.valid = true;
    cv.row = (a * (p.U - 1) + ui) * (p.V - 1);
    cv.t = t;
    cv.w = sw * sw;
    cv.fu = u_idx - ui;
    cv.ds_v = r.ds_v;
    cv.v0 = r.v0;
    return cv;
}

// ---------------------------------------------------------------------------
// Block order
// ---------------------------------------------------------------------------

// Tile (tx, ty) and z block of a CTA from its linear index.  Every CTA loops
// over all views, so the projection data a CTA reads per view is re-read from
// DRAM by each wave of CTAs unless the CTAs in flight share it: they must
// cover a compact region of the volume, whose projections are small patches
// of each view (a strip of rows along the whole volume width projects onto
// whole detector rows).  Tiles are therefore taken z block by z block and,
// inside a z block, in super-tiles of sx x sy tiles (about 64 x 64 voxels,
// one wave of CTAs) ordered row by row; edge super-tiles are narrower.
struct BpTile {
    int tx, ty, zb;
};

__device__ __forceinline__ BpTile bp_tile(long long linear, int tiles_x, int tiles_y, int sx,
                                          int sy) {
    const long long layer = (long long)tiles_x * tiles_y;
    BpTile t;
    t.zb = (int)(linear / layer);
    const long long r = linear - (long long)t.zb * layer;
    const long long band_tiles = (long long)sy * tiles_x;
    const int band = (int)(r / band_tiles);
    const long long rb = r - band * band_tiles;
    const int rows = min(sy, tiles_y - band * sy);
    const int col = (int)(rb / ((long long)sx * rows));
    const int rc = (int)(rb - (long long)col * sx * rows);
    const int cols = min(sx, tiles_x - col * sx);
    t.ty = band * sy + rc / cols;
    t.tx = col * sx + rc % cols;
    return t;
}

__host__ __device__ __forceinline__ int bp_super(int cta) { return cta >= 64 ? 1 : 64 / cta; }

// ---------------------------------------------------------------------------
// Forward (backprojection) kernel
// ---------------------------------------------------------------------------

// A CTA owns a cta_x x cta_y patch of (x, y) columns, one warp per column
// (at most kBpMaxWarps warps), and 32*KZ voxels of each along z.
//
// What bounds it is the L1 pipe: the 32 quads of a warp's load, 16 bytes each and
// 1.67 quads apart at magnification 1.67, take 8.5 of its cycles (4 if they were
// contiguous), and two of three come from L2.  So the six values of a (column, view)
// are read from shared memory (two broadcasts; six shuffles were a quarter of that
// pipe's work at KZ = 2), and the loads of four taps (one view's at KZ = 4, two
// views' at KZ = 2, four views' at KZ = 1) are issued before the first of them is
// used.  KZ = 4 now runs at 9.2 L1 cycles per load.
//
// Register caps by z depth (launch bounds cannot express "seven 128-thread CTAs per
// SM"): 72 leave 28 warps per SM, and the four loads in flight with them; 64 (KZ = 4:
// 256^3 7.2 ms for 6.5, 512^3 26.3 for 24.3) serialise the loads, 80 leave 24 warps
// (6.6, 25.2).  KZ = 3 holds three loads in 64.  CTAs of 2 x 2 columns: of 4 x 2, 72
// registers leave only 24 warps (6.7, 25.6).
//
// Before (KZ = 2 above 32 slices, shuffles, one tap at a time, 8 x 1 columns) -> now:
// 256^3 / 360 x 384^2 7.40 -> 6.48 ms; 512^3 / 180 x 768^2 28.1 -> 24.3; 128^3 / 180 x
// 256^2 0.640 -> 0.521; 90 x 133 x 121 / 200 x 187 x 161 0.527 -> 0.372; 64^3 / 90 x
// 128^2 0.070 -> 0.056; 24 x 40 x 40 / 30 x 48^2 0.028 -> 0.020.
template <int KZ, bool PIXDIV, bool FDK>
__global__ void __maxnreg__(KZ == 3 ? 64 : KZ == 8 ? 96 : 72) bp_forward_kernel(BpArgs p) {
    constexpr int kViews = KZ == 1 ? 4 : KZ == 2 ? 2 : 1;
    constexpr int kDepth = KZ >= 4 ? 4 : KZ;
    extern __shared__ __align__(16) unsigned char bp_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cx = p.cta_x, cy = p.cta_y, nw = cx * cy;
    float4* s_line = reinterpret_cast<float4*>(bp_smem) + 32 * warp;
    float2* s_rest = reinterpret_cast<float2*>(bp_smem + 512 * nw) + 32 * warp;
    float (*s_out)[kBpMaxWarps + 1] = reinterpret_cast<float (*)[kBpMaxWarps + 1]>(bp_smem);
    const int tiles_x = (p.W + cx - 1) / cx, tiles_y = (p.H + cy - 1) / cy;
    const BpTile tile = bp_tile((long long)blockIdx.y * gridDim.x + blockIdx.x, tiles_x, tiles_y,
                                bp_super(cx), bp_super(cy));
    const int xb = tile.tx * cx, yb = tile.ty * cy;
    const int x = xb + warp % cx, y = yb + warp / cx;
    const int zbase = tile.zb * 32 * KZ;
    const unsigned FULL = 0xffffffffu;

    // FP32 sums of up to 8 views, added into FP64 totals: the FDK terms of a
    // voxel cancel over the views (filtered projections change sign), and a
    // running FP32 sum over hundreds of views loses 1e-5 to 1e-4 of the
    // result to that cancellation
    double acc[KZ];
    float part[KZ];
    float pz[KZ];
#pragma unroll
    for (int k = 0; k < KZ; ++k) {
        acc[k] = 0.0;
        part[k] = 0.0f;
        const int z = zbase + lane + 32 * k;
        pz[k] = (z - p.D * 0.5f) * p.voxel_size + p.off_z;
    }
    if (x < p.W && y < p.H) {
        const float vx = (x - p.W * 0.5f) * p.voxel_size + p.off_x;
        const float vy = (y - p.H * 0.5f) * p.voxel_size + p.off_y;
        const int zlimit = p.D - zbase - lane;  // k valid while 32k < zlimit
        // a tap is valid iff 0 <= v_idx < V-1, i.e. its floor (exact from the
        // magic-number split, which maps NaN, infinities and values beyond
        // 2^22 outside [0, V-2]) as an unsigned index is below V-1
        const uint32_t vcount = (uint32_t)max(p.V - 1, 0);
        constexpr int kPairs = (KZ + 1) / 2;
        f32x2 pz2[kPairs];
#pragma unroll
        for (int k = 0; k < kPairs; ++k) pz2[k] = pack2(pz[2 * k], pz[2 * k + 1 < KZ ? 2 * k + 1 : 2 * k]);
        const f32x2 ip2 = pack2(p.inv_pixel, p.inv_pixel);
        const f32x2 npix2 = pack2(-p.pixel_size, -p.pixel_size);
        const f32x2 magic2 = pack2(kFloorMagic, kFloorMagic);
        for (int a0 = 0; a0 < p.A; a0 += 32) {
            ColumnView mine;
            mine.valid = false;
            if (a0 + lane < p.A) mine = column_view<PIXDIV>(p.vt[a0 + lane], a0 + lane, vx, vy, p);
            const unsigned valid_mask = __ballot_sync(FULL, mine.valid);
            const int nv = min(32, p.A - a0);
            __syncwarp();  // the last 32 views' have been read
            if (mine.valid) {
                s_line[lane] = make_float4(mine.t, mine.ds_v, mine.v0, mine.w);
                s_rest[lane] = make_float2(mine.fu, __int_as_float(mine.row));
            }
            __syncwarp();
            // views in chunks of 8, each chunk's FP32 partial sums added into
            // the FP64 totals after it
            for (int jb = 0; jb < nv; jb += 8) {
                const int je = min(jb + 8, nv);
                for (int j = jb; j < je; j += kViews) {
                    if (!((valid_mask >> j) & ((1u << kViews) - 1u))) continue;
                    // the taps of kViews views and kDepth steps of z: all positions and
                    // loads first, then the interpolations
#pragma unroll
                    for (int kb = 0; kb < KZ; kb += kDepth) {
                        ulonglong2 q[kViews][kDepth];
                        float fv[kViews][kDepth], fu[kViews], w[kViews];
                        bool in[kViews][kDepth];
#pragma unroll
                        for (int i = 0; i < kViews; ++i) {
                            const float4 line = s_line[j + i];
                            const float2 rest = s_rest[j + i];
                            const bool valid = kViews == 1 || (valid_mask >> (j + i)) & 1u;
                            const f32x2 t2 = pack2(line.x, line.x), d2 = pack2(line.y, line.y);
                            const f32x2 o2 = pack2(line.z, line.z);
                            w[i] = line.w;
                            fu[i] = rest.x;
                            const ulonglong2* __restrict__ rq =
                                reinterpret_cast<const ulonglong2*>(p.pquads) + __float_as_int(rest.y);
#pragma unroll
                            for (int k = 0; k < kDepth; k += 2) {
                                const f32x2 vp = fma2(t2, sub2(pz2[(kb + k) / 2], d2), d2);
                                const f32x2 vx2 = PIXDIV ? add2(div_by2(vp, npix2, ip2), o2)
                                                         : fma2(vp, ip2, o2);
                                const f32x2 f2 = add2_rd(vx2, magic2);
                                const float2 f = unpack2(sub2(vx2, sub2(f2, magic2)));
                                const uint2 bits = unpack2_bits(f2);
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    if (k + h >= kDepth) break;
                                    const uint32_t vi = (h ? bits.y : bits.x) - kFloorMagicBits;
                                    const bool ok = valid && 32 * (kb + k + h) < zlimit && vi < vcount;
                                    in[i][k + h] = ok;
                                    fv[i][k + h] = h ? f.y : f.x;
                                    q[i][k + h] = make_ulonglong2(0, 0);
                                    if (ok) q[i][k + h] = __ldg(rq + vi);
                                }
                            }
                        }
#pragma unroll
                        for (int i = 0; i < kViews; ++i)
#pragma unroll
                            for (int k = 0; k < kDepth; ++k) {
                                const float2 e = unpack2(lerp2(q[i][k].x, q[i][k].y,
                                                               pack2(fv[i][k], fv[i][k])));
                                if (in[i][k])
                                    part[kb + k] = fmaf(w[i], lerpf(e.x, e.y, fu[i]), part[kb + k]);
                            }
                    }
                }
#pragma unroll
                for (int k = 0; k < KZ; ++k) {
                    acc[k] += (double)part[k];
                    part[k] = 0.0f;
                }
            }
        }
    }
    // Transpose through shared memory (the views' values are done with); write rows
    // along X.
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KZ; ++k) {
        float val = FDK ? (float)(acc[k] * (double)p.out_scale) : (float)acc[k];
        if (FDK) {
            if (p.clamp) val = val < 0.0f ? 0.0f : val;  // clamp_min(0); NaN propagates
        }
        s_out[lane + 32 * k][warp] = val;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * KZ * nw; i += 32 * nw) {
        const int zl = i / nw, w = i - zl * nw;
        const int z = zbase + zl, xx = xb + w % cx, yy = yb + w / cx;
        if (z < p.D && xx < p.W && yy < p.H)
            p.volume[((long long)z * p.H + yy) * p.W + xx] = s_out[zl][w];
    }
}

// ---------------------------------------------------------------------------
// Backward kernel
// ---------------------------------------------------------------------------

// Column geometry of one (x, y, view) for the backward (bp.cu:139-174; the
// u/v indices use 1/pixel) and what the chain rule of bp.cu:213-292 needs.
struct ColumnGrad {
    bool ok;
    int ui;
    float t, w, fu, inv_q, du, m, sdn, denom, py;
    float ds_u, ds_n, ds_v, v0, c, s;
};

__device__ __forceinline__ ColumnGrad column_grad(const ViewRow& r, float vx, float vy, bool col_ok,
                                                  const BpArgs& p) {
    ColumnGrad g;
    g.c = r.c;
    g.s = r.s;
    g.ds_u = r.ds_u;
    g.ds_n = r.ds_n;
    g.ds_v = r.ds_v;
    g.v0 = r.v0;
    g.ui = 0;
    g.t = g.w = g.fu = g.inv_q = g.du = g.m = 0.f;
    const float px = vx * r.c + vy * r.s;
    g.py = -vx * r.s + vy * r.c;
    g.denom = r.sod + r.ds_n - g.py;
    g.sdn = r.sid + r.ds_n;
    g.ok = col_ok && g.denom > 1e-6f && g.sdn > 1e-6f;
    if (g.ok) {
        g.inv_q = 1.0f / g.denom;
        g.t = g.sdn * g.inv_q;
        g.du = px - r.ds_u;
        const float u_phys = r.ds_u + g.t * g.du;
        g.m = r.sod + r.ds_n;
        g.w = g.m * g.m * (g.inv_q * g.inv_q);
        const float u_idx = u_phys * p.inv_pixel + r.u0;
        g.ok = u_idx >= 0.0f && u_idx < (p.U - 1.0f);
        if (g.ok) {
            g.ui = (int)floorf(u_idx);
            g.fu = u_idx - g.ui;
        }
    }
    return g;
}

// The eight per-view geometry gradients of a (column, view) from its four Z
// sums (s_iu = sum g*Iu, s_iv = sum g*Iv, s_ivdv = sum g*Iv*dv, s_int = sum
// g*interp): the chain-rule coefficients of bp.cu:213-292 applied once.
__device__ __forceinline__ void column_terms(const ColumnGrad& g, float s_iu, float s_iv,
                                             float s_ivdv, float s_int, float ip,
                                             float (&terms)[8]) {
    const float inv_q2 = g.inv_q * g.inv_q, inv_q3 = inv_q2 * g.inv_q;
    const float m2 = g.m * g.m;
    const float b_sid = g.du * s_iu + s_ivdv;
    terms[1] = g.w * g.inv_q * ip * b_sid;
    const float dt_sod = -g.sdn * inv_q2;
    const float dw_sod = 2.0f * g.m * inv_q2 - 2.0f * m2 * inv_q3;
    terms[2] = dw_sod * s_int + g.w * ip * dt_sod * b_sid;
    const float dsu_b = g.ds_n, dsn_b = -g.ds_u, dq_b = g.du;
    const float dt_b = (dsn_b * g.denom - g.sdn * dq_b) * inv_q2;
    const float du_b = (1.0f - g.t) * dsu_b + g.t * g.py + g.du * dt_b;
    const float dw_b = 2.0f * g.m * inv_q2 * dsn_b - 2.0f * m2 * inv_q3 * dq_b;
    terms[0] = dw_b * s_int + g.w * ip * (du_b * s_iu + dt_b * s_ivdv);
    terms[3] = g.w * s_iu;
    terms[4] = g.w * s_iv;
    const float dsu_x = g.c, dsn_x = -g.s;
    const float dt_x = dsn_x * (g.denom - g.sdn) * inv_q2;
    const float du_x = (1.0f - g.t) * dsu_x + g.du * dt_x;
    const float dw_x = 2.0f * g.m * inv_q2 * dsn_x - 2.0f * m2 * inv_q3 * dsn_x;
    terms[5] = dw_x * s_int + g.w * ip * (du_x * s_iu + dt_x * s_ivdv);
    const float dsu_y = g.s, dsn_y = g.c;
    const float dt_y = dsn_y * (g.denom - g.sdn) * inv_q2;
    const float du_y = (1.0f - g.t) * dsu_y + g.du * dt_y;
    const float dw_y = 2.0f * g.m * inv_q2 * dsn_y - 2.0f * m2 * inv_q3 * dsn_y;
    terms[6] = dw_y * s_int + g.w * ip * (du_y * s_iu + dt_y * s_ivdv);
    terms[7] = g.w * (1.0f - g.t) * ip * s_iv;
}

// Sums of N (16 or 32) per-lane values over the warp, lane L receiving the
// sum of value L mod N: log2(N) butterfly steps, each halving the values a
// lane holds (N-1 shuffles for the N sums instead of 5 per sum), then the
// halves of the warp added.
template <int N>
__device__ __forceinline__ float warp_transpose_sum(float (&v)[N], int lane) {
    const unsigned FULL = 0xffffffffu;
#pragma unroll
    for (int h = N / 2; h >= 1; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float send = up ? v[k] : v[k + h];
            const float keep = up ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(FULL, send, h);
        }
    }
    float x = v[0];
#pragma unroll
    for (int o = N; o < 32; o <<= 1) x += __shfl_xor_sync(FULL, x, o);
    return x;
}

// Views whose four z-sums are reduced together (16 accumulators per lane).
constexpr int kBpGroup = 4;

// GP: projection gradient 0 = not computed (p.grad_projections null), 1 = four
// float reductions per voxel-view into grad_projections.  GEO: the geometry
// gradients (without them the projections are not read).
//
// A warp owns one (x, y) column and 32*KZ of its voxels along z.  Views go in
// passes of 32: lane j evaluates the column geometry of view a0+j (and, at
// the end of the pass, its chain rule).  The warp walks the pass's views
// kBpGroup at a time with that view's geometry broadcast by shuffles; per
// view every lane first issues the loads of its KZ taps together (an
// out-of-range tap loads the row's first quad and is masked), then adds its
// voxels' four products into registers.  The group's 4 x kBpGroup sums are
// reduced over the warp at once (warp_transpose_sum) and kept by the lane
// that owns the view; after the pass all 32 lanes apply the chain rule at
// once.
template <int KZ, int GP, bool GEO>
__global__ void __launch_bounds__(256) bp_backward_kernel(BpArgs p) {
    constexpr int G = kBpGroup;
    __shared__ double s_terms[GEO ? 8 : 1][32][8];
    if (p.only_if >= 0 && p.vt[0].gather != p.only_if) return;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cols_x = (p.W + 7) >> 3;
    const long long block_id = (long long)blockIdx.y * gridDim.x + blockIdx.x;
    const BpTile tile = bp_tile(block_id, cols_x, p.H, bp_super(8), bp_super(1));
    const int y = tile.ty;
    const int x = tile.tx * 8 + warp;
    const int zbase = tile.zb * 32 * KZ;
    const long long nblocks = (long long)gridDim.x * gridDim.y;
    const bool col_ok = x < p.W;
    const float vx = (x - p.W * 0.5f) * p.voxel_size + p.off_x;
    const float vy = (y - p.H * 0.5f) * p.voxel_size + p.off_y;
    const float ip = p.inv_pixel;

    float gval[KZ], pz[KZ];
#pragma unroll
    for (int k = 0; k < KZ; ++k) {
        const int z = zbase + lane + 32 * k;
        pz[k] = (z - p.D * 0.5f) * p.voxel_size + p.off_z;
        gval[k] = (col_ok && z < p.D) ? p.grad_volume[((long long)z * p.H + y) * p.W + x] : 0.0f;
    }
    const int zlimit = p.D - zbase - lane;
    const uint32_t vcount = (uint32_t)max(p.V - 1, 0);
    f32x2 pz2[KZ / 2 > 0 ? KZ / 2 : 1];
#pragma unroll
    for (int k = 0; k + 1 < KZ; k += 2) pz2[k / 2] = pack2(pz[k], pz[k + 1]);
    const f32x2 ip2 = pack2(p.inv_pixel, p.inv_pixel);
    const f32x2 magic2 = pack2(kFloorMagic, kFloorMagic);

    for (int a0 = 0; a0 < p.A; a0 += 32) {
        const int nv = min(32, p.A - a0);
        // the values the z loop needs from lane j's view (the rest of its
        // geometry is recomputed by the same lane for the chain rule)
        float my_t = 0.f, my_dsv = 0.f, my_v0 = 0.f, my_fu = 0.f, my_w = 0.f;
        int my_ui = 0;
        bool my_ok = false;
        if (lane < nv) {
            const ColumnGrad g = column_grad(p.vt[a0 + lane], vx, vy, col_ok, p);
            my_ok = g.ok;
            my_t = g.t;
            my_dsv = g.ds_v;
            my_v0 = g.v0;
            my_fu = g.fu;
            my_w = g.w;
            my_ui = g.ui;
        }
        const unsigned valid_mask = __ballot_sync(FULL, my_ok);
        // this lane's view: its four z-sums over the warp's voxels
        float m_iu = 0.f, m_iv = 0.f, m_ivdv = 0.f, m_int = 0.f;
        for (int b = 0; b < nv; b += G) {
            float acc[4 * G];
#pragma unroll
            for (int i = 0; i < 4 * G; ++i) acc[i] = 0.0f;
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const int j = b + i;
                if (!((valid_mask >> j) & 1u)) continue;  // warp-uniform
                const float t = __shfl_sync(FULL, my_t, j);
                const float dsv = __shfl_sync(FULL, my_dsv, j);
                const float v0 = __shfl_sync(FULL, my_v0, j);
                const float fu = __shfl_sync(FULL, my_fu, j);
                const int ui = __shfl_sync(FULL, my_ui, j);
                const int a = a0 + j;
                const ulonglong2* __restrict__ rq =
                    reinterpret_cast<const ulonglong2*>(p.pquads) + (a * (p.U - 1) + ui) * (p.V - 1);
                float w = 0.0f;
                float* __restrict__ gp = nullptr;
                if (GP) {
                    w = __shfl_sync(FULL, my_w, j);
                    gp = p.grad_projections + ((long long)a * p.U + ui) * p.V;
                }
                ulonglong2 q[KZ];
                float fvk[KZ], dvk[KZ];
                int vik[KZ];
                bool okk[KZ];
                // z voxels in pairs: v_idx and its floor split as packed f32x2;
                // a tap is valid iff its floor, as an unsigned index, is below V-1
                auto setup = [&](int k, float dv, uint32_t biased, float fv) {
                    const uint32_t vi = biased - kFloorMagicBits;
                    okk[k] = 32 * k < zlimit && vi < vcount;
                    vik[k] = okk[k] ? (int)vi : 0;
                    fvk[k] = fv;
                    dvk[k] = dv;
                    if (GEO) q[k] = __ldg(rq + vik[k]);
                };
                if constexpr (KZ % 2 == 0) {
                    const f32x2 t2 = pack2(t, t), d2 = pack2(dsv, dsv), o2 = pack2(v0, v0);
#pragma unroll
                    for (int k = 0; k < KZ; k += 2) {
                        const f32x2 dv2 = sub2(pz2[k / 2], d2);
                        const f32x2 vx2 = fma2(fma2(t2, dv2, d2), ip2, o2);
                        const f32x2 f2 = add2_rd(vx2, magic2);
                        const float2 fr = unpack2(sub2(vx2, sub2(f2, magic2)));
                        const uint2 bits = unpack2_bits(f2);
                        const float2 dv = unpack2(dv2);
                        setup(k, dv.x, bits.x, fr.x);
                        setup(k + 1, dv.y, bits.y, fr.y);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < KZ; ++k) {
                        const float dv = pz[k] - dsv;
                        const float v_phys = dsv + t * dv;
                        const FloorSplit fs = floor_split(v_phys * ip + v0);
                        setup(k, dv, fs.biased, fs.frac);
                    }
                }
#pragma unroll
                for (int k = 0; k < KZ; ++k) {
                    if (okk[k]) {
                        const float fv = fvk[k], dv = dvk[k];
                        const int vi = vik[k];
                        const float g = gval[k];
                        if (GEO) {
                        // column pairs (rows u, u+1) at v and v+1: the lerp along v
                        // and the difference along v as packed pairs
                        const float2 e = unpack2(lerp2(q[k].x, q[k].y, pack2(fv, fv)));
                        const float2 d = unpack2(sub2(q[k].y, q[k].x));
                        const float2 c0 = unpack2(q[k].x), c1 = unpack2(q[k].y);
                        const float interp = lerpf(e.x, e.y, fu);
                        const float iu = lerpf(c0.y - c0.x, c1.y - c1.x, fv);
                        const float iv = lerpf(d.x, d.y, fu);
                        acc[4 * i + 0] = fmaf(g, iu, acc[4 * i + 0]);
                        acc[4 * i + 1] = fmaf(g, iv, acc[4 * i + 1]);
                        acc[4 * i + 2] = fmaf(g * iv, dv, acc[4 * i + 2]);
                        acc[4 * i + 3] = fmaf(g, interp, acc[4 * i + 3]);
                        }
                        if (GP) {
                            const float gb = g * w;
                            const float g0 = gb * (1.0f - fu), g1 = gb * fu;
                            red_add_global(gp + vi, g0 * (1.0f - fv));
                            red_add_global(gp + p.V + vi, g1 * (1.0f - fv));
                            red_add_global(gp + vi + 1, g0 * fv);
                            red_add_global(gp + p.V + vi + 1, g1 * fv);
                        }
                    }
                }
            }
            if (!GEO) continue;
            // lane 4i+q: sum q of view b+i; the view's owner (lane b+i) keeps its four
            const float total = warp_transpose_sum<4 * G>(acc, lane);
            const int src = 4 * ((lane - b) & (G - 1));
            const float s_iu = __shfl_sync(FULL, total, src + 0);
            const float s_iv = __shfl_sync(FULL, total, src + 1);
            const float s_ivdv = __shfl_sync(FULL, total, src + 2);
            const float s_int = __shfl_sync(FULL, total, src + 3);
            if (lane >= b && lane < b + G) {
                m_iu = s_iu;
                m_iv = s_iv;
                m_ivdv = s_ivdv;
                m_int = s_int;
            }
        }
        if (!GEO) continue;
        float terms[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (my_ok) {
            const ColumnGrad g = column_grad(p.vt[a0 + lane], vx, vy, col_ok, p);
            column_terms(g, m_iu, m_iv, m_ivdv, m_int, ip, terms);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) s_terms[warp][lane][k] = (double)terms[k];
        __syncthreads();
        {
            const int j = threadIdx.x >> 3, k = threadIdx.x & 7;
            if (j < nv) {
                double acc = 0.0;
#pragma unroll
                for (int w = 0; w < 8; ++w) acc += s_terms[w][j][k];
                p.partials[((long long)(a0 + j) * 8 + k) * nblocks + block_id] = acc;
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) bp_reduce_partials_kernel(const double* __restrict__ partials,
                                                                 long long nblocks, GeometryGrad out) {
    const int a = blockIdx.x;
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* src = partials + ((long long)a * 8 + k) * nblocks;
    double acc = 0.0;
    for (long long i = lane; i < nblocks; i += 32) acc += src[i];
    acc = warp_sum(acc);
    if (lane == 0) out.g[k][a] = (float)acc;
}

// ---------------------------------------------------------------------------
// Projection gradient as a gather
// ---------------------------------------------------------------------------
//
// grad P[a,u,v] = sum over columns (x, y) and z of g w hat(u - u_idx) hat(v - v_idx),
// the adjoint of the bilinear taps.  Scattering it costs four float reductions
// per voxel-view, which bound that kernel (1.0-1.4e12 additions/s in L2).  Here a
// CTA takes a few detector bins b (u_idx in [b, b+1)) of one view and lists, bin
// by bin, the columns that project into it: those between the rays of the bin's
// two edges, found per row of the volume from the rays' equations with a margin
// and then tested exactly, so that every column falls into the bin its own FP32
// u_idx says.  A thread owns detector pixels v: per listed column it gathers the
// two voxels whose v_idx can lie within a pixel of v (more where a voxel is
// finer than a pixel), weights them by that v_idx, the backprojection's own, and
// adds the sum to rows u = b and b + 1 in registers.  Only a CTA's first and last
// row meet another CTA's: two additions onto zero, so the result does not
// depend on scheduling.
//
// Bound by issue (73 % of the slots): 30 instructions a column and pixel, the
// listing among them 2 %.

// Upstream volume as z-fastest columns, zeros around them:
// G[(y*W + x)*(D+3) + z + 1], z in [-1, D+1].
// grid: x = ceil(W/32) * H, y = ceil((D+3)/32); block (32, 8)
__global__ void __launch_bounds__(256) bp_columns_kernel(const float* __restrict__ g, int D, int H,
                                                         int W, const ViewRow* __restrict__ vt,
                                                         float* __restrict__ G) {
    __shared__ float tile[32][33];
    if (!vt[0].gather) return;
    const int xtiles = (W + 31) / 32;
    const int y = blockIdx.x / xtiles;
    const int x0 = (blockIdx.x - y * xtiles) * 32, z0 = blockIdx.y * 32 - 1;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int zl = ty; zl < 32; zl += 8) {
        const int z = z0 + zl, x = x0 + tx;
        tile[zl][tx] = (z >= 0 && z < D && x < W) ? __ldg(g + ((long long)z * H + y) * W + x) : 0.0f;
    }
    __syncthreads();
    for (int xl = ty; xl < 32; xl += 8) {
        const int x = x0 + xl, zp = z0 + 1 + tx;
        if (x < W && zp < D + 3) G[((long long)y * W + x) * (D + 3) + zp] = tile[tx][xl];
    }
}

constexpr int kAdjMaxWarps = 8;
constexpr int kAdjList = 96;  // columns that a warp lists between two passes over them

struct AdjColumn {
    float t, rt;   // magnification; d(z index)/d(v_phys - ds_v)
    float wa, wb;  // FDK weight times the bilinear weights of rows b and b + 1
};

// Where the ray of detector coordinate q = u_phys - ds_u crosses the rows of a
// volume axis, as a line over the row index: voxel coordinate e0 + e1*row, and
// the source's distance along the view's normal there, d0 + d1*row.  along_y:
// rows are y and the coordinate x, else the other way round.
struct AdjLine {
    float e0, e1, d0, d1;
};

__device__ __forceinline__ AdjLine adj_line(const ViewRow& r, float q, bool along_y, const BpArgs& p) {
    const float sdn = r.sid + r.ds_n, m = r.sod + r.ds_n;
    // w = alpha + beta*o solves u_phys = ds_u + sdn/denom*(px - ds_u) at row coordinate o
    const float k = 1.0f / (along_y ? q * r.s - sdn * r.c : q * r.c + sdn * r.s);
    const float alpha = (along_y ? -sdn * r.ds_u - q * m : q * m + sdn * r.ds_u) * k;
    const float beta = (along_y ? sdn * r.s + q * r.c : q * r.s - sdn * r.c) * k;
    const int rows = along_y ? p.H : p.W, cross = along_y ? p.W : p.H;
    const float off_o = along_y ? p.off_y : p.off_x, off_i = along_y ? p.off_x : p.off_y;
    const float o0 = off_o - rows * 0.5f * p.voxel_size;  // row 0
    const float w0 = alpha + beta * o0;
    AdjLine l;
    l.e0 = (w0 - off_i) / p.voxel_size + cross * 0.5f;
    l.e1 = beta;
    l.d0 = along_y ? m + w0 * r.s - o0 * r.c : m + o0 * r.s - w0 * r.c;
    l.d1 = (along_y ? beta * r.s - r.c : r.s - beta * r.c) * p.voxel_size;
    return l;
}

// The volume's corner columns: distance of one along the view's normal.
__device__ __forceinline__ float corner_distance(const ViewRow& r, const BpArgs& p, int c) {
    const float x = ((c & 1 ? p.W - 1 : 0) - p.W * 0.5f) * p.voxel_size + p.off_x;
    const float y = ((c & 2 ? p.H - 1 : 0) - p.H * 0.5f) * p.voxel_size + p.off_y;
    return r.sod + r.ds_n + x * r.s - y * r.c;
}

// First and last detector row that the volume can reach, with a margin, from its
// four corners' magnifications (all rows if a corner is not in front of the source).
__device__ __forceinline__ float2 adj_reach(const ViewRow& r, const BpArgs& p) {
    const float sdn = r.sid + r.ds_n;
    float tlo = FLT_MAX, thi = -FLT_MAX;
    bool front = true;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float denom = corner_distance(r, p, c);
        front = front && denom > 1e-3f * fabsf(r.sod);
        tlo = fminf(tlo, sdn / denom);
        thi = fmaxf(thi, sdn / denom);
    }
    const float za = -p.D * 0.5f * p.voxel_size + p.off_z - r.ds_v;
    const float zb = za + (p.D - 1) * p.voxel_size;
    const float lo = fminf(tlo * za, thi * za), hi = fmaxf(tlo * zb, thi * zb);
    return front ? make_float2((r.ds_v + lo) * p.inv_pixel + r.v0 - 2.0f,
                               (r.ds_v + hi) * p.inv_pixel + r.v0 + 2.0f)
                 : make_float2(-FLT_MAX, FLT_MAX);
}

// The view table, and in its rows whether every view is one for the gather.  With s a
// voxel's height in pixels: 1 or more in the farthest corner (below, a pixel has more
// than two voxels and the general sum runs: 1.6-3 times the scatter's time at
// 1.1-fold magnification), at most 5 in the middle (a column's pixels are mostly
// between two voxels: 1.1-1.8 times at 6-8), and a detector that the volume's shadow
// fills to `fill` (else the pixels beside it idle).  bp_may_gather has the
// measurements.  One block: a scan has hundreds of views.
__global__ void __launch_bounds__(256) bp_view_choice_kernel(Geometry g, BpArgs p, float fill,
                                                             ViewRow* __restrict__ vt) {
    bool ok = true;
    for (int a = threadIdx.x; a < p.A; a += 256) {
        const ViewRow r = view_row(g, a);
        vt[a] = r;
        float lo = FLT_MAX, hi = -FLT_MAX;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float d = corner_distance(r, p, c);
            lo = fminf(lo, d);
            hi = fmaxf(hi, d);
        }
        const float height = (r.sid + r.ds_n) * (p.voxel_size * p.inv_pixel);
        const float middle = 2.0f * height / (lo + hi);
        ok = ok && lo > 1e-3f * fabsf(r.sod) && height / hi >= 1.0001f && middle <= 5.0f &&
             p.D * middle >= fill * p.V;
    }
    ok = __syncthreads_and(ok);
    for (int a = threadIdx.x; a < p.A; a += 256) vt[a].gather = ok;
}

// Work item: `bins` bins of one view, one tile of V; NV pixels a thread, a warp's
// 32*NV of them contiguous.  Dynamic shared memory: the warps' lists.
template <int NV>
__global__ void __launch_bounds__(32 * kAdjMaxWarps, NV < 3 ? 4 : 3)
    bp_adjoint_kernel(BpArgs p, const float* __restrict__ G, int bins, int bin_blocks, int tiles) {
    extern __shared__ AdjColumn s_col[];  // [warps][kAdjList]
    __shared__ int s_count[kAdjMaxWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int warps = blockDim.x >> 5;
    unsigned* s_off = reinterpret_cast<unsigned*>(s_col + warps * kAdjList);
    const int tile = blockIdx.x % tiles;
    const int block = blockIdx.x / tiles;
    const int a = block / bin_blocks;
    const int b0 = (block - a * bin_blocks) * bins;
    // no bins where the views chose the scatter (returning here instead took 7 % of the
    // kernel's time: the compiler then allocates the loop's registers otherwise)
    const int b1 = p.vt[a].gather ? min(b0 + bins, p.U - 1) : b0;
    const ViewRow r = p.vt[a];
    const float vox = p.voxel_size;

    // this thread's detector pixels and their heights above the source
    float vf[NV], vp[NV], acc_a[NV], acc_b[NV];
    // the bilinear weight of a voxel at distance d from a pixel, as min(1 + below*d,
    // above0 - above*d) limited to [0, 1]: a tap exists for 0 <= v_idx < V-1 only, so
    // pixel 0 has no voxels below it, pixel V-1 none at or above it and pixels past
    // the detector none
    float below[NV], above[NV], above0[NV];
    const int v_first = (tile * warps + warp) * NV * 32 + lane;
    bool inner = true;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int v = v_first + 32 * j;
        vf[j] = (float)v;
        vp[j] = (vf[j] - r.v0) * p.pixel_size - r.ds_v;
        below[j] = v == 0 ? 1e30f : 1.0f;
        above[j] = v == p.V - 1 ? 1e30f : v >= p.V ? 0.0f : 1.0f;
        above0[j] = v >= p.V - 1 ? 0.0f : 1.0f;
        inner = inner && v > 0 && v < p.V - 1;
        acc_b[j] = 0.0f;
    }
    inner = __all_sync(0xffffffffu, inner);
    const float2 reach_v = adj_reach(r, p);
    // a warp whose pixels the volume cannot reach only lists
    const bool reached = (float)(v_first - lane + 32 * NV) >= reach_v.x &&
                         (float)(v_first - lane) <= reach_v.y;
    const auto weight = [&](int j, float d) {
        return fminf(__saturatef(fmaf(d, below[j], 1.0f)),
                     __saturatef(fmaf(d, -above[j], above0[j])));
    };
    const float half_z = p.D * 0.5f;
    const float zc = (r.ds_v - p.off_z) / vox + half_z;

    // The listed columns' contributions to rows b (acc_a) and b + 1 (acc_b), where
    // every voxel is at least a pixel high: the voxels within a pixel of v are
    // z0, the floor of the pixel's own z, and z0 + 1.  EDGE: some pixel of the
    // warp is at the detector's edge or past it.
    const f32x2 vox2 = pack2(vox, vox), off2 = pack2(p.off_z, p.off_z);
    const f32x2 dsv2 = pack2(r.ds_v, r.ds_v), ip2 = pack2(p.inv_pixel, p.inv_pixel);
    const f32x2 v02 = pack2(r.v0, r.v0);
    auto sum_list = [&](const AdjColumn* cols, const unsigned* offs, int count, auto edge) {
        constexpr bool EDGE = decltype(edge)::value;
        const unsigned top = (unsigned)p.D + 1u;
#pragma unroll 2
        for (int i = 0; i < count; ++i) {
            const AdjColumn col = cols[i];
            const float* __restrict__ g = G + offs[i] * (unsigned long long)(p.D + 3);
            const f32x2 t2 = pack2(col.t, col.t);
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const float f = __fadd_rd(fmaf(vp[j], col.rt, zc), kFloorMagic);
                // pixels beyond the column (any bit pattern) read its zeros
                const unsigned zi = min(__float_as_uint(f) - (kFloorMagicBits - 1u), top);
                const float ga = __ldg(g + zi), gb = __ldg(g + zi + 1);
                const float z0 = __fsub_rn(f, kFloorMagic) - half_z;
                // v_idx of the two voxels, the backprojection's arithmetic
                const f32x2 dv = sub2(fma2(pack2(z0, z0 + 1.0f), vox2, off2), dsv2);
                const f32x2 vi = fma2(fma2(t2, dv, dsv2), ip2, v02);
                const float2 d = unpack2(sub2(vi, pack2(vf[j], vf[j])));
                const float ka = EDGE ? weight(j, d.x) : __saturatef(1.0f - fabsf(d.x));
                const float kb = EDGE ? weight(j, d.y) : __saturatef(1.0f - fabsf(d.y));
                const float h = fmaf(kb, gb, ka * ga);
                acc_a[j] = fmaf(col.wa, h, acc_a[j]);
                acc_b[j] = fmaf(col.wb, h, acc_b[j]);
            }
        }
    };
    // The same for any pixel and voxel size; a voxel out of reach contributes
    // nothing even if it is not finite.
    auto sum_list_general = [&](const AdjColumn* cols, const unsigned* offs, int count) {
#pragma unroll 1
        for (int i = 0; i < count; ++i) {
            const AdjColumn col = cols[i];
            const float* __restrict__ g = G + offs[i] * (unsigned long long)(p.D + 3) + 1;
            const float reach = 1.0f / (col.t * (vox * p.inv_pixel)) + 1.0f;
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const float zf = fmaf(vp[j], col.rt, zc);
                const int z_lo = (int)fmaxf(ceilf(zf - reach), 0.0f);
                const int z_hi = (int)fminf(floorf(zf + reach), (float)(p.D - 1));
                float h = 0.0f;
#pragma unroll 1
                for (int z = z_lo; z <= z_hi; ++z) {
                    const float dv = fmaf(z - half_z, vox, p.off_z) - r.ds_v;
                    const float d = fmaf(fmaf(col.t, dv, r.ds_v), p.inv_pixel, r.v0) - vf[j];
                    const float k = weight(j, d);
                    if (k > 0.0f) h = fmaf(k, __ldg(g + z), h);
                }
                acc_a[j] = fmaf(col.wa, h, acc_a[j]);
                acc_b[j] = fmaf(col.wb, h, acc_b[j]);
            }
        }
    };

    const float sdn = r.sid + r.ds_n;
    const float front = 1e-3f * fabsf(r.sod);
    const float rt_scale = 1.0f / (sdn * vox);
    float* __restrict__ out = p.grad_projections + (long long)a * p.U * p.V;
    for (int b = b0; b < b1; ++b) {
        // row b starts with what the bin before it left
        float from[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) from[j] = acc_b[j];
        // rows of the volume along the axis that the bin's rays run along more
        const float q0 = ((float)b - r.u0) * p.pixel_size - r.ds_u;
        const float q1 = ((float)(b + 1) - r.u0) * p.pixel_size - r.ds_u;
        const float qm = 0.5f * (q0 + q1);
        const bool along_y = fabsf(qm * r.s - sdn * r.c) >= fabsf(qm * r.c + sdn * r.s);
        const int n_rows = along_y ? p.H : p.W, n_cross = along_y ? p.W : p.H;
        const AdjLine l0 = adj_line(r, q0, along_y, p), l1 = adj_line(r, q1, along_y, p);
        const float margin = 0.02f + 1e-5f * n_cross;
        // a second time, voxel by voxel, if a sum is not finite: the first lets
        // a voxel that is not finite reach pixels whose weight for it is zero
        for (int careful = 0;; ++careful) {
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                acc_a[j] = from[j];
                acc_b[j] = 0.0f;
            }
            for (int row0 = 0; row0 < n_rows; row0 += blockDim.x) {
                const int row = row0 + tid;
                int i = 0, i_end = 0;
                if (row < n_rows) {
                    // both crossings in front of the source: the columns between
                    // them; otherwise (or not finite) the whole row is tested
                    i_end = n_cross;
                    const float e0 = fmaf(l0.e1, (float)row, l0.e0);
                    const float e1 = fmaf(l1.e1, (float)row, l1.e0);
                    if (fmaf(l0.d1, (float)row, l0.d0) > front &&
                        fmaf(l1.d1, (float)row, l1.d0) > front && fabsf(e0) < 1e9f &&
                        fabsf(e1) < 1e9f) {
                        i = (int)fmaxf(ceilf(fminf(e0, e1) - margin), 0.0f);
                        i_end = (int)fminf(floorf(fmaxf(e0, e1) + margin) + 1.0f, (float)n_cross);
                    }
                }
                // every warp lists its rows' columns in its own list, in order; all
                // lists are summed when every warp is through or has a full one
                bool more;
                do {
                    int count = 0;
                    bool fine = false;  // a listed voxel is less than a pixel high
                    while (count <= kAdjList - 32 && __any_sync(0xffffffffu, i < i_end)) {
                        bool take = false;
                        AdjColumn col;
                        unsigned off = 0;
                        if (i < i_end) {
                            const int x = along_y ? i : row, y = along_y ? row : i;
                            const float vx = (x - p.W * 0.5f) * vox + p.off_x;
                            const float vy = (y - p.H * 0.5f) * vox + p.off_y;
                            const ColumnGrad cg = column_grad(r, vx, vy, true, p);
                            take = cg.ok && cg.ui == b;
                            col.t = cg.t;
                            col.rt = cg.denom * rt_scale;
                            col.wa = cg.w * (1.0f - cg.fu);
                            col.wb = cg.w * cg.fu;
                            off = (unsigned)(y * (long long)p.W + x);
                            fine = fine || (take && cg.t * (vox * p.inv_pixel) < 1.0001f);
                            ++i;
                        }
                        const unsigned mask = __ballot_sync(0xffffffffu, take);
                        if (take) {
                            const int at =
                                warp * kAdjList + count + __popc(mask & ((1u << lane) - 1u));
                            s_col[at] = col;
                            s_off[at] = off;
                        }
                        count += __popc(mask);
                    }
                    if (lane == 0) s_count[warp] = count;
                    more = __syncthreads_or(i < i_end);
                    fine = __syncthreads_or(fine);
                    if (reached) {
                        for (int list = 0; list < warps; ++list) {
                            const AdjColumn* cols = s_col + list * kAdjList;
                            const unsigned* offs = s_off + list * kAdjList;
                            const int n = s_count[list];
                            if (fine || careful) sum_list_general(cols, offs, n);
                            else if (inner) sum_list(cols, offs, n, std::false_type());
                            else sum_list(cols, offs, n, std::true_type());
                        }
                    }
                    __syncthreads();
                } while (more);
            }
            bool bad = false;
#pragma unroll
            for (int j = 0; j < NV; ++j) bad = bad || !isfinite(acc_a[j]) || !isfinite(acc_b[j]);
            if (!__syncthreads_or(bad && !careful)) break;
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int v = v_first + 32 * j;
            if (v < p.V) {
                float* o = out + (long long)b * p.V + v;
                if (b == b0) red_add_global(o, acc_a[j]);  // the CTA before adds its last row
                else *o = acc_a[j];
                if (b == b1 - 1) red_add_global(o + p.V, acc_b[j]);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------

// Z values per lane: a warp covers 32*KZ voxels of a column.  Fewer keep the projection
// rows that a CTA reads per view short, so that they stay in L1; more amortise the
// per-(column, view) geometry.  The forward's choice is bp_forward_tile's.  Backward at
// 256^3 / 360 x 384^2, 8 columns a CTA, KZ = 2 / 4 / 8: 12.6 / 10.5 / 10.9 ms without the
// projection gradient, 22.9 / 25.1 / 28.7 ms with it.

// Tile rules registered by the autotuner (dgc_bp_add_tile_rule): the first
// rule with D <= d_max and A <= a_max applies; a zero field keeps the
// built-in choice.
namespace {
struct BpTileRule {
    int d_max, a_max, kz_forward, kz_backward, cta_x, cta_y;
};
std::mutex g_rule_mutex;
BpTileRule g_rules[kBpMaxTileRules];
int g_rule_count = 0;

bool bp_rule(int D, int A, BpTileRule& out) {
    std::lock_guard<std::mutex> lock(g_rule_mutex);
    for (int i = 0; i < g_rule_count; ++i)
        if (D <= g_rules[i].d_max && A <= g_rules[i].a_max) {
            out = g_rules[i];
            return true;
        }
    return false;
}

bool valid_kz(int k) { return k == 0 || k == 1 || k == 2 || k == 4 || k == 8; }
}  // namespace

int bp_add_tile_rule(int d_max, int a_max, int kz_forward, int kz_backward, int cta_x, int cta_y) {
    if (d_max < 1 || a_max < 1 || !valid_kz(kz_forward) || !valid_kz(kz_backward)) return -1;
    const bool cta_default = cta_x == 0 && cta_y == 0;
    if (!cta_default && (cta_x < 1 || cta_y < 1 || cta_x * cta_y > kBpMaxWarps)) return -1;
    std::lock_guard<std::mutex> lock(g_rule_mutex);
    if (g_rule_count >= kBpMaxTileRules) return -2;
    g_rules[g_rule_count++] = BpTileRule{d_max, a_max, kz_forward, kz_backward, cta_x, cta_y};
    return 0;
}

void bp_clear_tile_rules() {
    std::lock_guard<std::mutex> lock(g_rule_mutex);
    g_rule_count = 0;
}

static int bp_nominal_kz(int D) { return D <= 32 ? 1 : 2; }

int bp_kz_forward(int D, int A) {
    BpTileRule r;
    if (bp_rule(D, A, r) && r.kz_forward) return r.kz_forward;
    return bp_nominal_kz(D);
}

int bp_kz_backward(int D, int A) {
    BpTileRule r;
    if (bp_rule(D, A, r) && r.kz_backward) return r.kz_backward;
    return D <= 32 ? 1 : D <= 64 ? 2 : 4;
}

// Column patch of a forward CTA (cx*cy <= kBpMaxWarps); 8 x 1 built in.
void bp_forward_cta(int D, int A, int& cx, int& cy) {
    BpTileRule r;
    if (bp_rule(D, A, r) && r.cta_x) {
        cx = r.cta_x;
        cy = r.cta_y;
        return;
    }
    cx = 8;
    cy = 1;
}

void bp_grid(int D, int H, int W, int kz, unsigned& gx, unsigned& gy) {
    gx = (unsigned)(((W + 7) / 8) * (long long)H);
    gy = (unsigned)ceil_div(D, 32 * kz);
}

long long bp_backward_blocks(int D, int H, int W, int kz) {
    unsigned gx, gy;
    bp_grid(D, H, W, kz, gx, gy);
    return (long long)gx * gy;
}

namespace {
template <int KZ>
int launch_bp_forward_kz(const BpArgs& p, bool pixdiv, bool fdk, dim3 grid, cudaStream_t s) {
    const unsigned threads = 32u * (unsigned)(p.cta_x * p.cta_y);
    // a column's values of 32 views, then the transposed tile in their place
    const size_t smem = std::max<size_t>(
        threads * (sizeof(float4) + sizeof(float2)),
        sizeof(float) * 32 * KZ * (kBpMaxWarps + 1));
    if (fdk) {
        if (pixdiv) bp_forward_kernel<KZ, true, true><<<grid, threads, smem, s>>>(p);
        else bp_forward_kernel<KZ, false, true><<<grid, threads, smem, s>>>(p);
    } else {
        if (pixdiv) bp_forward_kernel<KZ, true, false><<<grid, threads, smem, s>>>(p);
        else bp_forward_kernel<KZ, false, false><<<grid, threads, smem, s>>>(p);
    }
    DGC_LAUNCH_CHECK("bp_forward_kernel");
    return DGC_OK;
}

template <int KZ>
int launch_bp_backward_kz(const BpArgs& p, int gp, bool geo, dim3 grid, cudaStream_t s) {
    if (!geo) bp_backward_kernel<KZ, 1, false><<<grid, 256, 0, s>>>(p);
    else if (gp) bp_backward_kernel<KZ, 1, true><<<grid, 256, 0, s>>>(p);
    else bp_backward_kernel<KZ, 0, true><<<grid, 256, 0, s>>>(p);
    DGC_LAUNCH_CHECK("bp_backward_kernel");
    return DGC_OK;
}
}  // namespace

void bp_forward_tile(int D, int H, int W, int A, int& kz, int& cx, int& cy) {
    BpTileRule r;
    const bool asked = bp_rule(D, A, r) && (r.kz_forward || r.cta_x);
    if (asked || (long long)ceil_div(W, 2) * ceil_div(H, 2) > INT_MAX) {
        kz = asked && r.kz_forward ? r.kz_forward : bp_nominal_kz(D);
        cx = asked && r.cta_x ? r.cta_x : 8;
        cy = asked && r.cta_x ? r.cta_y : 1;
        return;
    }
    // The kernel's own choice: 2 x 2 columns and the fewest blocks of up to 128 slices,
    // each no deeper than it needs to be (KZ = 2 / 3 / 4, ms: 70 x 256^2, 180 views 1.62 /
    // 1.21 / -, 96 x 128^2, 180 views 0.50 / 0.45 / -, 128^3 0.54 / 0.70 / 0.52, 160^3, 200
    // views 1.12 / 1.08 / 1.29, 192^3, 360 views 3.37 / 3.45 / 3.85, 256^3 6.65 / 7.08 /
    // 6.48)
    cx = cy = 2;
    kz = ceil_div(D, 32 * (long long)ceil_div(D, 128));
    // Where few columns leave the chip idle, the shallowest blocks that are still one
    // wave (28 warps per SM at 72 registers): 91 x 26 x 31, 337 views 0.146 -> 0.081 ms;
    // 213 x 3 x 25, 344 views 0.233 -> 0.126; 228 x 40 x 22, 103 views 0.071 -> 0.058 (two
    // waves of 32 slices: 0.071).  With deep blocks 353 x 16 x 7, 291 views took 0.192 ms
    // against the former 8 x 1 columns' 0.173, and takes 0.089.
    for (int k = 1; k < kz; ++k)
        if ((long long)W * H * ceil_div(D, 32 * k) <= 148 * 28) kz = k;
}

int bp_launch_forward(const BpArgs& args, bool fdk, cudaStream_t s) {
    DGC_TRACE(fdk ? "bp_forward_kernel<fdk>" : "bp_forward_kernel", s);
    BpArgs p = args;
    int kz = 0;
    bp_forward_tile(p.D, p.H, p.W, p.A, kz, p.cta_x, p.cta_y);
    const bool pixdiv = !is_pow2_float(p.pixel_size);
    const dim3 grid((unsigned)(ceil_div(p.W, p.cta_x) * (long long)ceil_div(p.H, p.cta_y)),
                    (unsigned)ceil_div(p.D, 32 * kz));
    switch (kz) {
        case 1: return launch_bp_forward_kz<1>(p, pixdiv, fdk, grid, s);
        case 2: return launch_bp_forward_kz<2>(p, pixdiv, fdk, grid, s);
        case 3: return launch_bp_forward_kz<3>(p, pixdiv, fdk, grid, s);
        case 4: return launch_bp_forward_kz<4>(p, pixdiv, fdk, grid, s);
        default: return launch_bp_forward_kz<8>(p, pixdiv, fdk, grid, s);
    }
}

int bp_launch_backward(const BpArgs& p, cudaStream_t s) {
    DGC_TRACE(p.grad_projections ? "bp_backward_kernel<gp>" : "bp_backward_kernel", s);
    // the Z blocking the caller sized the partials for (a rule added by another
    // thread in between must not change the grid)
    const int kz = p.kz_backward ? p.kz_backward : bp_kz_backward(p.D, p.A);
    unsigned gx, gy;
    bp_grid(p.D, p.H, p.W, kz, gx, gy);
    const int gp = p.grad_projections ? 1 : 0;
    const bool geo = p.partials != nullptr;
    const dim3 grid(gx, gy);
    switch (kz) {
        case 1: return launch_bp_backward_kz<1>(p, gp, geo, grid, s);
        case 2: return launch_bp_backward_kz<2>(p, gp, geo, grid, s);
        case 4: return launch_bp_backward_kz<4>(p, gp, geo, grid, s);
        default: return launch_bp_backward_kz<8>(p, gp, geo, grid, s);
    }
}

size_t bp_column_floats(int D, int H, int W) { return (size_t)(D + 3) * H * W; }

// Gather or scatter?  The scatter's work is the voxels; the gather's the columns
// times the detector's rows and, beside them, its lists: per (bin, row of the volume)
// whatever there is to find.  So it wants deep columns, many of them in a bin and
// views enough to fill the chip; what it wants of the magnification the views know
// (bp_view_choice_kernel).  Measured over 506 random scans and cubes (20 to 300 voxels a
// side, 1 to 400 views, 1.1- to 6-fold magnification, voxels of 0.5 to 4 pixels, a
// shadow of half to twice the detector), the projection gradient alone: the scans
// that this takes to the gather need 0.58 to 1.5 times the scatter's time, 1.9 below
// 20000 columns x views (30 us, half of them launches; the sums are reproducible
// there too) and 1.2 at most above 0.1 ms.  A rule by sizes and voxel / pixel alone took 181 of
// them, of which 123 were slower, up to 12 times.  Gather / scatter: 10.0 / 18.5 ms
// (256^3 / 360 x 384^2), 1.07 / 1.63 (128^3 / 180 x 256^2), 0.103 / 0.142 (64^3 / 90 x
// 117^2); with 4 views 0.78 to 2.1 times.
// With the geometry gradients the scatter shares its march with theirs, and the gather
// gains only on large volumes: 20.4 / 24.4 ms at 256^3 / 360 x 384^2, 1.81 / 1.98 at
// 128^3 / 180 x 234^2, but 1.1 to 1.9 times slower below the line drawn here.  What a
// launch that was not taken costs: 10-30 us.
bool bp_may_gather(int A, int U, int V, int D, int H, int W, bool with_geometry) {
    const long long area = (long long)H * W;
    if (D > 1 << 20) return false;  // bp_columns' grid
    if (with_geometry) return D >= 100 && V >= 48 && area >= 25LL * (U - 1) && area * A >= 1600000;
    return A >= 6 && D >= 48 && V >= 48 && area >= 15LL * (U - 1);
}

int bp_view_choice(const Geometry& g, const BpArgs& p, bool with_geometry, ViewRow* vt,
                   cudaStream_t s) {
    DGC_TRACE("bp_view_choice", s);
    bp_view_choice_kernel<<<1, 256, 0, s>>>(g, p, with_geometry ? 0.9f : 0.75f, vt);
    DGC_LAUNCH_CHECK("bp_view_choice");
    return DGC_OK;
}

int bp_launch_gather(const BpArgs& p, float* columns, cudaStream_t s) {
    {
        DGC_TRACE("bp_columns", s);
        const dim3 grid((unsigned)(ceil_div(p.W, 32) * (long long)p.H), (unsigned)ceil_div(p.D + 3, 32));
        bp_columns_kernel<<<grid, dim3(32, 8), 0, s>>>(p.grad_volume, p.D, p.H, p.W, p.vt,
                                                     columns);
        DGC_LAUNCH_CHECK("bp_columns");
    }
    DGC_TRACE("bp_adjoint_kernel", s);
    // pixels a thread and warps a CTA: the fewest idle slots, a column's own
    // instructions (about 10) against 25 a pixel; a warp that the volume's shadow
    // does not reach costs little (its rows at about twofold magnification: the host
    // does not know the views')
    const float shadow = 2.2f * p.D * p.voxel_size * p.inv_pixel;
    int nv = 1, warps = 1, tiles = 1;
    float best = FLT_MAX;
    for (int n = 1; n <= 3; ++n) {
        const int t = ceil_div(p.V, 32LL * n * kAdjMaxWarps);
        const int w = ceil_div(ceil_div(p.V, t), 32 * n);
        const float slots = std::min(32.0f * n * w * t, shadow + 32.0f * n);
        const float cost = slots * (25.0f + 10.0f / n);
        if (cost < best) {
            best = cost;
            nv = n;
            warps = w;
            tiles = t;
        }
    }
    // bins per CTA: up to 16, as many as leave every SM some 32 CTAs (one instead of
    // two where even these leave fewer: 0.6-0.9 of the time with 1 to 16 views)
    int bins = 16;
    while (bins > 1 && (long long)p.A * ceil_div(p.U - 1, bins) * tiles < 148LL * 32) bins >>= 1;
    const int bin_blocks = ceil_div(p.U - 1, bins);
    const unsigned grid = (unsigned)((long long)p.A * bin_blocks * tiles);
    const size_t smem = (size_t)warps * kAdjList * (sizeof(AdjColumn) + sizeof(unsigned));
    switch (nv) {
        case 1: bp_adjoint_kernel<1><<<grid, 32 * warps, smem, s>>>(p, columns, bins, bin_blocks, tiles); break;
        case 2: bp_adjoint_kernel<2><<<grid, 32 * warps, smem, s>>>(p, columns, bins, bin_blocks, tiles); break;
        default: bp_adjoint_kernel<3><<<grid, 32 * warps, smem, s>>>(p, columns, bins, bin_blocks, tiles); break;
    }
    DGC_LAUNCH_CHECK("bp_adjoint_kernel");
    return DGC_OK;
}

__global__ void clamp_volume_kernel(float* __restrict__ v, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float x = v[i];
        v[i] = x < 0.0f ? 0.0f : x;  // as the FDK epilogue: NaN propagates
    }
}

int bp_clamp_volume(float* volume, long long n, cudaStream_t s) {
    DGC_TRACE("clamp_volume", s);
    const int blocks = (int)std::min<long long>((n + 255) / 256, 148LL * 16);
    clamp_volume_kernel<<<blocks, 256, 0, s>>>(volume, n);
    DGC_LAUNCH_CHECK("clamp_volume");
    return DGC_OK;
}

int bp_reduce_partials(const double* partials, int A, long long nblocks, const GeometryGrad& out,
                       cudaStream_t s) {
    DGC_TRACE("bp_reduce_partials", s);
    bp_reduce_partials_kernel<<<A, 256, 0, s>>>(partials, nblocks, out);
    DGC_LAUNCH_CHECK("bp_reduce_partials");
    return DGC_OK;
}

}  // namespace dgc
