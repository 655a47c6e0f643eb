// gsv_render.cu -- forward / backward tile kernels and the gradient finalize.
//
// Forward, tile edge 8 (the reference default): one CTA per tile, one warp per 4x4x4
//   block of it, eight lanes per (Gaussian, block), see forward_tile.
//
// Backward, tile edge 8: one lane per (Gaussian, 4x4x4 block of the tile),
//   see backward_tile.
//
// Tile edge 4: the same walks, one warp per tile.  Other tile edges: a generic
// one-voxel-per-thread kernel pair.
//
// Reference semantics (3DGS/3dgsVC/gaussian/cuda_ext/tile_voxelize_cuda_kernel.cu):
//   forward  :118-141  vol = sum_{g in list(tile), m <= 9} exp(-m/2) rho_g
//   backward :217-252  dL/drho, dL/dcenter, dL/dcov_inv for included pairs
#include <cstdio>

#include "gsv_common.cuh"

using namespace gsv;

namespace gsv {
int layout_for(gsv_shape shape, int64_t n, int64_t cap, int flags, GaussLayout* G, PairLayout* P,
               int64_t* ntiles);
}

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;

struct RenderArgs {
    // native Gaussians
    const Rec* recs;
    const float4* ext;  // conservative tight extent of each inclusion set (voxels)
    // reference-compatible Gaussians
    const float* centers;
    const float* cov_inv;
    const float* den_r;
    const float* den_i;
    const float* half_shape;
    // binning
    const int2* ranges;
    const int32_t* pair_ids;
    int32_t d, h, w, ts, nth, ntw;
    int64_t ntiles;
    float hs[3], ih[3];  // native half shape and its reciprocal
    // forward outputs
    float* vol;    // complex64 interleaved
    float* vol_r;  // planar
    float* vol_i;
    // backward inputs / outputs
    const float* gvol;  // complex64 interleaved
    const float* gv_r;  // planar
    const float* gv_i;
    float* accum;     // [n, 12] moments (native, atomics)
    float* partials;  // [pairs, 12] moments (native, deterministic), at each pair's emission index ...
    uint8_t* kept;    // ... of the pairs marked here; the others add nothing
    const int64_t* offsets;  // per-Gaussian first emission index (binning scan)
    int64_t capacity;        // pair capacity (bound of every emission index)
    float* g_center;  // compat outputs
    float* g_cov;
    float* g_dr;
    float* g_di;
    int chunk;  // Gaussians staged per warp chunk (<= 32)
    int cull;   // skip Gaussians / row slots outside the tight extent
    int split;  // backward: CTAs that may share one (half) tile's list ...
    int part;   // ... one for each started `part` positions
    // finalize
    gsv_params prm;
    gsv_grads grd;
    int64_t dstride;  // element stride of the density gradients
    const int4* boxes;
};

template <bool COMPAT>
__device__ __forceinline__ void compat_ih(const RenderArgs& a, float ih[3]) {
    if (COMPAT) {
#pragma unroll
        for (int k = 0; k < 3; ++k) ih[k] = __fdiv_rn(1.0f, __ldg(a.half_shape + k));
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) ih[k] = a.ih[k];
    }
}

template <bool COMPAT>
__device__ __forceinline__ Rec load_rec(const RenderArgs& a, int gid, const float ih[3]) {
    Rec r;
    if (!COMPAT) {
        const float4* p = reinterpret_cast<const float4*>(a.recs + gid);
        const float4 x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
        r.c0 = x.x; r.c1 = x.y; r.c2 = x.z; r.q00 = x.w;
        r.q01x2 = y.x; r.q02x2 = y.y; r.q11 = y.z; r.q12x2 = y.w;
        r.q22 = z.x; r.rho_r = z.y; r.rho_i = z.z; r.pad = 0.0f;
    } else {
        float m9[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) m9[k] = __ldg(a.cov_inv + int64_t(gid) * 9 + k);
        float qc[6];
        qcoef_from_covinv(m9, ih, qc);
        r.c0 = __ldg(a.centers + int64_t(gid) * 3);
        r.c1 = __ldg(a.centers + int64_t(gid) * 3 + 1);
        r.c2 = __ldg(a.centers + int64_t(gid) * 3 + 2);
        r.q00 = qc[0]; r.q01x2 = qc[1]; r.q02x2 = qc[2]; r.q11 = qc[3]; r.q12x2 = qc[4]; r.q22 = qc[5];
        r.rho_r = __ldg(a.den_r + gid);
        r.rho_i = __ldg(a.den_i + gid);
        r.pad = 0.0f;
    }
    return r;
}

__device__ __forceinline__ void decode_tile(const RenderArgs& a, int64_t tile, int& d0, int& h0, int& w0) {
    const int64_t per = int64_t(a.nth) * a.ntw;
    d0 = int(tile / per) * a.ts;
    const int64_t rem = tile % per;
    h0 = int(rem / a.ntw) * a.ts;
    w0 = int(rem % a.ntw) * a.ts;
}

// Reduce-scatter of 16 per-lane values over the warp: afterwards lane l
// holds the warp total of value (l >> 1) in v[0] (lanes l and l^1 agree).
__device__ __forceinline__ float warp_reduce_scatter16(float v[16], int lane) {
    {
        const bool hi = lane & 16;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float send = hi ? v[i] : v[i + 8];
            const float keep = hi ? v[i + 8] : v[i];
            v[i] = keep + __shfl_xor_sync(kFull, send, 16);
        }
    }
    {
        const bool hi = lane & 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float send = hi ? v[i] : v[i + 4];
            const float keep = hi ? v[i + 4] : v[i];
            v[i] = keep + __shfl_xor_sync(kFull, send, 8);
        }
    }
    {
        const bool hi = lane & 4;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float send = hi ? v[i] : v[i + 2];
            const float keep = hi ? v[i + 2] : v[i];
            v[i] = keep + __shfl_xor_sync(kFull, send, 4);
        }
    }
    {
        const bool hi = lane & 2;
        const float send = hi ? v[0] : v[1];
        const float keep = hi ? v[1] : v[0];
        v[0] = keep + __shfl_xor_sync(kFull, send, 2);
    }
    return v[0] + __shfl_xor_sync(kFull, v[0], 1);
}

// Whether a Gaussian's moments add anything.  With none of its voxels included they are all zero, and its
// coefficients may be NaN or infinite: 0 * NaN must not reach the gradient, which is zero (the reference
// sums over included voxels only, tile_voxelize_cuda_kernel.cu:217-252).
__device__ __forceinline__ bool any_moment(const float m[kMom]) {
    bool any = false;
#pragma unroll
    for (int i = 0; i < kMom; ++i) any |= m[i] != 0.f;
    return any;
}

// Compat outputs for one (tile, Gaussian): every lane holds `tot` (lane 2i
// holds moment i); lanes 0..13 issue one atomic each.
__device__ __forceinline__ void compat_emit(const RenderArgs& a, const Rec& g, int gid, float tot,
                                            int lane, const float ih[3]) {
    float m[kMom];
#pragma unroll
    for (int i = 0; i < kMom; ++i) m[i] = __shfl_sync(kFull, tot, 2 * i);
    if (!any_moment(m)) return;  // warp-uniform
    float out;
    switch (lane) {
        case 0: out = m[0]; break;
        case 1: out = m[1]; break;
        // dL/dcenter_a = -2 sum_b Q_ab S1_b   (reference: -2 (M d)_a / hs_a, .cu:241-243)
        case 2: out = -(2.0f * g.q00 * m[2] + g.q01x2 * m[3] + g.q02x2 * m[4]); break;
        case 3: out = -(g.q01x2 * m[2] + 2.0f * g.q11 * m[3] + g.q12x2 * m[4]); break;
        case 4: out = -(g.q02x2 * m[2] + g.q12x2 * m[3] + 2.0f * g.q22 * m[4]); break;
        // dL/dcov_inv_ab = sum a d_a d_b = S2_ab / (hs_a hs_b)  (.cu:244-252)
        case 5: out = m[5] * ih[0] * ih[0]; break;
        case 6: case 8: out = m[6] * ih[0] * ih[1]; break;
        case 7: case 11: out = m[7] * ih[0] * ih[2]; break;
        case 9: out = m[8] * ih[1] * ih[1]; break;
        case 10: case 12: out = m[9] * ih[1] * ih[2]; break;
        case 13: out = m[10] * ih[2] * ih[2]; break;
        default: out = 0.0f; break;
    }
    if (lane == 0) atomicAdd(a.g_dr + gid, out);
    else if (lane == 1) atomicAdd(a.g_di + gid, out);
    else if (lane < 5) atomicAdd(a.g_center + int64_t(gid) * 3 + (lane - 2), out);
    else if (lane < 14) {
        // lanes 5..13 -> cov entries 0..8 in row-major order
        const int e = lane - 5;
        atomicAdd(a.g_cov + int64_t(gid) * 9 + e, out);
    }
}

// Emission index of the pair (Gaussian gid, tile (td, th, tw)): the
// Gaussian's first index plus the tile's raster position in its tile box --
// where binning emitted it.  Per-pair partials stored at this index lie
// contiguously per Gaussian, in tile raster order.  -1: past the pair capacity
// (overflow, flagged), the partial is dropped.
__device__ __forceinline__ int32_t emission_index(const RenderArgs& a, int gid, int td, int th, int tw) {
    const int4 b = __ldg(a.boxes + gid);
    const int t0 = b.x & 0xffff, t1 = (b.x >> 16) & 0xffff, t2 = b.y & 0xffff;
    const int n1 = b.z & 0xffff, n2 = (b.z >> 16) & 0xffff;
    const int64_t e = __ldg(a.offsets + gid) + (int64_t(td - t0) * n1 + (th - t1)) * n2 + (tw - t2);
    return e < a.capacity ? int32_t(e) : -1;
}

// ---------------------------------------------------------------------------
// 4x4x4 blocks: the unit the render kernels evaluate
// ---------------------------------------------------------------------------

constexpr int kBlk = 4;                     // edge of a block
constexpr int kBlkVox = kBlk * kBlk * kBlk;
// Above this magnitude a density or an upstream gradient may overflow a product that a voxel outside
// the cutoff must not see; such inputs (and NaN) take the guarded loop.
constexpr float kBig = 1e15f;

__device__ __forceinline__ float4 rec_quad(const Rec& r, int i) {
    return i == 0 ? make_float4(r.c0, r.c1, r.c2, r.q00)
                  : (i == 1 ? make_float4(r.q01x2, r.q02x2, r.q11, r.q12x2) : make_float4(r.q22, r.rho_r, r.rho_i, 0.f));
}
__device__ __forceinline__ Rec rec_of(float4 x, float4 y, float4 z) {
    Rec r;
    r.c0 = x.x; r.c1 = x.y; r.c2 = x.z; r.q00 = x.w;
    r.q01x2 = y.x; r.q02x2 = y.y; r.q11 = y.z; r.q12x2 = y.w;
    r.q22 = z.x; r.rho_r = z.y; r.rho_i = z.z; r.pad = 0.0f;
    return r;
}

// Separating plane of a Gaussian's inclusion set and a block, from the block centre's offset e to the
// Gaussian: with n = Q e (the gradient there, up to a factor), the block's voxels x satisfy
// n.x >= m(e) - 1.5 |n|_1, and {m <= 9} lies in n.x <= 3 sqrt(m(e)).  `thr`: plane_by_k.  On
// fits' Gaussians 93-96% of the blocks kept by this test and the extent hold an included voxel;
// the extent's box alone keeps 1.4 to 1.6 times as many.
__device__ __forceinline__ bool plane_separates(float n0, float n1, float n2, float e0, float e1, float e2, float thr,
                                                float factor) {
    const float m = fmaf(n0, e0, fmaf(n1, e1, n2 * e2));
    const float t = fmaf(-1.515f, fabsf(n0) + fabsf(n1) + fabsf(n2), factor * m);
    return t > 0.0f && t * t > thr * m;
}

// Offset of a Gaussian's coordinate c to the centre of the block whose first voxel is v.  FP32 holds the centre
// below 2^23, which binned grids (`binned`: at most 65535 tiles on an axis) stay under; above it the offset goes
// by the first voxel.  (By the first voxel always: one more addition each, the batched forward of four volumes 6 us
// slower in 863.)
__device__ __forceinline__ float centre_offset(int v, float c, bool binned) {
    return binned ? (float(v) + 1.5f) - c : (float(v) - c) + 1.5f;
}

// Which of a tile's eight blocks (bit 4 bd + 2 bh + bw) may hold a voxel the Gaussian includes.
// x: its tight extent (w: the plane threshold); without `use_box` only the planes are tried.
__device__ __forceinline__ unsigned block_mask8(const Rec& r, float4 x, int d0, int h0, int w0, bool use_box) {
    unsigned in = 0xff;
    if (use_box) {
        const float lo0 = __fsub_rn(r.c0, x.x), hi0 = __fadd_rn(r.c0, x.x);
        const float lo1 = __fsub_rn(r.c1, x.y), hi1 = __fadd_rn(r.c1, x.y);
        const float lo2 = __fsub_rn(r.c2, x.z), hi2 = __fadd_rn(r.c2, x.z);
        in = ((lo0 <= float(d0 + 3) && hi0 >= float(d0)) ? 0x0fu : 0u) |
             ((lo0 <= float(d0 + 7) && hi0 >= float(d0 + 4)) ? 0xf0u : 0u);
        in &= ((lo1 <= float(h0 + 3) && hi1 >= float(h0)) ? 0x33u : 0u) |
              ((lo1 <= float(h0 + 7) && hi1 >= float(h0 + 4)) ? 0xccu : 0u);
        in &= ((lo2 <= float(w0 + 3) && hi2 >= float(w0)) ? 0x55u : 0u) |
              ((lo2 <= float(w0 + 7) && hi2 >= float(w0 + 4)) ? 0xaau : 0u);
    }
    const float thr = x.w, factor = plane_factor(thr);
    const float h01 = 0.5f * r.q01x2, h02 = 0.5f * r.q02x2, h12 = 0.5f * r.q12x2;
#pragma unroll
    for (int bd = 0; bd < 2; ++bd) {
        const float e0 = centre_offset(d0 + 4 * bd, r.c0, use_box);
#pragma unroll
        for (int bh = 0; bh < 2; ++bh) {
            const float e1 = centre_offset(h0 + 4 * bh, r.c1, use_box);
            const float a0 = fmaf(h01, e1, r.q00 * e0), a1 = fmaf(h01, e0, r.q11 * e1), a2 = fmaf(h02, e0, h12 * e1);
#pragma unroll
            for (int bw = 0; bw < 2; ++bw) {
                const float e2 = centre_offset(w0 + 4 * bw, r.c2, use_box);
                if (plane_separates(fmaf(h02, e2, a0), fmaf(h12, e2, a1), fmaf(r.q22, e2, a2), e0, e1, e2, thr, factor))
                    in &= ~(1u << (4 * bd + 2 * bh + bw));
            }
        }
    }
    return in;
}

// Packed pairs of FP32 (two rows of a block at once): each half rounds as the scalar operation does.
typedef float2 f32x2;
__device__ __forceinline__ f32x2 dup2(float x) { return make_float2(x, x); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float sum2(f32x2 x) {
    return x.x + x.y;
}

// The staged upstream gradient of a block: rows j, j + 1 (j even) of a plane side by side, one float4
// {re j, re j+1, im j, im j+1} per voxel column.
__device__ __forceinline__ int grad_at(int i, int j, int k) { return ((i * 2 + (j >> 1)) * kBlk + k) * 4 + (j & 1); }

// One Gaussian's 11 moments over one block, all in one lane.  gs: the block's staged upstream gradient;
// v0..v2: the block's first voxel.  The weight of an excluded voxel is zero.  Bound by FP32 issue:
// packed pairs of rows take 39 issue slots per row of four voxels where the scalar form takes 66, and
// the FMA pipe the same time.
__device__ __forceinline__ void block_moments(const Rec& g, const float* gs, float v0, float v1, float v2,
                                              float mom[kMomStride]) {
    f32x2 e1[2], e1s[2], qe[2], e2[kBlk], e2s[kBlk];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const float lo = __fsub_rn(v1 + float(2 * p), g.c1), hi = __fsub_rn(v1 + float(2 * p + 1), g.c1);
        e1[p] = make_float2(lo, hi);
        e1s[p] = mul2(e1[p], e1[p]);
        qe[p] = mul2(mul2(dup2(g.q11), e1[p]), e1[p]);
    }
#pragma unroll
    for (int k = 0; k < kBlk; ++k) {
        e2[k] = dup2(__fsub_rn(v2 + float(k), g.c2));
        e2s[k] = mul2(e2[k], e2[k]);
    }
    const f32x2 hr = dup2(-0.5f * g.rho_r), hi = dup2(-0.5f * g.rho_i);
    const f32x2 q01 = dup2(g.q01x2), q12 = dup2(g.q12x2), q22 = dup2(g.q22), scale = dup2(kNegHalfLog2e);
    const f32x2 zero = dup2(0.f);
    f32x2 Dr = zero, Di = zero, M11 = zero, M12 = zero, M22 = zero;
    float S0 = 0.f, S1 = 0.f, S2 = 0.f, M00 = 0.f, M01 = 0.f, M02 = 0.f;
#pragma unroll 2
    for (int i = 0; i < kBlk; ++i) {
        const float e0s = __fsub_rn(v0 + float(i), g.c0);
        const f32x2 e0 = dup2(e0s), q0e = dup2(__fmul_rn(g.q00, e0s)), qb = dup2(__fmul_rn(g.q02x2, e0s));
        f32x2 P0, P1, P2;  // the plane's sums of a, a e1, a e2
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            // row_a, row_b
            const f32x2 A = fma2(fma2(q01, e1[p], q0e), e0, qe[p]);
            const f32x2 B = fma2(q12, e1[p], qb);
            f32x2 R0, R1;
#pragma unroll
            for (int k = 0; k < kBlk; ++k) {
                const float4 gv = *reinterpret_cast<const float4*>(gs + grad_at(i, 2 * p, k));
                const f32x2 gr = make_float2(gv.x, gv.y), gi = make_float2(gv.z, gv.w);
                const f32x2 m = fma2(fma2(q22, e2[k], B), e2[k], A);  // row_m
                const f32x2 x = mul2(m, scale);
                const float wl = ex2_approx(x.x), wh = ex2_approx(x.y);
                const f32x2 w = make_float2(m.x <= kCut ? wl : 0.f, m.y <= kCut ? wh : 0.f);
                const f32x2 a = mul2(w, fma2(hr, gr, mul2(hi, gi)));
                Dr = fma2(w, gr, Dr);
                Di = fma2(w, gi, Di);
                R0 = k ? add2(R0, a) : a;
                R1 = k ? fma2(a, e2[k], R1) : mul2(a, e2[k]);
                M22 = fma2(a, e2s[k], M22);
            }
            P0 = p ? add2(P0, R0) : R0;
            P1 = p ? fma2(e1[p], R0, P1) : mul2(e1[p], R0);
            P2 = p ? add2(P2, R1) : R1;
            M11 = fma2(e1s[p], R0, M11);
            M12 = fma2(e1[p], R1, M12);
        }
        const float p0 = sum2(P0), p1 = sum2(P1), p2 = sum2(P2), u = e0s * p0;
        S0 += u;
        S1 += p1;
        S2 += p2;
        M00 = fmaf(e0s, u, M00);
        M01 = fmaf(e0s, p1, M01);
        M02 = fmaf(e0s, p2, M02);
    }
    mom[0] = sum2(Dr); mom[1] = sum2(Di); mom[2] = S0; mom[3] = S1; mom[4] = S2;
    mom[5] = M00; mom[6] = M01; mom[7] = M02; mom[8] = sum2(M11); mom[9] = sum2(M12);
    mom[10] = sum2(M22); mom[11] = 0.f;
}

// block_moments for infinite, NaN or huge inputs: a voxel outside the cutoff takes part in no product, and
// a Gaussian with no voxel inside adds exactly zero.
__device__ __noinline__ void block_moments_guarded(const Rec& g, const float* gs, float v0, float v1, float v2,
                                                   float mom[kMomStride]) {
    const float hr = -0.5f * g.rho_r, hi = -0.5f * g.rho_i;
    for (int i = 0; i < kMomStride; ++i) mom[i] = 0.f;
    for (int i = 0; i < kBlk; ++i)
        for (int j = 0; j < kBlk; ++j) {
            const float e0 = __fsub_rn(v0 + float(i), g.c0), e1 = __fsub_rn(v1 + float(j), g.c1);
            const float A = row_a(g, e0, e1), B = row_b(g, e0, e1);
            for (int k = 0; k < kBlk; ++k) {
                const float e2 = __fsub_rn(v2 + float(k), g.c2);
                const float m = row_m(g.q22, A, B, e2);
                if (!(m <= kCut)) continue;
                const float gr = gs[grad_at(i, j, k)], gi = gs[grad_at(i, j, k) + 2];
                const float w = ex2_approx(m * kNegHalfLog2e);
                const float a = w * fmaf(hi, gi, hr * gr);
                mom[0] = fmaf(w, gr, mom[0]);
                mom[1] = fmaf(w, gi, mom[1]);
                mom[2] = fmaf(a, e0, mom[2]);
                mom[3] = fmaf(a, e1, mom[3]);
                mom[4] = fmaf(a, e2, mom[4]);
                mom[5] = fmaf(a * e0, e0, mom[5]);
                mom[6] = fmaf(a * e0, e1, mom[6]);
                mom[7] = fmaf(a * e0, e2, mom[7]);
                mom[8] = fmaf(a * e1, e1, mom[8]);
                mom[9] = fmaf(a * e1, e2, mom[9]);
                mom[10] = fmaf(a * e2, e2, mom[10]);
            }
        }
}

// Whether a Gaussian needs block_moments_guarded.
__device__ __forceinline__ bool needs_guard(const Rec& r) {
    return !(fabsf(r.rho_r) <= kBig && fabsf(r.rho_i) <= kBig && fabsf(r.c0) <= kBig && fabsf(r.c1) <= kBig &&
             fabsf(r.c2) <= kBig);
}

// A lane's moments: the packed loop's, or the guarded one's where the tile's gradient (`guard`) or the lane's
// own Gaussian needs it.  The two round differently, so each lane keeps to its own: which Gaussians share
// a warp depends on the cull and the execution shape, and must not show in their gradients.
__device__ __forceinline__ void moments_of(const Rec& g, const float* gs, float v0, float v1, float v2, bool guard,
                                           float m[kMomStride]) {
    const bool wild = guard || needs_guard(g);
    if (!guard) block_moments(g, gs, v0, v1, v2, m);
    if (__any_sync(kFull, wild)) {
        float mg[kMomStride];
        block_moments_guarded(g, gs, v0, v1, v2, mg);
#pragma unroll
        for (int i = 0; i < kMomStride; ++i) m[i] = wild ? mg[i] : m[i];
    }
}

// The moments of one (tile, Gaussian) pair to the gradients of the reference's own parameters.
__device__ __forceinline__ void compat_emit_lane(const RenderArgs& a, const Rec& g, int gid, const float m[kMomStride],
                                                 const float ih[3]) {
    if (!any_moment(m)) return;
    atomicAdd(a.g_dr + gid, m[0]);
    atomicAdd(a.g_di + gid, m[1]);
    // dL/dcenter_a = -2 sum_b Q_ab S1_b   (reference: -2 (M d)_a / hs_a, .cu:241-243)
    float* gc = a.g_center + int64_t(gid) * 3;
    atomicAdd(gc, -(2.0f * g.q00 * m[2] + g.q01x2 * m[3] + g.q02x2 * m[4]));
    atomicAdd(gc + 1, -(g.q01x2 * m[2] + 2.0f * g.q11 * m[3] + g.q12x2 * m[4]));
    atomicAdd(gc + 2, -(g.q02x2 * m[2] + g.q12x2 * m[3] + 2.0f * g.q22 * m[4]));
    // dL/dcov_inv_ab = sum a d_a d_b = S2_ab / (hs_a hs_b)  (.cu:244-252)
    float* gm = a.g_cov + int64_t(gid) * 9;
    const float c01 = m[6] * ih[0] * ih[1], c02 = m[7] * ih[0] * ih[2], c12 = m[9] * ih[1] * ih[2];
    atomicAdd(gm, m[5] * ih[0] * ih[0]);
    atomicAdd(gm + 1, c01);
    atomicAdd(gm + 2, c02);
    atomicAdd(gm + 3, c01);
    atomicAdd(gm + 4, m[8] * ih[1] * ih[1]);
    atomicAdd(gm + 5, c12);
    atomicAdd(gm + 6, c02);
    atomicAdd(gm + 7, c12);
    atomicAdd(gm + 8, m[10] * ih[2] * ih[2]);
}

// ---------------------------------------------------------------------------
// Tile edge 8: forward
// ---------------------------------------------------------------------------

// One warp per 4^3 block, eight lanes per Gaussian: a lane owns two neighbouring rows of four voxels
// (packed as pairs), a warp evaluates four Gaussians at a time, and the four partial blocks are summed
// once at the end.  The CTA stages its tile's list in chunks, one position per thread, with the blocks
// each Gaussian may reach; every warp then walks its own block's Gaussians.  A pair takes 16 issue slots,
// 16 slots of the FMA pipe and 16 of the exponential unit (per scheduler), so all three bound it; sixteen
// lanes per Gaussian in scalar form take 23 issue slots.  128x128x96/50k 195 -> 140 us, 500k 463 -> 308 us,
// against whole rows of a tile per lane (4x8x8 voxels a warp, 11-25% of them inside the cutoff).
// Arriving records early (cp.async into a second buffer, one barrier a chunk) measured 147 us, chunks of
// 512 positions 140 to 142 us.
// The sum of a voxel depends on the kept Gaussians alone: without the cull the others are walked too,
// after the kept ones, and add zeros.
constexpr int kFwdRec = 5;  // float4 per staged Gaussian, see FwdRec

// c0, q00, q02x2, - | -c1 twice, q01x2 twice | q11 twice, q12x2 twice | -c2 twice, q22 twice | rho twice each
__device__ __forceinline__ void store_fwd_rec(float4* dst, const Rec& r) {
    dst[0] = make_float4(r.c0, r.q00, r.q02x2, 0.f);
    dst[1] = make_float4(-r.c1, -r.c1, r.q01x2, r.q01x2);
    dst[2] = make_float4(r.q11, r.q11, r.q12x2, r.q12x2);
    dst[3] = make_float4(-r.c2, -r.c2, r.q22, r.q22);
    dst[4] = make_float4(r.rho_r, r.rho_r, r.rho_i, r.rho_i);
}
// A record no voxel includes (its quadratic is NaN), which fills up a list.
__device__ __forceinline__ void store_null_rec(float4* dst) {
    const float nan = __int_as_float(0x7fffffff);
#pragma unroll
    for (int i = 0; i < kFwdRec; ++i) dst[i] = make_float4(nan, 0.f, 0.f, 0.f);
    dst[4] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// The lane's place in its warp's block and its sums: voxels (v0, v1 + {0, 1}, v2 + k).
struct BlockSums {
    float v0;
    f32x2 v1, re[kBlk], im[kBlk];
    float v2;
};

__device__ __forceinline__ BlockSums block_sums(int d0, int h0, int w0, int lane) {
    BlockSums s;
    s.v0 = float(d0 + ((lane >> 1) & 3));
    s.v1 = make_float2(float(h0 + 2 * (lane & 1)), float(h0 + 2 * (lane & 1) + 1));
    s.v2 = float(w0);
#pragma unroll
    for (int k = 0; k < kBlk; ++k) s.re[k] = s.im[k] = make_float2(0.f, 0.f);
    return s;
}

// Adds the Gaussians of `list` (byte offsets of staged records), or the first n records without one; n is a
// multiple of four.
// GUARD: some density is infinite or NaN, so an excluded voxel must not multiply it.
template <bool GUARD>
__device__ __forceinline__ void add_gaussians(BlockSums& s, const float4* recs, const uint16_t* list, int n, int lane) {
    const f32x2 scale = dup2(kNegHalfLog2e);
    const char* base = reinterpret_cast<const char*>(recs);
#pragma unroll 2
    for (int j = lane >> 3; j < n; j += 4) {
        const float4* r = reinterpret_cast<const float4*>(base + (list ? int(list[j]) : j * int(kFwdRec * sizeof(float4))));
        const float4 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3], r4 = r[4];
        const float e0 = __fsub_rn(s.v0, r0.x);
        const f32x2 e1 = add2(s.v1, make_float2(r1.x, r1.y));
        const f32x2 qe = mul2(mul2(make_float2(r2.x, r2.y), e1), e1);
        // row_a, row_b
        const f32x2 A = fma2(fma2(make_float2(r1.z, r1.w), e1, dup2(__fmul_rn(r0.y, e0))), dup2(e0), qe);
        const f32x2 B = fma2(make_float2(r2.z, r2.w), e1, dup2(__fmul_rn(r0.z, e0)));
        const f32x2 nc2 = make_float2(r3.x, r3.y), q22 = make_float2(r3.z, r3.w);
        const f32x2 rr = make_float2(r4.x, r4.y), ri = make_float2(r4.z, r4.w);
#pragma unroll
        for (int k = 0; k < kBlk; ++k) {
            const f32x2 e2 = add2(dup2(s.v2 + float(k)), nc2);
            const f32x2 m = fma2(fma2(q22, e2, B), e2, A);  // row_m
            const f32x2 x = mul2(m, scale);
            const float wl = ex2_approx(x.x), wh = ex2_approx(x.y);
            if (GUARD) {
                if (m.x <= kCut) {
                    s.re[k].x = fmaf(wl, rr.x, s.re[k].x);
                    s.im[k].x = fmaf(wl, ri.x, s.im[k].x);
                }
                if (m.y <= kCut) {
                    s.re[k].y = fmaf(wh, rr.x, s.re[k].y);
                    s.im[k].y = fmaf(wh, ri.x, s.im[k].y);
                }
            } else {
                const f32x2 w = make_float2(m.x <= kCut ? wl : 0.f, m.y <= kCut ? wh : 0.f);
                s.re[k] = fma2(w, rr, s.re[k]);
                s.im[k] = fma2(w, ri, s.im[k]);
            }
        }
    }
}

__device__ __noinline__ void add_gaussians_guarded(BlockSums& s, const float4* recs, const uint16_t* list, int n,
                                                   int lane) {
    add_gaussians<true>(s, recs, list, n, lane);
}

// Sums the warp's four partial blocks ((0 + 1) + (2 + 3)) and stores the block: lane group q keeps
// columns 2 (q % 2), + 1 of row q / 2 of the lane's two.
template <bool PLANAR>
__device__ __forceinline__ void store_block(const RenderArgs& a, const BlockSums& s, int d0, int h0, int w0, int lane) {
    const bool kp = lane & 8, row = lane & 16;
    f32x2 re[2], im[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const f32x2 sr = kp ? s.re[i] : s.re[i + 2], kr = kp ? s.re[i + 2] : s.re[i];
        const f32x2 si = kp ? s.im[i] : s.im[i + 2], ki = kp ? s.im[i + 2] : s.im[i];
        re[i].x = kr.x + __shfl_xor_sync(kFull, sr.x, 8);
        re[i].y = kr.y + __shfl_xor_sync(kFull, sr.y, 8);
        im[i].x = ki.x + __shfl_xor_sync(kFull, si.x, 8);
        im[i].y = ki.y + __shfl_xor_sync(kFull, si.y, 8);
    }
    float vr[2], vi[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        vr[i] = (row ? re[i].y : re[i].x) + __shfl_xor_sync(kFull, row ? re[i].x : re[i].y, 16);
        vi[i] = (row ? im[i].y : im[i].x) + __shfl_xor_sync(kFull, row ? im[i].x : im[i].y, 16);
    }
    const int gd = d0 + ((lane >> 1) & 3), gh = h0 + 2 * (lane & 1) + (row ? 1 : 0), gw = w0 + (kp ? 2 : 0);
    if (gd >= a.d || gh >= a.h) return;
    const int64_t flat = (int64_t(gd) * a.h + gh) * a.w + gw;
    if (PLANAR) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (gw + i < a.w) {
                a.vol_r[flat + i] = vr[i];
                a.vol_i[flat + i] = vi[i];
            }
    } else if (gw + 1 < a.w && (a.w & 1) == 0) {
        reinterpret_cast<float4*>(a.vol)[flat >> 1] = make_float4(vr[0], vi[0], vr[1], vi[1]);
    } else {
        float2* out = reinterpret_cast<float2*>(a.vol) + flat;
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (gw + i < a.w) out[i] = make_float2(vr[i], vi[i]);
    }
}

// Shared memory of a forward CTA of BLOCKS warps; a chunk of the list is a position per thread.
template <int BLOCKS>
struct __align__(16) FwdStage {
    float4 rec[BLOCKS * 32 + 1][kFwdRec];  // the last one is the null record
    uint16_t list[BLOCKS][BLOCKS * 32 + 8];
    uint8_t mask[BLOCKS * 32];
};

__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) <= 3.402823466e38f); }

// Forward of one tile (RPL = 2: eight warps) or of its half `sub` (RPL = 1: four).  Barriers: every thread of
// the CTA must call it for the same (tile, sub).
template <bool COMPAT, bool PLANAR, int RPL>
__device__ __forceinline__ void forward_tile(const RenderArgs& a, int64_t tile, int sub, FwdStage<4 * RPL>& S) {
    constexpr int kChunk = 4 * RPL * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int d0, h0, w0;
    decode_tile(a, tile, d0, h0, w0);
    const int2 rg = a.ranges[tile];
    const int blk = 4 * (RPL == 1 ? sub : 0) + warp;  // bit 4 bd + 2 bh + bw
    const int bd = d0 + (blk >> 2) * kBlk, bh = h0 + ((blk >> 1) & 1) * kBlk, bw = w0 + (blk & 1) * kBlk;
    BlockSums sums = block_sums(bd, bh, bw, lane);
    float ih[3];
    compat_ih<COMPAT>(a, ih);
    int rank = 0;  // of the block's next Gaussian, modulo four
    int next = rg.x + int(threadIdx.x) < rg.y ? __ldg(a.pair_ids + rg.x + threadIdx.x) : 0;
    for (int base = rg.x; base < rg.y; base += kChunk) {
        const bool listed = base + int(threadIdx.x) < rg.y;
        const int gid = next;
        if (base + kChunk + int(threadIdx.x) < rg.y) next = __ldg(a.pair_ids + base + kChunk + threadIdx.x);
        unsigned in = 0;
        bool bad = false;
        if (listed) {
            const Rec r = load_rec<COMPAT>(a, gid, ih);
            const float4 x = COMPAT ? make_float4(0.f, 0.f, 0.f, plane_threshold(r)) : __ldg(a.ext + gid);
            in = block_mask8(r, x, d0, h0, w0, !COMPAT);
            bad = not_finite(r.rho_r) || not_finite(r.rho_i);
            if (in || !a.cull) store_fwd_rec(S.rec[threadIdx.x], r);
        }
        S.mask[threadIdx.x] = uint8_t(in);
        if (threadIdx.x == 0) store_null_rec(S.rec[kChunk]);
        const bool guard = __syncthreads_or(bad);
        // this warp's Gaussians, in list order; the lane group is their rank in the whole list modulo four,
        // however it is cut into chunks
        constexpr uint16_t kNull = kChunk * kFwdRec * sizeof(float4);
        uint16_t* list = S.list[warp];
        int n = rank;
        if (lane < rank) list[lane] = kNull;
#pragma unroll
        for (int s = 0; s < kChunk / 32; ++s) {
            const bool hit = (S.mask[s * 32 + lane] >> blk) & 1u;
            const unsigned bal = __ballot_sync(kFull, hit);
            if (hit) list[n + __popc(bal & ((1u << lane) - 1u))] = uint16_t((s * 32 + lane) * kFwdRec * sizeof(float4));
            n += __popc(bal);
        }
        rank = n & 3;
        if (!a.cull) {  // and the ones the cull would drop, behind them
            for (int s = 0; s < kChunk / 32; ++s) {
                const bool miss = base + s * 32 + lane < rg.y && !((S.mask[s * 32 + lane] >> blk) & 1u);
                const unsigned bal = __ballot_sync(kFull, miss);
                if (miss) list[n + __popc(bal & ((1u << lane) - 1u))] = uint16_t((s * 32 + lane) * kFwdRec * sizeof(float4));
                n += __popc(bal);
            }
        }
        if (lane < ((-n) & 3)) list[n + lane] = kNull;
        __syncwarp();
        n = (n + 3) & ~3;
        if (guard) {
            BlockSums copy = sums;  // so that the sums themselves stay in registers
            add_gaussians_guarded(copy, &S.rec[0][0], list, n, lane);
            sums = copy;
        } else {
            add_gaussians<false>(sums, &S.rec[0][0], list, n, lane);
        }
        __syncthreads();
    }
    store_block<PLANAR>(a, sums, bd, bh, bw, lane);
}

// 64 registers, 32 warps an SM: 24 warps of 80 registers measured 2-8% slower on full grids.
template <bool COMPAT, bool PLANAR, int RPL>
__global__ void __launch_bounds__(128 * RPL, 8 / RPL) k_forward8(const RenderArgs a) {
    __shared__ FwdStage<4 * RPL> stage;
    constexpr int subs = 2 / RPL;
    forward_tile<COMPAT, PLANAR, RPL>(a, blockIdx.x / subs, blockIdx.x % subs, stage);
}

// ---------------------------------------------------------------------------
// Tile edge 8: backward
// ---------------------------------------------------------------------------

// One lane per (Gaussian, 4^3 block): the lane walks the block's 64 voxels and keeps the Gaussian's
// moments to itself, so nothing is reduced across lanes.  (The kernel before it had a warp's lanes
// share one Gaussian over 4x8x8 voxels: 13 shuffles and as many selects per pair, and 16 voxels per
// lane of which 11-25% were inside the cutoff; the blocks kept here are 23-45% inside.)  A warp stages
// up to kBwdCap kept Gaussians of its share of the tile's list, lists their (Gaussian, block) tasks
// block by block, and deals the tasks to its lanes 32 at a time; a Gaussian's tasks add up in shared
// memory in block order, so its pair total does not depend on which lanes ran them.
constexpr int kBwdCap = 80;
constexpr int kGradStride = 2 * kBlkVox + 4;  // floats per block of the staged gradient: two blocks' rows in other banks

struct __align__(16) BwdStage {
    float4 rec[kBwdCap][3];
    float4 mom[kBwdCap][3];
    int32_t gid[kBwdCap];
    int32_t pidx[kBwdCap];          // deterministic: emission index of the pair
    uint16_t task[kBwdCap * 8];     // Gaussian slot | block << 8, by block
    uint8_t mask[kBwdCap];
};

// Backward of one tile (RPL = 2) or of its half `sub` (RPL = 1).  One CTA barrier.
template <bool COMPAT, bool DET, int RPL>
__device__ __forceinline__ void backward_tile(const RenderArgs& a, int64_t tile, int sub, BwdStage* stage,
                                              float* grad, int part) {
    static_assert(!DET || RPL == 2, "deterministic partials need the whole tile in one CTA");
    const int2 rg = a.ranges[tile];
    // a long list is shared by up to a.split CTAs
    const int parts = min(a.split, (rg.y - rg.x + a.part - 1) / a.part);
    if (part >= parts) return;  // CTA-uniform; also every CTA of an empty tile
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int d0, h0, w0;
    decode_tile(a, tile, d0, h0, w0);

    // The tile's upstream gradient, by block (zero outside the volume): thread t takes half a row.
    bool guard = false;
    {
        const int row = threadIdx.x >> 1, bw = threadIdx.x & 1;
        const int ld = row >> 3, lh = row & 7;
        const int gd = d0 + ld, gh = h0 + lh, gw = w0 + kBlk * bw;
        const bool row_ok = gd < a.d && gh < a.h;
        const int64_t flat = (int64_t(gd) * a.h + gh) * a.w + gw;
        const int blk = (ld >> 2) * 4 + (lh >> 2) * 2 + bw;
        float* dst = grad + blk * kGradStride;
#pragma unroll
        for (int k = 0; k < kBlk; ++k) {
            float2 x = make_float2(0.f, 0.f);
            if (row_ok && gw + k < a.w)
                x = COMPAT ? make_float2(__ldg(a.gv_r + flat + k), __ldg(a.gv_i + flat + k))
                           : __ldg(reinterpret_cast<const float2*>(a.gvol) + flat + k);
            guard |= !(fabsf(x.x) <= kBig && fabsf(x.y) <= kBig);
            dst[grad_at(ld & 3, lh & 3, k)] = x.x;
            dst[grad_at(ld & 3, lh & 3, k) + 2] = x.y;
        }
    }
    guard = __syncthreads_or(guard);

    float ih[3];
    compat_ih<COMPAT>(a, ih);
    constexpr int kWords = (kBwdCap + 31) / 32;
    BwdStage& S = stage[warp];
    // list positions of this warp: first, first + stride, ... (part `part` of the tile's CTAs)
    const int stride = kWarps * parts, first = part * kWarps + warp;
    const int mine = rg.y - rg.x > first ? (rg.y - rg.x - first + stride - 1) / stride : 0;
    const unsigned blocks = RPL == 2 ? 0xffu : 0xfu << (4 * sub);
    const int32_t* ids = a.pair_ids + rg.x + first;
    const bool mine_lane = lane < a.chunk;
    // the next round's Gaussian, loaded one round ahead
    int next = mine_lane && lane < mine ? __ldg(ids + stride * lane) : 0;
    for (int i0 = 0; i0 < mine;) {
        int kept = 0;
        for (; i0 < mine && kept + a.chunk <= kBwdCap; i0 += a.chunk) {
            Rec r;
            const int gid = next;
            unsigned in = 0;
            const bool listed = mine_lane && i0 + lane < mine;
            if (mine_lane && i0 + a.chunk + lane < mine) next = __ldg(ids + stride * (i0 + a.chunk + lane));
            if (listed) {
                r = load_rec<COMPAT>(a, gid, ih);
                in = blocks;
                if (a.cull) {
                    const float4 x = COMPAT ? make_float4(0.f, 0.f, 0.f, plane_threshold(r)) : __ldg(a.ext + gid);
                    in &= block_mask8(r, x, d0, h0, w0, !COMPAT);
                }
            }
            const unsigned keep = __ballot_sync(kFull, in != 0);
            if (in) {
                const int pos = kept + __popc(keep & ((1u << lane) - 1u));
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    S.rec[pos][i] = rec_quad(r, i);
                    S.mom[pos][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                S.gid[pos] = gid;
                S.mask[pos] = uint8_t(in);
                if (DET) S.pidx[pos] = emission_index(a, gid, d0 >> 3, h0 >> 3, w0 >> 3);
            }
            kept += __popc(keep);
        }
        __syncwarp();
        // tasks, block by block, each block's Gaussians in list order
        int tasks = 0;
        unsigned mask[kWords];
#pragma unroll
        for (int s = 0; s < kWords; ++s) mask[s] = lane + 32 * s < kept ? S.mask[lane + 32 * s] : 0u;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
#pragma unroll
            for (int s = 0; s < kWords; ++s) {
                const bool hit = (mask[s] >> b) & 1u;
                const unsigned bal = __ballot_sync(kFull, hit);
                if (hit) S.task[tasks + __popc(bal & ((1u << lane) - 1u))] = uint16_t((lane + 32 * s) | (b << 8));
                tasks += __popc(bal);
            }
        }
        __syncwarp();
        for (int t0 = 0; t0 < tasks; t0 += 32) {
            const bool on = t0 + lane < tasks;
            const unsigned task = S.task[on ? t0 + lane : tasks - 1];
            const int slot = task & 0xff, b = task >> 8;
            const Rec g = rec_of(S.rec[slot][0], S.rec[slot][1], S.rec[slot][2]);
            const float* gs = grad + b * kGradStride;
            const float v0 = float(d0 + (b >> 2) * kBlk), v1 = float(h0 + ((b >> 1) & 1) * kBlk),
                        v2 = float(w0 + (b & 1) * kBlk);
            float m[kMomStride];
            moments_of(g, gs, v0, v1, v2, guard, m);
            // a Gaussian may have two of its blocks among these lanes: one block at a time
            const int b_end = __shfl_sync(kFull, b, 31);
            for (int bb = __shfl_sync(kFull, b, 0); bb <= b_end; ++bb) {
                if (on && b == bb) {
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        float4 x = S.mom[slot][i];
                        x.x += m[4 * i];
                        x.y += m[4 * i + 1];
                        x.z += m[4 * i + 2];
                        x.w += m[4 * i + 3];
                        S.mom[slot][i] = x;
                    }
                }
                __syncwarp();
            }
        }
        for (int k = lane; k < kept; k += 32) {
            const int gid = S.gid[k];
            if (COMPAT) {
                float m[kMomStride];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const float4 x = S.mom[k][i];
                    m[4 * i] = x.x; m[4 * i + 1] = x.y; m[4 * i + 2] = x.z; m[4 * i + 3] = x.w;
                }
                compat_emit_lane(a, rec_of(S.rec[k][0], S.rec[k][1], S.rec[k][2]), gid, m, ih);
            } else {
                if (DET && S.pidx[k] < 0) continue;
                float4* dst = reinterpret_cast<float4*>(DET ? a.partials + int64_t(S.pidx[k]) * kMomStride
                                                            : a.accum + int64_t(gid) * kMomStride);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    if (DET) dst[i] = S.mom[k][i];
                    else atomicAdd(dst + i, S.mom[k][i]);
                }
                if (DET) a.kept[S.pidx[k]] = 1;
            }
        }
        __syncwarp();
    }
}

template <bool COMPAT, bool DET, int RPL>
__global__ void __launch_bounds__(kThreads, 4) k_backward8(const RenderArgs a) {
    __shared__ __align__(16) BwdStage stage[kWarps];
    __shared__ __align__(16) float grad[8 * kGradStride];
    constexpr int subs = 2 / RPL;
    const int part = blockIdx.x % a.split, rest = blockIdx.x / a.split;
    backward_tile<COMPAT, DET, RPL>(a, rest / subs, rest % subs, stage, grad, part);
}

// ---------------------------------------------------------------------------
// Tile edge 4: a tile is one block; one warp per tile (four tiles per CTA, no CTA barrier), with the walks
// of the 8^3 kernels.  96^3/40k: forward 167 -> 129 us, backward 418 -> 149 us against two voxels per lane
// and a warp per Gaussian.
// ---------------------------------------------------------------------------

// Whether the tile's block may hold a voxel the Gaussian includes (block_mask8 of one block).
__device__ __forceinline__ bool block_hit(const Rec& r, float4 x, int d0, int h0, int w0, bool use_box) {
    if (use_box && !(__fsub_rn(r.c0, x.x) <= float(d0 + 3) && __fadd_rn(r.c0, x.x) >= float(d0) &&
                     __fsub_rn(r.c1, x.y) <= float(h0 + 3) && __fadd_rn(r.c1, x.y) >= float(h0) &&
                     __fsub_rn(r.c2, x.z) <= float(w0 + 3) && __fadd_rn(r.c2, x.z) >= float(w0)))
        return false;
    const float h01 = 0.5f * r.q01x2, h02 = 0.5f * r.q02x2, h12 = 0.5f * r.q12x2;
    const float e0 = centre_offset(d0, r.c0, use_box), e1 = centre_offset(h0, r.c1, use_box),
                e2 = centre_offset(w0, r.c2, use_box);
    return !plane_separates(fmaf(r.q00, e0, fmaf(h01, e1, h02 * e2)), fmaf(h01, e0, fmaf(r.q11, e1, h12 * e2)),
                            fmaf(h02, e0, fmaf(h12, e1, r.q22 * e2)), e0, e1, e2, x.w, plane_factor(x.w));
}

// A listed Gaussian of a 4^3 tile and whether its block is kept.
template <bool COMPAT>
__device__ __forceinline__ bool load_hit4(const RenderArgs& a, int gid, int d0, int h0, int w0, const float ih[3], Rec& r) {
    r = load_rec<COMPAT>(a, gid, ih);
    const float4 x = COMPAT ? make_float4(0.f, 0.f, 0.f, plane_threshold(r)) : __ldg(a.ext + gid);
    return block_hit(r, x, d0, h0, w0, !COMPAT);
}

// A chunk of a tile's list: two positions per lane, loaded together (one at a time 10% slower; copying the
// next chunk's records to shared memory during the walk, cp.async, 10% slower too).
constexpr int kFwd4Chunk = 64;

struct __align__(16) FwdStage4 {
    float4 rec[kFwd4Chunk + 12][kFwdRec];
};

template <bool COMPAT, bool PLANAR>
__global__ void __launch_bounds__(kThreads, 5) k_forward4(const RenderArgs a) {
    __shared__ FwdStage4 stage[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t tile = int64_t(blockIdx.x) * kWarps + warp;
    if (tile >= a.ntiles) return;  // warp-uniform; no CTA barrier below
    int d0, h0, w0;
    decode_tile(a, tile, d0, h0, w0);
    const int2 rg = a.ranges[tile];
    float ih[3];
    compat_ih<COMPAT>(a, ih);
    BlockSums sums = block_sums(d0, h0, w0, lane);
    FwdStage4& S = stage[warp];
    int rank = 0;  // of the tile's next kept Gaussian, modulo four
    int next[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) next[p] = rg.x + 32 * p + lane < rg.y ? __ldg(a.pair_ids + rg.x + 32 * p + lane) : 0;
    for (int base = rg.x; base < rg.y; base += kFwd4Chunk) {
        // kept Gaussians from the front, the ones the cull drops (only without it) from the back
        constexpr int kBack = kFwd4Chunk + 8;
        int n = rank, back = kBack;
        bool bad = false;
        if (lane < rank) store_null_rec(S.rec[lane]);
        Rec r[2];
        bool hit[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int at = base + 32 * p + lane;
            hit[p] = false;
            if (at < rg.y) {
                hit[p] = load_hit4<COMPAT>(a, next[p], d0, h0, w0, ih, r[p]);
                bad |= not_finite(r[p].rho_r) || not_finite(r[p].rho_i);
            }
            if (at + kFwd4Chunk < rg.y) next[p] = __ldg(a.pair_ids + at + kFwd4Chunk);
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const unsigned kept = __ballot_sync(kFull, hit[p]);
            if (hit[p]) store_fwd_rec(S.rec[n + __popc(kept & ((1u << lane) - 1u))], r[p]);
            n += __popc(kept);
            if (!a.cull) {
                const bool miss = base + 32 * p + lane < rg.y && !hit[p];
                const unsigned drop = __ballot_sync(kFull, miss);
                if (miss) store_fwd_rec(S.rec[back - 1 - __popc(drop & ((1u << lane) - 1u))], r[p]);
                back -= __popc(drop);
            }
        }
        rank = n & 3;
        const int back_n = kBack - back;
        if (lane < ((-n) & 3)) store_null_rec(S.rec[n + lane]);
        if (lane < ((-back_n) & 3)) store_null_rec(S.rec[kBack + lane]);
        __syncwarp();
        n = (n + 3) & ~3;
        if (__any_sync(kFull, bad)) {
            BlockSums copy = sums;
            add_gaussians_guarded(copy, &S.rec[0][0], nullptr, n, lane);
            add_gaussians_guarded(copy, &S.rec[back][0], nullptr, (back_n + 3) & ~3, lane);
            sums = copy;
        } else {
            add_gaussians<false>(sums, &S.rec[0][0], nullptr, n, lane);
            if (back_n) add_gaussians<false>(sums, &S.rec[back][0], nullptr, (back_n + 3) & ~3, lane);
        }
        __syncwarp();
    }
    store_block<PLANAR>(a, sums, d0, h0, w0, lane);
}

constexpr int kBwd4Ring = 64;

struct __align__(16) BwdStage4 {
    float4 rec[kBwd4Ring][3];
    float grad[2 * kBlkVox];
    int32_t gid[kBwd4Ring];
    int32_t pidx[kBwd4Ring];  // deterministic: emission index of the pair
};

template <bool COMPAT, bool DET>
__global__ void __launch_bounds__(kThreads, 4) k_backward4(const RenderArgs a) {
    __shared__ BwdStage4 stage[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t tile = int64_t(blockIdx.x) * kWarps + warp;
    if (tile >= a.ntiles) return;  // warp-uniform; no CTA barrier below
    const int2 rg = a.ranges[tile];
    if (rg.x >= rg.y) return;
    int d0, h0, w0;
    decode_tile(a, tile, d0, h0, w0);
    float ih[3];
    compat_ih<COMPAT>(a, ih);
    BwdStage4& S = stage[warp];
    bool guard = false;
    {  // the tile's upstream gradient: a lane takes half a row
        const int i = lane >> 3, j = (lane >> 1) & 3, k0 = 2 * (lane & 1);
        const int gd = d0 + i, gh = h0 + j, gw = w0 + k0;
        const bool row_ok = gd < a.d && gh < a.h;
        const int64_t flat = (int64_t(gd) * a.h + gh) * a.w + gw;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float2 x = make_float2(0.f, 0.f);
            if (row_ok && gw + k < a.w)
                x = COMPAT ? make_float2(__ldg(a.gv_r + flat + k), __ldg(a.gv_i + flat + k))
                           : __ldg(reinterpret_cast<const float2*>(a.gvol) + flat + k);
            guard |= !(fabsf(x.x) <= kBig && fabsf(x.y) <= kBig);
            S.grad[grad_at(i, j, k0 + k)] = x.x;
            S.grad[grad_at(i, j, k0 + k) + 2] = x.y;
        }
        guard = __any_sync(kFull, guard);
    }
    const float v0 = float(d0), v1 = float(h0), v2 = float(w0);
    // the kept Gaussians wait in a ring until there is one for every lane (or no more to come)
    int head = 0, tail = 0;
    int next = rg.x + lane < rg.y ? __ldg(a.pair_ids + rg.x + lane) : 0;
    for (int base = rg.x; base < rg.y || head < tail;) {
        for (; base < rg.y && tail - head < 32; base += 32) {
            const int gid = next;
            if (base + 32 + lane < rg.y) next = __ldg(a.pair_ids + base + 32 + lane);
            const bool listed = base + lane < rg.y;
            Rec r;
            bool hit = false;
            if (listed) {
                hit = load_hit4<COMPAT>(a, gid, d0, h0, w0, ih, r) || !a.cull;
            }
            const unsigned kept = __ballot_sync(kFull, hit);
            if (hit) {
                const int at = (tail + __popc(kept & ((1u << lane) - 1u))) & (kBwd4Ring - 1);
#pragma unroll
                for (int i = 0; i < 3; ++i) S.rec[at][i] = rec_quad(r, i);
                S.gid[at] = gid;
                if (DET) S.pidx[at] = emission_index(a, gid, d0 >> 2, h0 >> 2, w0 >> 2);
            }
            tail += __popc(kept);
        }
        __syncwarp();
        if (head == tail) break;  // nothing kept to the end of the list
        const bool on = lane < tail - head;
        const int at = (head + min(lane, tail - head - 1)) & (kBwd4Ring - 1);
        const Rec g = rec_of(S.rec[at][0], S.rec[at][1], S.rec[at][2]);
        const int gid = S.gid[at];
        float m[kMomStride];
        moments_of(g, S.grad, v0, v1, v2, guard, m);
        if (on && !(DET && S.pidx[at] < 0)) {
            if (COMPAT) {
                compat_emit_lane(a, g, gid, m, ih);
            } else {
                float4* dst = reinterpret_cast<float4*>(DET ? a.partials + int64_t(S.pidx[at]) * kMomStride
                                                            : a.accum + int64_t(gid) * kMomStride);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const float4 x = make_float4(m[4 * i], m[4 * i + 1], m[4 * i + 2], m[4 * i + 3]);
                    if (DET) dst[i] = x;
                    else atomicAdd(dst + i, x);
                }
                if (DET) a.kept[S.pidx[at]] = 1;
            }
        }
        head = min(head + 32, tail);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Generic tile edge: one voxel per thread, Gaussians staged per CTA.
// ---------------------------------------------------------------------------

template <bool COMPAT, bool PLANAR>
__global__ void __launch_bounds__(kThreads) k_forward_generic(const RenderArgs a) {
    __shared__ Rec srec[kThreads];
    const int64_t tile = blockIdx.x;
    int d0, h0, w0;
    decode_tile(a, tile, d0, h0, w0);
    const int2 rg = a.ranges[tile];
    const int ts = a.ts;
    const int nvox = ts * ts * ts;
    float ih[3];
    compat_ih<COMPAT>(a, ih);
    for (int c0 = 0; c0 < nvox; c0 += kThreads) {  // uniform trip count
        const int vid = c0 + threadIdx.x;
        const int ld = vid / (ts * ts), lh = (vid / ts) % ts, lw = vid % ts;
        const int gd = d0 + ld, gh = h0 + lh, gw = w0 + lw;
        const bool valid = vid < nvox && gd < a.d && gh < a.h && gw < a.w;
        const float v0 = float(gd), v1 = float(gh), v2 = float(gw);
        float ar = 0.f, ai = 0.f;
        for (int base = rg.x; base < rg.y; base += kThreads) {  // uniform trip count
            const int cnt = min(kThreads, rg.y - base);
            __syncthreads();
            if (threadIdx.x < cnt) srec[threadIdx.x] = load_rec<COMPAT>(a, __ldg(a.pair_ids + base + threadIdx.x), ih);
            __syncthreads();
            for (int j = 0; j < cnt; ++j) {
                const Rec g = srec[j];
                const float e0 = __fsub_rn(v0, g.c0), e1 = __fsub_rn(v1, g.c1), e2 = __fsub_rn(v2, g.c2);
                const float m = row_m(g.q22, row_a(g, e0, e1), row_b(g, e0, e1), e2);
                if (m <= kCut) {
                    const float wgt = ex2_approx(m * kNegHalfLog2e);
                    ar = fmaf(wgt, g.rho_r, ar);
                    ai = fmaf(wgt, g.rho_i, ai);
                }
            }
        }
        if (valid) {
            const int64_t flat = (int64_t(gd) * a.h + gh) * a.w + gw;
            if (PLANAR) {
                a.vol_r[flat] = ar;
                a.vol_i[flat] = ai;
            } else {
                reinterpret_cast<float2*>(a.vol)[flat] = make_float2(ar, ai);
            }
        }
    }
}

template <bool COMPAT, bool DET>
__global__ void __launch_bounds__(kThreads) k_backward_generic(const RenderArgs a) {
    __shared__ Rec srec[32];
    __shared__ int sgid[32];
    __shared__ int32_t sidx[32];
    __shared__ float sred[kWarps][kMom];
    const int64_t tile = blockIdx.x;
    const int2 rg = a.ranges[tile];
    if (rg.x >= rg.y) return;
    int d0, h0, w0;
    decode_tile(a, tile, d0, h0, w0);
    const int ts = a.ts;
    const int nvox = ts * ts * ts;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float ih[3];
    compat_ih<COMPAT>(a, ih);
    for (int base = rg.x; base < rg.y; base += 32) {
        const int cnt = min(32, rg.y - base);
        __syncthreads();
        if (threadIdx.x < cnt) {
            const int gid = __ldg(a.pair_ids + base + threadIdx.x);
            sgid[threadIdx.x] = gid;
            srec[threadIdx.x] = load_rec<COMPAT>(a, gid, ih);
            if (DET) sidx[threadIdx.x] = emission_index(a, gid, d0 / ts, h0 / ts, w0 / ts);
        }
        __syncthreads();
        for (int j = 0; j < cnt; ++j) {
            const Rec g = srec[j];
            float v[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = 0.f;
            for (int vid = threadIdx.x; vid < nvox; vid += kThreads) {
                const int ld = vid / (ts * ts), lh = (vid / ts) % ts, lw = vid % ts;
                const int gd = d0 + ld, gh = h0 + lh, gw = w0 + lw;
                if (gd >= a.d || gh >= a.h || gw >= a.w) continue;
                const float e0 = __fsub_rn(float(gd), g.c0), e1 = __fsub_rn(float(gh), g.c1);
                const float e2 = __fsub_rn(float(gw), g.c2);
                const float m = row_m(g.q22, row_a(g, e0, e1), row_b(g, e0, e1), e2);
                if (!(m <= kCut)) continue;
                const int64_t flat = (int64_t(gd) * a.h + gh) * a.w + gw;
                float gr, gi;
                if (COMPAT) {
                    gr = __ldg(a.gv_r + flat);
                    gi = __ldg(a.gv_i + flat);
                } else {
                    const float2 x = __ldg(reinterpret_cast<const float2*>(a.gvol) + flat);
                    gr = x.x;
                    gi = x.y;
                }
                const float wgt = ex2_approx(m * kNegHalfLog2e);
                const float av = wgt * fmaf(-0.5f * g.rho_i, gi, (-0.5f * g.rho_r) * gr);
                v[0] = fmaf(wgt, gr, v[0]);
                v[1] = fmaf(wgt, gi, v[1]);
                v[2] = fmaf(av, e0, v[2]);
                v[3] = fmaf(av, e1, v[3]);
                v[4] = fmaf(av, e2, v[4]);
                v[5] = fmaf(av * e0, e0, v[5]);
                v[6] = fmaf(av * e0, e1, v[6]);
                v[7] = fmaf(av * e0, e2, v[7]);
                v[8] = fmaf(av * e1, e1, v[8]);
                v[9] = fmaf(av * e1, e2, v[9]);
                v[10] = fmaf(av * e2, e2, v[10]);
            }
            const float tot = warp_reduce_scatter16(v, lane);
            if (!(lane & 1) && (lane >> 1) < kMom) sred[warp][lane >> 1] = tot;
            __syncthreads();
            // warp 0 combines the four warps in a fixed order
            if (warp == 0) {
                float t = 0.f;
                if (lane < kMom) t = ((sred[0][lane] + sred[1][lane]) + sred[2][lane]) + sred[3][lane];
                // compat_emit expects moment i in lane 2i
                const float spread = __shfl_sync(kFull, t, lane >> 1);
                const int gid = sgid[j];
                if (COMPAT) {
                    compat_emit(a, g, gid, spread, lane, ih);
                } else if (DET) {
                    if (lane < kMom && sidx[j] >= 0) a.partials[int64_t(sidx[j]) * kMomStride + lane] = t;
                    if (lane == 0 && sidx[j] >= 0) a.kept[sidx[j]] = 1;
                } else {
                    if (lane < kMom) atomicAdd(a.accum + int64_t(gid) * kMomStride + lane, t);
                }
            }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// Finalize: moments -> dL/d(positions, scales, rotations, density).
// Chain rule of tile_voxelizer.py:284-290 and :77-84 (the torch autograd
// tail of the reference), in FP32.
// ---------------------------------------------------------------------------

// What the deterministic gather reads of one volume.
struct DetView {
    const int4* boxes;
    const int64_t* offsets;
    const float* partials;
    const uint8_t* kept;
    int64_t capacity;
};
__device__ __forceinline__ DetView det_view(const RenderArgs& a) {
    return DetView{a.boxes, a.offsets, a.partials, a.kept, a.capacity};
}

// Deterministic moments of 4 R Gaussians (base .. base + 4 R - 1 of `total`), R rounds
// of four with eight lanes each: a Gaussian's per-pair partials sit contiguously at
// its emission indices, in tile raster order, and the pairs the backward kept are
// marked.  Lane l of the eight takes entries l, l + 8, ... and a fixed xor tree sums
// the lanes (a Gaussian of more than kGatherGroup pairs: the whole warp, l + 32, ...).
// Either order depends only on the tile box, so the result is bitwise reproducible
// and does not depend on R.  Lane 4 r + q ends with the moments of round r's
// Gaussian q.  `locate(x, view, g)`: volume and row of Gaussian x.
constexpr int kGatherGroup = 256;

__device__ __forceinline__ void add_partial(float mo[kMom], const float* src) {
    const float4* p = reinterpret_cast<const float4*>(src);
    const float4 x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
    mo[0] += x.x; mo[1] += x.y; mo[2] += x.z; mo[3] += x.w;
    mo[4] += y.x; mo[5] += y.y; mo[6] += y.z; mo[7] += y.w;
    mo[8] += z.x; mo[9] += z.y; mo[10] += z.z;
}

// First emission index of a Gaussian's pairs and how many of them have partials.
__device__ __forceinline__ int det_pairs(const DetView& v, int64_t g, int64_t& first) {
    first = v.offsets[g];
    const int64_t left = v.capacity - first;  // past the capacity (overflow, flagged) there are none
    return int(left <= 0 ? 0 : min(int64_t(v.boxes[g].w), left));
}

template <int R, typename Locate>
__device__ __forceinline__ void gather_det(const Locate& locate, int64_t base, int64_t total, int lane, float mo[kMom]) {
#pragma unroll
    for (int i = 0; i < kMom; ++i) mo[i] = 0.f;
    // lane 4 r + q: where its Gaussian's marks and partials are
    unsigned long long my_kept = 0, my_partials = 0;
    int my_cnt = 0;
    if (lane < 4 * R && base + lane < total) {
        DetView v;
        int64_t g, first;
        locate(base + lane, v, g);
        my_cnt = det_pairs(v, g, first);
        my_kept = (unsigned long long)(v.kept + first);
        my_partials = (unsigned long long)(v.partials + first * kMomStride);
    }
#pragma unroll 1
    for (int r = 0; r < R; ++r) {
        const int from = 4 * r + (lane >> 3);
        const uint8_t* kept = reinterpret_cast<const uint8_t*>(__shfl_sync(kFull, my_kept, from));
        const float* partials = reinterpret_cast<const float*>(__shfl_sync(kFull, my_partials, from));
        const int cnt = __shfl_sync(kFull, my_cnt, from);
        float part[kMom];
#pragma unroll
        for (int i = 0; i < kMom; ++i) part[i] = 0.f;
        if (cnt <= kGatherGroup) {
            for (int c = lane & 7; c < cnt; c += 16) {  // two entries in flight
                const bool on0 = __ldg(kept + c), on1 = c + 8 < cnt && __ldg(kept + c + 8);
                if (on0) add_partial(part, partials + c * kMomStride);
                if (on1) add_partial(part, partials + (c + 8) * kMomStride);
            }
        }
#pragma unroll
        for (int off = 4; off >= 1; off >>= 1)
#pragma unroll
            for (int i = 0; i < kMom; ++i) part[i] += __shfl_xor_sync(kFull, part[i], off);
        for (unsigned big = __ballot_sync(kFull, cnt > kGatherGroup && (lane & 7) == 0); big; big &= big - 1) {
            const int src = __ffs(big) - 1;
            const uint8_t* bk = reinterpret_cast<const uint8_t*>(__shfl_sync(kFull, (unsigned long long)kept, src));
            const float* bp = reinterpret_cast<const float*>(__shfl_sync(kFull, (unsigned long long)partials, src));
            const int n = __shfl_sync(kFull, cnt, src);
            float all[kMom];
#pragma unroll
            for (int i = 0; i < kMom; ++i) all[i] = 0.f;
            for (int c = lane; c < n; c += 32)
                if (__ldg(bk + c)) add_partial(all, bp + int64_t(c) * kMomStride);
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
                for (int i = 0; i < kMom; ++i) all[i] += __shfl_xor_sync(kFull, all[i], off);
            if ((lane & ~7) == src)
#pragma unroll
                for (int i = 0; i < kMom; ++i) part[i] = all[i];
        }
#pragma unroll
        for (int i = 0; i < kMom; ++i) {
            const float t = __shfl_sync(kFull, part[i], (lane & 3) * 8);
            if ((lane >> 2) == r) mo[i] = t;
        }
    }
}

// Moments of one Gaussian from the atomic accumulators, which are cleared once
// read: the preprocess clears them too, so the atomic backward always starts
// from zero without a memset of its own.
__device__ __forceinline__ void take_moments(const RenderArgs& a, int64_t g, float mo[kMom]) {
    float4* acc4 = reinterpret_cast<float4*>(a.accum + g * kMomStride);
    const float4 x = acc4[0], y = acc4[1], z = acc4[2];
    acc4[0] = acc4[1] = acc4[2] = make_float4(0.f, 0.f, 0.f, 0.f);
    mo[0] = x.x; mo[1] = x.y; mo[2] = x.z; mo[3] = x.w;
    mo[4] = y.x; mo[5] = y.y; mo[6] = y.z; mo[7] = y.w;
    mo[8] = z.x; mo[9] = z.y; mo[10] = z.z;
}

// Chain rule of one Gaussian from its 11 moments.
__device__ __forceinline__ void finalize_one(const RenderArgs& a, int64_t g, const float mo[kMom]) {
    const gsv_params& p = a.prm;
    const gsv_grads& out = a.grd;
    const Rec R = a.recs[g];
    // dL/dcenter_vox, then dcenter/dpositions = 0.5 * shape = hs   (:284).
    // The reference sums this over included pairs only: a Gaussian with none
    // (e.g. NaN coefficients) gets exactly 0, not 0 * NaN.
    const bool has_center = mo[2] != 0.f || mo[3] != 0.f || mo[4] != 0.f;
    const float dc0 = has_center ? -(2.0f * R.q00 * mo[2] + R.q01x2 * mo[3] + R.q02x2 * mo[4]) : 0.f;
    const float dc1 = has_center ? -(R.q01x2 * mo[2] + 2.0f * R.q11 * mo[3] + R.q12x2 * mo[4]) : 0.f;
    const float dc2 = has_center ? -(R.q02x2 * mo[2] + R.q12x2 * mo[3] + 2.0f * R.q22 * mo[4]) : 0.f;
    out.positions[g * 3 + 0] = dc0 * a.hs[0];
    out.positions[g * 3 + 1] = dc1 * a.hs[1];
    out.positions[g * 3 + 2] = dc2 * a.hs[2];
    out.density_r[g * a.dstride] = mo[0];
    out.density_i[g * a.dstride] = mo[1];
    // dL/dM (normalised units), symmetric.
    float G[9];
    G[0] = mo[5] * a.ih[0] * a.ih[0];
    G[1] = G[3] = mo[6] * a.ih[0] * a.ih[1];
    G[2] = G[6] = mo[7] * a.ih[0] * a.ih[2];
    G[4] = mo[8] * a.ih[1] * a.ih[1];
    G[5] = G[7] = mo[9] * a.ih[1] * a.ih[2];
    G[8] = mo[10] * a.ih[2] * a.ih[2];
    // Rebuild R(qn), si = 1/(s+1e-8) and T = R diag(si).
    float q[4], s[3];
#pragma unroll
    for (int k = 0; k < 4; ++k) q[k] = p.rotations[g * 4 + k];
#pragma unroll
    for (int k = 0; k < 3; ++k) s[k] = p.scales[g * 3 + k];
    const float nrm = sqrtf(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
    const float den = nrm + 1e-8f;
    const float w = q[0] / den, x = q[1] / den, y = q[2] / den, z = q[3] / den;
    float r[9];
    r[0] = 1.f - 2.f * y * y - 2.f * z * z;
    r[1] = 2.f * x * y - 2.f * z * w;
    r[2] = 2.f * x * z + 2.f * y * w;
    r[3] = 2.f * x * y + 2.f * z * w;
    r[4] = 1.f - 2.f * x * x - 2.f * z * z;
    r[5] = 2.f * y * z - 2.f * x * w;
    r[6] = 2.f * x * z - 2.f * y * w;
    r[7] = 2.f * y * z + 2.f * x * w;
    r[8] = 1.f - 2.f * x * x - 2.f * y * y;
    float si[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) si[j] = 1.0f / (s[j] + 1e-8f);
    // dL/dT = (G + G^T) T = 2 G T
    float gr[9], gsi[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k) acc += G[i * 3 + k] * (r[k * 3 + j] * si[j]);
            const float gt = 2.0f * acc;
            gr[i * 3 + j] = gt * si[j];
            gsi[j] += gt * r[i * 3 + j];
        }
#pragma unroll
    for (int j = 0; j < 3; ++j) out.scales[g * 3 + j] = -gsi[j] * si[j] * si[j];
    float gn[4];
    gn[0] = 2.f * (-z * gr[1] + y * gr[2] + z * gr[3] - x * gr[5] - y * gr[6] + x * gr[7]);
    gn[1] = 2.f * (y * gr[1] + z * gr[2] + y * gr[3] - 2.f * x * gr[4] - w * gr[5] + z * gr[6] + w * gr[7] -
                   2.f * x * gr[8]);
    gn[2] = 2.f * (-2.f * y * gr[0] + x * gr[1] + w * gr[2] + x * gr[3] + z * gr[5] - w * gr[6] + z * gr[7] -
                   2.f * y * gr[8]);
    gn[3] = 2.f * (-2.f * z * gr[0] - w * gr[1] + x * gr[2] + w * gr[3] - 2.f * z * gr[4] + y * gr[5] +
                   x * gr[6] + y * gr[7]);
    const float dot = gn[0] * w + gn[1] * x + gn[2] * y + gn[3] * z;
    const float corr = nrm > 0.f ? dot / (nrm * den) : 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) out.rotations[g * 4 + k] = gn[k] / den - q[k] * corr;
}

__global__ void __launch_bounds__(256) k_finalize(const RenderArgs a) {
    const int64_t g = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (g >= a.prm.n) return;
    float mo[kMom];
    take_moments(a, g, mo);
    finalize_one(a, g, mo);
}

// The deterministic backward's gather and chain rule, 4 R Gaussians per warp.
template <int R>
__global__ void __launch_bounds__(256) k_finalize_det(const RenderArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t base = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * (4 * R);
    const DetView view = det_view(a);
    float mo[kMom];
    gather_det<R>([&](int64_t x, DetView& v, int64_t& g) { v = view; g = x; }, base, a.prm.n, lane, mo);
    if (lane < 4 * R && base + lane < a.prm.n) finalize_one(a, base + lane, mo);
}

// ---------------------------------------------------------------------------
// Batched persistent launches: many volumes, one launch.  The descriptor
// table (one RenderArgs per volume) and prefix sums of tiles, Gaussians and
// pair capacities live in device memory; CTAs pull global tile indices from
// an atomic counter until the work runs out.
// ---------------------------------------------------------------------------

struct BatchTable {
    RenderArgs* items;
    int64_t* tile_prefix;   // [count + 1]
    int64_t* gauss_prefix;  // [count + 1]
    int64_t* cap_prefix;    // [count + 1]  deterministic: 16-byte words of marks
    unsigned long long* counters;  // [2]: forward, backward work counters
    int count;
    int det;
};

__device__ __forceinline__ int find_item(const int64_t* prefix, int count, int64_t x) {
    int lo = 0, hi = count;  // largest i with prefix[i] <= x
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(256, 4) k_forward8_batched(const BatchTable t) {
    __shared__ FwdStage<8> stage;
    __shared__ long long s_next;
    const int64_t total = t.tile_prefix[t.count];
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_next = (long long)atomicAdd(&t.counters[0], 1ull);
        __syncthreads();
        const int64_t gt = s_next;
        if (gt >= total) break;
        const int i = find_item(t.tile_prefix, t.count, gt);
        forward_tile<false, false, 2>(t.items[i], gt - t.tile_prefix[i], 0, stage);
    }
}

template <bool DET>
__global__ void __launch_bounds__(kThreads, 4) k_backward8_batched(const BatchTable t) {
    __shared__ __align__(16) BwdStage stage[kWarps];
    __shared__ __align__(16) float grad[8 * kGradStride];
    __shared__ long long s_next;
    const int64_t total = t.tile_prefix[t.count];
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_next = (long long)atomicAdd(&t.counters[1], 1ull);
        __syncthreads();
        const int64_t gt = s_next;
        if (gt >= total) break;
        const int i = find_item(t.tile_prefix, t.count, gt);
        backward_tile<false, DET, 2>(t.items[i], gt - t.tile_prefix[i], 0, stage, grad, 0);
    }
}

__global__ void __launch_bounds__(256) k_finalize_batched(const BatchTable t) {
    const int64_t total = t.gauss_prefix[t.count];
    for (int64_t x = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; x < total;
         x += int64_t(gridDim.x) * blockDim.x) {
        const int i = find_item(t.gauss_prefix, t.count, x);
        float mo[kMom];
        take_moments(t.items[i], x - t.gauss_prefix[i], mo);
        finalize_one(t.items[i], x - t.gauss_prefix[i], mo);
    }
}

// k_finalize_det over every volume's Gaussians.
__global__ void __launch_bounds__(256) k_finalize_det_batched(const BatchTable t) {
    constexpr int R = 4;
    const int lane = threadIdx.x & 31;
    const int64_t total = t.gauss_prefix[t.count];
    const int64_t warps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t base = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * (4 * R); base < total;
         base += warps * (4 * R)) {  // warp-uniform
        float mo[kMom];
        gather_det<R>(
            [&](int64_t x, DetView& v, int64_t& g) {
                const int i = find_item(t.gauss_prefix, t.count, x);
                v = det_view(t.items[i]);
                g = x - t.gauss_prefix[i];
            },
            base, total, lane, mo);
        if (lane < 4 * R && base + lane < total) {
            const int i = find_item(t.gauss_prefix, t.count, base + lane);
            finalize_one(t.items[i], base + lane - t.gauss_prefix[i], mo);
        }
    }
}

// Clears every volume's marks of kept pairs (16 at a time; the marks' buffer is longer than its capacity).
__global__ void __launch_bounds__(256) k_clear_kept_batched(const BatchTable t) {
    const int64_t total = t.cap_prefix[t.count];
    for (int64_t x = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; x < total; x += int64_t(gridDim.x) * blockDim.x) {
        const int i = find_item(t.cap_prefix, t.count, x);
        reinterpret_cast<uint4*>(t.items[i].kept)[x - t.cap_prefix[i]] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// ---------------------------------------------------------------------------
// Work census of the tile-8 kernels (diagnostic, no gradients): per listed
// (tile, Gaussian) pair it replays the render kernels' decisions with their
// arithmetic -- the 4x4x4 blocks kept, the row-form quadratic and the FP32
// cutoff -- and counts
//   out[0]  included candidates (m <= 9, voxel inside the volume),
//   out[1]  candidates the kernels evaluate m for (voxels of kept blocks),
//   out[2]  exponentials they issue (every voxel of a kept block),
//   out[3]  kept blocks without any included voxel.
// The inclusion count covers every listed block, kept or not, so it also
// checks that the cull drops no included voxel.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_count_work(const RenderArgs a, unsigned long long* out) {
    const int64_t tile = blockIdx.x;
    const int2 rg = a.ranges[tile];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int d0, h0, w0;
    decode_tile(a, tile, d0, h0, w0);
    unsigned long long c_inc = 0, c_eval = 0, c_empty = 0;
    for (int p = rg.x + warp; p < rg.y; p += kWarps) {
        const int gid = __ldg(a.pair_ids + p);
        float ih[3];
        compat_ih<false>(a, ih);
        const Rec g = load_rec<false>(a, gid, ih);
        const unsigned in = a.cull ? block_mask8(g, __ldg(a.ext + gid), d0, h0, w0, true) : 0xffu;
        for (int b = 0; b < 8; ++b) {
            bool any = false;
#pragma unroll
            for (int t = 0; t < kBlkVox / 32; ++t) {
                const int v = lane + 32 * t;
                const int gd = d0 + (b >> 2) * kBlk + (v >> 4), gh = h0 + ((b >> 1) & 1) * kBlk + ((v >> 2) & 3),
                          gw = w0 + (b & 1) * kBlk + (v & 3);
                const float e0 = __fsub_rn(float(gd), g.c0), e1 = __fsub_rn(float(gh), g.c1);
                const float m = row_m(g.q22, row_a(g, e0, e1), row_b(g, e0, e1), __fsub_rn(float(gw), g.c2));
                const bool inside = m <= kCut;
                c_inc += (inside && gd < a.d && gh < a.h && gw < a.w) ? 1 : 0;
                any |= inside;
            }
            any = __any_sync(kFull, any);
            if ((in >> b) & 1u) {
                c_eval += kBlkVox / 32;
                if (!any && lane == 0) c_empty += 1;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c_inc += __shfl_xor_sync(kFull, c_inc, o);
        c_eval += __shfl_xor_sync(kFull, c_eval, o);
        c_empty += __shfl_xor_sync(kFull, c_empty, o);
    }
    if (lane == 0) {
        atomicAdd(out, c_inc);
        atomicAdd(out + 1, c_eval);
        atomicAdd(out + 2, c_eval);
        atomicAdd(out + 3, c_empty);
    }
}

int grid_for(int64_t items, int block) {
    int64_t g = (items + block - 1) / block;
    return int(g < 1 ? 1 : g);
}

template <typename T>
const T* cat(const void* base, size_t off) {
    return reinterpret_cast<const T*>(static_cast<const char*>(base) + off);
}
template <typename T>
T* mat(void* base, size_t off) {
    return reinterpret_cast<T*>(static_cast<char*>(base) + off);
}

void fill_shape(RenderArgs& a, gsv_shape s) {
    a.d = s.d; a.h = s.h; a.w = s.w; a.ts = s.tile_size;
    a.nth = (s.h + s.tile_size - 1) / s.tile_size;
    a.ntw = (s.w + s.tile_size - 1) / s.tile_size;
    a.ntiles = int64_t((s.d + s.tile_size - 1) / s.tile_size) * a.nth * a.ntw;
    a.chunk = 32;
    a.cull = 1;
    a.dstride = 1;
    // Backward, 8^3 tiles: 592 CTAs are resident, so with few tiles a long list is worth two CTAs, with
    // many it only adds half-filled groups.  Measured with 1 and 2 CTAs, a second one from 512 list
    // positions on, us: 128x128x96/50k, 3072 tiles 208 and 192; 128x128x96/500k 468 and 429; 165^3/155k,
    // 9261 tiles 526 and 537; 256x256x160/2M, 20480 tiles 2253 and 2330.  Below two resident rounds
    // shorter lists are worth it too (from 256 on: 64^3/20k, 512 tiles 43 and 40; 100x84x60/20k, 1144
    // tiles 113 and 88).
    a.split = a.ntiles < 8 * 592 ? 2 : 1;
    a.part = a.ntiles < 2 * 592 ? 256 : 512;
    const float sh[3] = {float(s.d), float(s.h), float(s.w)};
    for (int k = 0; k < 3; ++k) {
        a.hs[k] = sh[k] * 0.5f;
        a.ih[k] = 1.0f / a.hs[k];
    }
}

bool shape_ok(int32_t ts, int32_t d, int32_t h, int32_t w) {
    return ts > 0 && d > 0 && h > 0 && w > 0 && d < (1 << 24) && h < (1 << 24) && w < (1 << 24);
}

}  // namespace

extern "C" {

int gsv_forward(gsv_shape shape, int64_t n, const void* ws_gauss, const void* ws_pairs,
                int64_t capacity, float* volume, void* stream) {
    return gsv_forward_ex(shape, n, ws_gauss, ws_pairs, capacity, volume, nullptr, stream);
}

static bool tuning_ok(const gsv_tuning* t) {
    return !t || ((t->rows_per_lane == 1 || t->rows_per_lane == 2) && t->chunk >= 1 && t->chunk <= 32 &&
                  (t->split == 0 || t->split == 1 || t->split == 2 || t->split == 4));
}

int gsv_forward_ex(gsv_shape shape, int64_t n, const void* ws_gauss, const void* ws_pairs, int64_t capacity,
                   float* volume, const gsv_tuning* tuning, void* stream) {
    if (!tuning_ok(tuning)) return GSV_ERR_INVALID_ARGUMENT;
    GaussLayout G;
    PairLayout P;
    int64_t ntiles = 0;
    if (layout_for(shape, n, capacity, 0, &G, &P, &ntiles) != GSV_OK || !ws_gauss || !volume ||
        (capacity > 0 && !ws_pairs))
        return GSV_ERR_INVALID_ARGUMENT;
    if (ntiles > int64_t(INT32_MAX)) return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RenderArgs a{};
    fill_shape(a, shape);
    a.recs = cat<Rec>(ws_gauss, G.rec);
    a.ext = cat<float4>(ws_gauss, G.ext);
    a.ranges = cat<int2>(ws_gauss, G.ranges);
    a.pair_ids = capacity > 0 ? cat<int32_t>(ws_pairs, P.vals_out) : nullptr;
    a.vol = volume;
    const int rpl = tuning ? tuning->rows_per_lane : 2;
    if (tuning) {
        a.chunk = tuning->chunk;
        a.cull = !(tuning->flags & GSV_TUNE_NO_CULL);
    }
    if (shape.tile_size == 8 && rpl == 2) k_forward8<false, false, 2><<<unsigned(ntiles), 256, 0, st>>>(a);
    else if (shape.tile_size == 8) k_forward8<false, false, 1><<<unsigned(2 * ntiles), 128, 0, st>>>(a);
    else if (shape.tile_size == 4)
        k_forward4<false, false><<<unsigned((ntiles + kWarps - 1) / kWarps), kThreads, 0, st>>>(a);
    else k_forward_generic<false, false><<<unsigned(ntiles), kThreads, 0, st>>>(a);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

int gsv_backward(const gsv_params* p, gsv_shape shape, void* ws_gauss, void* ws_pairs,
                 int64_t capacity, const float* grad_volume, const gsv_grads* grads, int flags,
                 void* stream) {
    return gsv_backward_ex(p, shape, ws_gauss, ws_pairs, capacity, grad_volume, grads, flags, nullptr, stream);
}

int gsv_backward_ex(const gsv_params* p, gsv_shape shape, void* ws_gauss, void* ws_pairs, int64_t capacity,
                    const float* grad_volume, const gsv_grads* grads, int flags, const gsv_tuning* tuning,
                    void* stream) {
    return gsv_backward_strided(p, shape, ws_gauss, ws_pairs, capacity, grad_volume, grads, 1, flags, tuning, stream);
}

int gsv_backward_strided(const gsv_params* p, gsv_shape shape, void* ws_gauss, void* ws_pairs, int64_t capacity,
                         const float* grad_volume, const gsv_grads* grads, int64_t density_stride, int flags,
                         const gsv_tuning* tuning, void* stream) {
    if (!tuning_ok(tuning) || density_stride < 1) return GSV_ERR_INVALID_ARGUMENT;
    GaussLayout G;
    PairLayout P;
    int64_t ntiles = 0;
    const bool det = flags & GSV_BACKWARD_DETERMINISTIC;
    if (!p || !grads || layout_for(shape, p->n, capacity, flags, &G, &P, &ntiles) != GSV_OK || !ws_gauss ||
        !grad_volume || (capacity > 0 && !ws_pairs))
        return GSV_ERR_INVALID_ARGUMENT;
    const int64_t n = p->n;
    if (n == 0) return GSV_OK;
    if (!grads->positions || !grads->scales || !grads->rotations || !grads->density_r || !grads->density_i ||
        !p->scales || !p->rotations)
        return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RenderArgs a{};
    fill_shape(a, shape);
    a.recs = cat<Rec>(ws_gauss, G.rec);
    a.ext = cat<float4>(ws_gauss, G.ext);
    a.ranges = cat<int2>(ws_gauss, G.ranges);
    a.pair_ids = capacity > 0 ? cat<int32_t>(ws_pairs, P.vals_out) : nullptr;
    a.gvol = grad_volume;
    a.accum = mat<float>(ws_gauss, G.accum);
    a.partials = det ? mat<float>(ws_pairs, P.partials) : nullptr;
    a.kept = det ? mat<uint8_t>(ws_pairs, P.keys_in) : nullptr;  // the unsorted keys are no longer needed
    a.offsets = cat<int64_t>(ws_gauss, G.offsets);
    a.boxes = cat<int4>(ws_gauss, G.box);
    a.capacity = capacity;
    // The atomic accumulators are zero here: the preprocess clears them and
    // k_finalize clears them again after reading.  The deterministic mode
    // marks the pairs whose partials it writes and does not touch them.
    if (tuning) {
        a.chunk = tuning->chunk;
        a.cull = !(tuning->flags & GSV_TUNE_NO_CULL);
        if (tuning->split > 0) a.split = tuning->split;
    }
    if (ntiles * 2 * a.split > int64_t(INT32_MAX)) return GSV_ERR_INVALID_ARGUMENT;
    const int rpl = (tuning && !det) ? tuning->rows_per_lane : 2;  // deterministic: whole tiles
    const unsigned sp = unsigned(a.split);
    if (capacity > 0) {
        if (det) GSV_CUDA_TRY(cudaMemsetAsync(a.kept, 0, size_t(capacity), st));
        if (shape.tile_size == 8) {
            if (det) k_backward8<false, true, 2><<<unsigned(ntiles) * sp, kThreads, 0, st>>>(a);
            else if (rpl == 2) k_backward8<false, false, 2><<<unsigned(ntiles) * sp, kThreads, 0, st>>>(a);
            else k_backward8<false, false, 1><<<unsigned(2 * ntiles) * sp, kThreads, 0, st>>>(a);
        } else {
            const unsigned g4 = unsigned((ntiles + kWarps - 1) / kWarps);
            if (shape.tile_size == 4 && det) k_backward4<false, true><<<g4, kThreads, 0, st>>>(a);
            else if (shape.tile_size == 4) k_backward4<false, false><<<g4, kThreads, 0, st>>>(a);
            else if (det) k_backward_generic<false, true><<<unsigned(ntiles), kThreads, 0, st>>>(a);
            else k_backward_generic<false, false><<<unsigned(ntiles), kThreads, 0, st>>>(a);
        }
        GSV_LAUNCH_CHECK();
    }
    a.prm = *p;
    a.grd = *grads;
    a.dstride = density_stride;
    // Four Gaussians a warp while the warps are few, 32 (every lane busy in the chain rule) above.  Whole
    // backward with 4 and 32, 11 pairs a Gaussian, us: 30,000 65 and 70; 48,000 84 and 86; 56,000 91 and 91;
    // 65,000 101 and 98; 131,000 189 and 179; 400,000 369 and 320; the same within 1% on other grids.
    if (det && capacity > 0 && n < 57344) k_finalize_det<1><<<grid_for(n, 32), 256, 0, st>>>(a);
    else if (det && capacity > 0) k_finalize_det<8><<<grid_for(n, 256), 256, 0, st>>>(a);
    else k_finalize<<<grid_for(n, 256), 256, 0, st>>>(a);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

int gsv_count_work(gsv_shape shape, int64_t n, const void* ws_gauss, const void* ws_pairs, int64_t capacity,
                   const gsv_tuning* tuning, unsigned long long* out, void* stream) {
    if (!tuning_ok(tuning) || shape.tile_size != 8 || !out) return GSV_ERR_INVALID_ARGUMENT;
    GaussLayout G;
    PairLayout P;
    int64_t ntiles = 0;
    if (layout_for(shape, n, capacity, 0, &G, &P, &ntiles) != GSV_OK || !ws_gauss || (capacity > 0 && !ws_pairs))
        return GSV_ERR_INVALID_ARGUMENT;
    if (ntiles > int64_t(INT32_MAX)) return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    GSV_CUDA_TRY(cudaMemsetAsync(out, 0, 4 * sizeof(unsigned long long), st));
    if (capacity == 0 || n == 0) return GSV_OK;
    RenderArgs a{};
    fill_shape(a, shape);
    a.recs = cat<Rec>(ws_gauss, G.rec);
    a.ext = cat<float4>(ws_gauss, G.ext);
    a.ranges = cat<int2>(ws_gauss, G.ranges);
    a.pair_ids = cat<int32_t>(ws_pairs, P.vals_out);
    if (tuning) a.cull = !(tuning->flags & GSV_TUNE_NO_CULL);
    k_count_work<<<unsigned(ntiles), kThreads, 0, st>>>(a, out);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

int gsv_tile_forward(const float* centers, const float* cov_inv, const float* density_r,
                     const float* density_i, const int32_t* tile_ranges, const int32_t* pair_ids,
                     const float* half_shape, int64_t n, int64_t num_tiles, int32_t tile_size,
                     int32_t d, int32_t h, int32_t w, float* vol_r, float* vol_i, void* stream) {
    if (!shape_ok(tile_size, d, h, w) || n < 0 || !tile_ranges || !half_shape || !vol_r || !vol_i)
        return GSV_ERR_INVALID_ARGUMENT;
    gsv_shape s{d, h, w, tile_size};
    RenderArgs a{};
    fill_shape(a, s);
    if (num_tiles != a.ntiles || num_tiles > int64_t(INT32_MAX)) return GSV_ERR_INVALID_ARGUMENT;
    if (n > 0 && (!centers || !cov_inv || !density_r || !density_i)) return GSV_ERR_INVALID_ARGUMENT;
    a.centers = centers;
    a.cov_inv = cov_inv;
    a.den_r = density_r;
    a.den_i = density_i;
    a.half_shape = half_shape;
    a.ranges = reinterpret_cast<const int2*>(tile_ranges);
    a.pair_ids = pair_ids;
    a.vol_r = vol_r;
    a.vol_i = vol_i;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (tile_size == 8) k_forward8<true, true, 2><<<unsigned(num_tiles), 256, 0, st>>>(a);
    else if (tile_size == 4)
        k_forward4<true, true><<<unsigned((num_tiles + kWarps - 1) / kWarps), kThreads, 0, st>>>(a);
    else k_forward_generic<true, true><<<unsigned(num_tiles), kThreads, 0, st>>>(a);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

int gsv_tile_backward(const float* centers, const float* cov_inv, const float* density_r,
                      const float* density_i, const int32_t* tile_ranges, const int32_t* pair_ids,
                      const float* half_shape, const float* grad_vol_r, const float* grad_vol_i,
                      int64_t n, int64_t num_tiles, int32_t tile_size, int32_t d, int32_t h,
                      int32_t w, float* grad_centers, float* grad_cov_inv, float* grad_den_r,
                      float* grad_den_i, void* stream) {
    if (!shape_ok(tile_size, d, h, w) || n < 0 || !tile_ranges || !half_shape || !grad_vol_r ||
        !grad_vol_i)
        return GSV_ERR_INVALID_ARGUMENT;
    gsv_shape s{d, h, w, tile_size};
    RenderArgs a{};
    fill_shape(a, s);
    if (num_tiles != a.ntiles || num_tiles > int64_t(INT32_MAX)) return GSV_ERR_INVALID_ARGUMENT;
    if (n == 0) return GSV_OK;
    if (!centers || !cov_inv || !density_r || !density_i || !grad_centers || !grad_cov_inv ||
        !grad_den_r || !grad_den_i)
        return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    GSV_CUDA_TRY(cudaMemsetAsync(grad_centers, 0, size_t(n) * 3 * sizeof(float), st));
    GSV_CUDA_TRY(cudaMemsetAsync(grad_cov_inv, 0, size_t(n) * 9 * sizeof(float), st));
    GSV_CUDA_TRY(cudaMemsetAsync(grad_den_r, 0, size_t(n) * sizeof(float), st));
    GSV_CUDA_TRY(cudaMemsetAsync(grad_den_i, 0, size_t(n) * sizeof(float), st));
    a.centers = centers;
    a.cov_inv = cov_inv;
    a.den_r = density_r;
    a.den_i = density_i;
    a.half_shape = half_shape;
    a.ranges = reinterpret_cast<const int2*>(tile_ranges);
    a.pair_ids = pair_ids;
    a.gv_r = grad_vol_r;
    a.gv_i = grad_vol_i;
    a.g_center = grad_centers;
    a.g_cov = grad_cov_inv;
    a.g_dr = grad_den_r;
    a.g_di = grad_den_i;
    if (tile_size == 8) k_backward8<true, false, 2><<<unsigned(num_tiles * a.split), kThreads, 0, st>>>(a);
    else if (tile_size == 4)
        k_backward4<true, false><<<unsigned((num_tiles + kWarps - 1) / kWarps), kThreads, 0, st>>>(a);
    else k_backward_generic<true, false><<<unsigned(num_tiles), kThreads, 0, st>>>(a);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

size_t gsv_batch_workspace_bytes(int count) {
    if (count <= 0 || count > (1 << 16)) return 0;
    return align_up(size_t(count) * sizeof(RenderArgs)) + 3 * align_up(size_t(count + 1) * sizeof(int64_t)) +
           align_up(2 * sizeof(unsigned long long));
}

int gsv_batch_setup(const gsv_batch_item* items, int count, int flags, void* ws_batch, size_t ws_bytes,
                    void* stream) {
    if (!items || count <= 0 || !ws_batch || ws_bytes < gsv_batch_workspace_bytes(count))
        return GSV_ERR_INVALID_ARGUMENT;
    const bool det = flags & GSV_BACKWARD_DETERMINISTIC;
    RenderArgs* host = new RenderArgs[count];
    int64_t* pre = new int64_t[3 * (count + 1)];
    int64_t *tp = pre, *gp = pre + count + 1, *cp = pre + 2 * (count + 1);
    tp[0] = gp[0] = cp[0] = 0;
    int rc = GSV_OK;
    for (int i = 0; i < count && rc == GSV_OK; ++i) {
        const gsv_batch_item& it = items[i];
        GaussLayout G;
        PairLayout P;
        int64_t ntiles = 0;
        if (it.shape.tile_size != 8 || layout_for(it.shape, it.params.n, it.capacity, flags, &G, &P, &ntiles) != GSV_OK ||
            !it.ws_gauss || (it.capacity > 0 && !it.ws_pairs)) {
            rc = GSV_ERR_INVALID_ARGUMENT;
            break;
        }
        RenderArgs a{};
        fill_shape(a, it.shape);
        a.recs = cat<Rec>(it.ws_gauss, G.rec);
        a.ext = cat<float4>(it.ws_gauss, G.ext);
        a.ranges = cat<int2>(it.ws_gauss, G.ranges);
        a.pair_ids = it.capacity > 0 ? cat<int32_t>(it.ws_pairs, P.vals_out) : nullptr;
        a.vol = it.volume;
        a.gvol = it.grad_volume;
        a.accum = mat<float>(const_cast<void*>(it.ws_gauss), G.accum);
        a.partials = det && it.capacity > 0 ? mat<float>(const_cast<void*>(it.ws_pairs), P.partials) : nullptr;
        a.kept = det && it.capacity > 0 ? mat<uint8_t>(const_cast<void*>(it.ws_pairs), P.keys_in) : nullptr;
        a.prm = it.params;
        a.grd = it.grads;
        a.boxes = cat<int4>(it.ws_gauss, G.box);
        a.offsets = cat<int64_t>(it.ws_gauss, G.offsets);
        a.capacity = it.capacity;
        a.chunk = (it.chunk >= 1 && it.chunk <= 32) ? it.chunk : 32;
        a.split = 1;  // one work item per tile
        host[i] = a;
        tp[i + 1] = tp[i] + ntiles;
        gp[i + 1] = gp[i] + it.params.n;
        cp[i + 1] = cp[i] + (det ? (it.capacity + 15) / 16 : 0);
    }
    if (rc == GSV_OK) {
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        char* base = static_cast<char*>(ws_batch);
        const size_t o_items = 0, o_pre = align_up(size_t(count) * sizeof(RenderArgs));
        cudaError_t e = cudaMemcpyAsync(base + o_items, host, size_t(count) * sizeof(RenderArgs),
                                        cudaMemcpyHostToDevice, st);
        for (int k = 0; k < 3 && e == cudaSuccess; ++k)
            e = cudaMemcpyAsync(base + o_pre + k * align_up(size_t(count + 1) * sizeof(int64_t)),
                                pre + k * (count + 1), size_t(count + 1) * sizeof(int64_t), cudaMemcpyHostToDevice,
                                st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            gsv_detail_set_error(e, "gsv_batch_setup upload", __FILE__, __LINE__);
            rc = GSV_ERR_CUDA;
        }
    }
    delete[] host;
    delete[] pre;
    return rc;
}

namespace {
BatchTable batch_table(void* ws_batch, int count, int det) {
    BatchTable t{};
    char* base = static_cast<char*>(ws_batch);
    const size_t o_pre = align_up(size_t(count) * sizeof(RenderArgs));
    const size_t step = align_up(size_t(count + 1) * sizeof(int64_t));
    t.items = reinterpret_cast<RenderArgs*>(base);
    t.tile_prefix = reinterpret_cast<int64_t*>(base + o_pre);
    t.gauss_prefix = reinterpret_cast<int64_t*>(base + o_pre + step);
    t.cap_prefix = reinterpret_cast<int64_t*>(base + o_pre + 2 * step);
    t.counters = reinterpret_cast<unsigned long long*>(base + o_pre + 3 * step);
    t.count = count;
    t.det = det;
    return t;
}

// Persistent grid: every SM filled to the kernel's occupancy.
int persistent_grid(const void* kernel, int threads) {
    int dev = 0, sms = 148, per_sm = 4;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) != cudaSuccess || per_sm < 1)
        per_sm = 4;
    return sms * per_sm;
}
}  // namespace

int gsv_forward_batched(void* ws_batch, int count, void* stream) {
    if (!ws_batch || count <= 0) return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    BatchTable t = batch_table(ws_batch, count, 0);
    GSV_CUDA_TRY(cudaMemsetAsync(t.counters, 0, 2 * sizeof(unsigned long long), st));
    k_forward8_batched<<<persistent_grid(reinterpret_cast<const void*>(k_forward8_batched), 256), 256, 0, st>>>(t);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

int gsv_backward_batched(void* ws_batch, int count, int flags, void* stream) {
    if (!ws_batch || count <= 0) return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool det = flags & GSV_BACKWARD_DETERMINISTIC;
    BatchTable t = batch_table(ws_batch, count, det);
    GSV_CUDA_TRY(cudaMemsetAsync(t.counters, 0, 2 * sizeof(unsigned long long), st));
    // every volume's accumulators are zero: its preprocess cleared them and
    // k_finalize(_batched) clears them again after reading
    const int grid = persistent_grid(reinterpret_cast<const void*>(k_finalize_batched), 256);
    if (det) {
        k_clear_kept_batched<<<grid, 256, 0, st>>>(t);
        GSV_LAUNCH_CHECK();
        k_backward8_batched<true><<<persistent_grid(reinterpret_cast<const void*>(k_backward8_batched<true>), kThreads), kThreads, 0, st>>>(t);
        GSV_LAUNCH_CHECK();
        k_finalize_det_batched<<<grid, 256, 0, st>>>(t);
    } else {
        k_backward8_batched<false><<<persistent_grid(reinterpret_cast<const void*>(k_backward8_batched<false>), kThreads), kThreads, 0, st>>>(t);
        GSV_LAUNCH_CHECK();
        k_finalize_batched<<<grid, 256, 0, st>>>(t);
    }
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

}  // extern "C"
