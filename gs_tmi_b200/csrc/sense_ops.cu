// sense_ops.cu -- fused elementwise kernels of the SENSE data-consistency
// term around the 3-D FFTs (which stay torch.fft / cuFFT).
//
// The plain 3DGSMR loss (3DGS/3dgsVC/trainers/trainer.py:256-268) is
//   L = sum_c || M * fft3c(S_c x) - y_c ||^2,
//   fft3c = fftshift o fftn(ortho) o ifftshift over the last three axes.
// Evaluated op by op it streams the [C, V] coil images through memory about
// ten times per iteration (coil product, two shifts, mask, residual, square,
// sum, and as many again in the backward).  Here the shifts are folded into
// the index arithmetic of three kernels:
//   expand  : X[c, k]  = S[c, i] x[i],            i = k + n/2 (mod n) per axis
//   residual: R[c, j]  = M[k] Kp[c, j] - y[c, k],  k = j + n/2 (mod n),
//             L = sum |R|^2 (fixed-order two-stage sum), Kp <- 2 M R in place
//             (the gradient of L with respect to Kp = fftn(X))
//   adjoint : g[i]     = sum_c conj(S[c, i]) G[c, k], k = i - n/2 (mod n),
//             G = ifftn(2 M R) (the adjoint of an orthonormal fftn)
// so that the data term costs expand + fftn + residual + ifftn + adjoint.
// g is the gradient of L with respect to x in torch's convention for
// complex tensors (conj-Wirtinger times 2: d|z|^2 -> 2 z).
#include <cuComplex.h>

#include <type_traits>

#include "gsv_common.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kResidualBlocks = 1184;  // fixed: the loss sum order does not depend on the device

struct Geo {
    int32_t d, h, w;
    int64_t v;  // d*h*w
};

// a + s (|s| < n) wrapped into [0, n): one step of fftshift / ifftshift
__device__ __forceinline__ int wrap(int a, int s, int n) {
    const int t = a + s;
    return t >= n ? t - n : (t < 0 ? t + n : t);
}

// N complex values (N = 2: one 16-byte access) and N reals.
template <int N>
struct Cx {
    float2 v[N];
};
template <int N, bool RO = true>  // RO: nothing writes the array meanwhile
__device__ __forceinline__ Cx<N> load_cx(const float2* p) {
    Cx<N> r;
    if (N == 2) {
        const float4 x = RO ? __ldg(reinterpret_cast<const float4*>(p)) : *reinterpret_cast<const float4*>(p);
        r.v[0] = make_float2(x.x, x.y);
        r.v[N - 1] = make_float2(x.z, x.w);
    } else {
        r.v[0] = RO ? __ldg(p) : *p;
    }
    return r;
}
template <int N>
__device__ __forceinline__ void store_cx(float2* p, const Cx<N>& r) {
    if (N == 2) *reinterpret_cast<float4*>(p) = make_float4(r.v[0].x, r.v[0].y, r.v[N - 1].x, r.v[N - 1].y);
    else *p = r.v[0];
}

// The kernels give a thread N neighbouring voxels of a row and walk the coils there, so that the volume,
// the mask and the index arithmetic are taken once for all coils.  Bound by memory; kUnroll coils' loads are
// in flight together.  N = 2 needs rows of a multiple of four (their half shift is even) and 16-byte
// aligned arrays.  128x128x96 with 8 coils, us, against a row of one coil per warp: expand 47 -> 32,
// residual 78 -> 44, adjoint 40 -> 35 (214, 308 and 214 MB read and written: 6.7, 7.0 and 6.1 TB/s).
constexpr int kUnroll = 4;

// Voxel group x (of v / N, I: an index type that holds it): its element offset and that of the place
// shifted by sign * n/2 on every axis.
template <int N, typename I>
__device__ __forceinline__ void place_of(const Geo& g, I x, int sign, int64_t& own, int64_t& shifted) {
    const I groups = I(g.w / N);
    const I row = x / groups;
    const int c = int(x - row * groups) * N;
    const int a = int(row / I(g.h)), b = int(row - I(a) * I(g.h));
    own = (int64_t(a) * g.h + b) * g.w + c;
    shifted = (int64_t(wrap(a, sign * (g.d / 2), g.d)) * g.h + wrap(b, sign * (g.h / 2), g.h)) * g.w +
              wrap(c, sign * (g.w / 2), g.w);
}

template <int N, typename I>
__global__ void __launch_bounds__(kThreads) k_expand(const float2* __restrict__ x, const float2* __restrict__ s,
                                                     int32_t nc, Geo g, float scale, float2* __restrict__ out) {
    const I i = I(blockIdx.x) * kThreads + threadIdx.x;
    if (i >= I(g.v / N)) return;
    int64_t own, src;
    place_of<N, I>(g, i, +1, own, src);  // X[c, k] = (S x)[c, k + n/2]
    Cx<N> b = load_cx<N>(x + src);
#pragma unroll
    for (int k = 0; k < N; ++k) b.v[k] = make_float2(b.v[k].x * scale, b.v[k].y * scale);
    for (int c0 = 0; c0 < nc; c0 += kUnroll) {
        Cx<N> a[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
            if (c0 + u < nc) a[u] = load_cx<N>(s + int64_t(c0 + u) * g.v + src);
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
            if (c0 + u < nc) {
                Cx<N> r;
#pragma unroll
                for (int k = 0; k < N; ++k)
                    r.v[k] = make_float2(a[u].v[k].x * b.v[k].x - a[u].v[k].y * b.v[k].y,
                                         a[u].v[k].x * b.v[k].y + a[u].v[k].y * b.v[k].x);
                store_cx<N>(out + int64_t(c0 + u) * g.v + own, r);
            }
    }
}

// Block sum in a fixed order, to partial[blockIdx.x].
__device__ __forceinline__ void block_partial(float acc, float* __restrict__ partial) {
    __shared__ float red[kThreads / 32];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = 0.f;
        for (int i = 0; i < kThreads / 32; ++i) b += red[i];
        partial[blockIdx.x] = b;
    }
}

template <int N, typename I>
__global__ void __launch_bounds__(kThreads) k_residual(float2* __restrict__ kp, const float* __restrict__ mask,
                                                       const float2* __restrict__ y, int32_t nc, Geo g,
                                                       float* __restrict__ partial) {
    float acc = 0.f;
    for (I i = I(blockIdx.x) * kThreads + threadIdx.x; i < I(g.v / N); i += I(gridDim.x) * kThreads) {
        int64_t own, nat;
        place_of<N, I>(g, i, +1, own, nat);  // Kp[c, j] is fft3c's entry [c, j + n/2]
        float m[N];
#pragma unroll
        for (int k = 0; k < N; ++k) m[k] = __ldg(mask + nat + k);
        for (int c0 = 0; c0 < nc; c0 += kUnroll) {
            Cx<N> z[kUnroll], t[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
                if (c0 + u < nc) {
                    z[u] = load_cx<N, false>(kp + int64_t(c0 + u) * g.v + own);
                    t[u] = load_cx<N>(y + int64_t(c0 + u) * g.v + nat);
                }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
                if (c0 + u < nc) {
                    Cx<N> r;
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        const float rr = fmaf(m[k], z[u].v[k].x, -t[u].v[k].x), ri = fmaf(m[k], z[u].v[k].y, -t[u].v[k].y);
                        acc = fmaf(rr, rr, fmaf(ri, ri, acc));
                        r.v[k] = make_float2(2.f * m[k] * rr, 2.f * m[k] * ri);
                    }
                    store_cx<N>(kp + int64_t(c0 + u) * g.v + own, r);
                }
        }
    }
    block_partial(acc, partial);
}

__global__ void k_sum_partials(const float* __restrict__ partial, int n, float* __restrict__ loss) {
    __shared__ double red[256];
    double a = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) a += partial[i];
    red[threadIdx.x] = a;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = float(red[0]);
}

template <int N, typename I>
__global__ void __launch_bounds__(kThreads) k_adjoint(const float2* __restrict__ gk, const float2* __restrict__ s,
                                                      int32_t nc, Geo g, float scale, float2* __restrict__ out) {
    const I x = I(blockIdx.x) * kThreads + threadIdx.x;
    if (x >= I(g.v / N)) return;
    int64_t i, k;
    place_of<N, I>(g, x, -1, i, k);  // (S x).grad[i] = X.grad[i - n/2]
    Cx<N> a;
#pragma unroll
    for (int e = 0; e < N; ++e) a.v[e] = make_float2(0.f, 0.f);
    for (int c0 = 0; c0 < nc; c0 += kUnroll) {
        Cx<N> sc[kUnroll], z[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
            if (c0 + u < nc) {
                sc[u] = load_cx<N>(s + int64_t(c0 + u) * g.v + i);
                z[u] = load_cx<N>(gk + int64_t(c0 + u) * g.v + k);
            }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
            if (c0 + u < nc)
#pragma unroll
                for (int e = 0; e < N; ++e) {
                    a.v[e].x = fmaf(sc[u].v[e].x, z[u].v[e].x, fmaf(sc[u].v[e].y, z[u].v[e].y, a.v[e].x));  // conj(s) * z
                    a.v[e].y = fmaf(sc[u].v[e].x, z[u].v[e].y, fmaf(-sc[u].v[e].y, z[u].v[e].x, a.v[e].y));
                }
    }
#pragma unroll
    for (int e = 0; e < N; ++e) a.v[e] = make_float2(a.v[e].x * scale, a.v[e].y * scale);
    store_cx<N>(out + i, a);
}

__device__ __forceinline__ float cabs(float2 z) { return sqrtf(fmaf(z.x, z.x, z.y * z.y)); }
__device__ __forceinline__ float sgn(float x) { return x > 0.f ? 1.f : (x < 0.f ? -1.f : 0.f); }

// TV(|x|) = sum over the three axes of |m[i + e_a] - m[i]|, m = |x|
// (3DGS/3dgsVC/losses/losses.py:18-26, MagnitudeTVLoss), and its gradient in
// torch's convention: dTV/dm_i (a sum of signs) times x_i / |x_i| (0 at 0).
__global__ void __launch_bounds__(kThreads) k_tv(const float2* __restrict__ x, Geo g, float* __restrict__ partial,
                                                 float2* __restrict__ grad) {
    const int rows = g.d * g.h;
    const int64_t sd = int64_t(g.h) * g.w, sh = g.w;
    float acc = 0.f;
    // a warp takes a row (a patch of magnitudes in shared memory, one square root a voxel instead of seven,
    // measured the same: the quotients and signs bound it)
    const int lane = threadIdx.x & 31;
    for (int r = (blockIdx.x * kThreads + threadIdx.x) >> 5; r < rows; r += gridDim.x * (kThreads / 32)) {
        const int a = r / g.h, b = r - a * g.h;
        for (int c = lane; c < g.w; c += 32) {
            const int64_t i = int64_t(r) * g.w + c;
            const float2 z = __ldg(x + i);
            const float m = cabs(z);
            float dm = 0.f;
            if (a + 1 < g.d) { const float t = cabs(__ldg(x + i + sd)) - m; acc += fabsf(t); dm -= sgn(t); }
            if (b + 1 < g.h) { const float t = cabs(__ldg(x + i + sh)) - m; acc += fabsf(t); dm -= sgn(t); }
            if (c + 1 < g.w) { const float t = cabs(__ldg(x + i + 1)) - m; acc += fabsf(t); dm -= sgn(t); }
            if (a > 0) dm += sgn(m - cabs(__ldg(x + i - sd)));
            if (b > 0) dm += sgn(m - cabs(__ldg(x + i - sh)));
            if (c > 0) dm += sgn(m - cabs(__ldg(x + i - 1)));
            grad[i] = m > 0.f ? make_float2(dm * z.x / m, dm * z.y / m) : make_float2(0.f, 0.f);
        }
    }
    block_partial(acc, partial);
}

bool geo_ok(int32_t nc, int32_t d, int32_t h, int32_t w) {
    return nc > 0 && d > 0 && h > 0 && w > 0 && int64_t(nc) * d * h < (int64_t(1) << 31);
}

bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }
unsigned blocks_for(int64_t items) { return unsigned((items + kThreads - 1) / kThreads); }

// Calls f(N, I) for the voxels per thread and the index type that a call needs.
template <typename F>
void by_form(const Geo& g, bool pairs, F&& f) {
    using Two = std::integral_constant<int, 2>;
    using One = std::integral_constant<int, 1>;
    if (g.v < (int64_t(1) << 31)) {
        if (pairs) f(Two{}, uint32_t{});
        else f(One{}, uint32_t{});
    } else {
        if (pairs) f(Two{}, int64_t{});
        else f(One{}, int64_t{});
    }
}

}  // namespace

extern "C" {

size_t gsv_sense_workspace_bytes(void) { return size_t(kResidualBlocks) * sizeof(float); }

int gsv_sense_expand_scaled(const float* volume, const float* coils, int32_t ncoils, int32_t d, int32_t h, int32_t w,
                            float scale, float* out, void* stream) {
    if (!volume || !coils || !out || !geo_ok(ncoils, d, h, w)) return GSV_ERR_INVALID_ARGUMENT;
    const Geo g{d, h, w, int64_t(d) * h * w};
    const bool pairs = w % 4 == 0 && aligned(volume, 16) && aligned(coils, 16) && aligned(out, 16);
    by_form(g, pairs, [&](auto n, auto i) {
        k_expand<decltype(n)::value, decltype(i)>
            <<<blocks_for(g.v / decltype(n)::value), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
                reinterpret_cast<const float2*>(volume), reinterpret_cast<const float2*>(coils), ncoils, g, scale,
                reinterpret_cast<float2*>(out));
    });
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

int gsv_sense_expand(const float* volume, const float* coils, int32_t ncoils, int32_t d, int32_t h, int32_t w,
                     float* out, void* stream) {
    return gsv_sense_expand_scaled(volume, coils, ncoils, d, h, w, 1.0f, out, stream);
}

int gsv_sense_residual(float* kspace, const float* mask, const float* measured, int32_t ncoils, int32_t d,
                       int32_t h, int32_t w, float* loss, void* ws, size_t ws_bytes, void* stream) {
    if (!kspace || !mask || !measured || !loss || !ws || ws_bytes < gsv_sense_workspace_bytes() ||
        !geo_ok(ncoils, d, h, w))
        return GSV_ERR_INVALID_ARGUMENT;
    const Geo g{d, h, w, int64_t(d) * h * w};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float* partial = static_cast<float*>(ws);
    const bool pairs = w % 4 == 0 && aligned(kspace, 16) && aligned(measured, 16);
    by_form(g, pairs, [&](auto n, auto i) {
        k_residual<decltype(n)::value, decltype(i)><<<kResidualBlocks, kThreads, 0, st>>>(
            reinterpret_cast<float2*>(kspace), mask, reinterpret_cast<const float2*>(measured), ncoils, g, partial);
    });
    GSV_LAUNCH_CHECK();
    k_sum_partials<<<1, 256, 0, st>>>(partial, kResidualBlocks, loss);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

int gsv_sense_adjoint_scaled(const float* kgrad_image, const float* coils, int32_t ncoils, int32_t d, int32_t h,
                             int32_t w, float scale, float* volume_grad, void* stream) {
    if (!kgrad_image || !coils || !volume_grad || !geo_ok(ncoils, d, h, w)) return GSV_ERR_INVALID_ARGUMENT;
    const Geo g{d, h, w, int64_t(d) * h * w};
    const bool pairs = w % 4 == 0 && aligned(kgrad_image, 16) && aligned(coils, 16) && aligned(volume_grad, 16);
    by_form(g, pairs, [&](auto n, auto i) {
        k_adjoint<decltype(n)::value, decltype(i)>
            <<<blocks_for(g.v / decltype(n)::value), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
                reinterpret_cast<const float2*>(kgrad_image), reinterpret_cast<const float2*>(coils), ncoils, g, scale,
                reinterpret_cast<float2*>(volume_grad));
    });
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

int gsv_sense_adjoint(const float* kgrad_image, const float* coils, int32_t ncoils, int32_t d, int32_t h,
                      int32_t w, float* volume_grad, void* stream) {
    return gsv_sense_adjoint_scaled(kgrad_image, coils, ncoils, d, h, w, 1.0f, volume_grad, stream);
}

int gsv_tv_magnitude(const float* volume, int32_t d, int32_t h, int32_t w, float* loss, float* grad, void* ws,
                     size_t ws_bytes, void* stream) {
    if (!volume || !loss || !grad || !ws || ws_bytes < gsv_sense_workspace_bytes() || !geo_ok(1, d, h, w))
        return GSV_ERR_INVALID_ARGUMENT;
    const Geo g{d, h, w, int64_t(d) * h * w};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float* partial = static_cast<float*>(ws);
    k_tv<<<kResidualBlocks, kThreads, 0, st>>>(reinterpret_cast<const float2*>(volume), g, partial,
                                                             reinterpret_cast<float2*>(grad));
    GSV_LAUNCH_CHECK();
    k_sum_partials<<<1, 256, 0, st>>>(partial, kResidualBlocks, loss);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

}  // extern "C"
