// mlp_tcgen05.cu -- BF16 tensor-core GEMM with fused epilogues for the
// warm-start MLP (sm_100a, tcgen05 + TMEM).
//
//   C[m, n] = sum_k A[m, k] * B[n, k]      (BF16 operands, FP32 accumulate)
//
// A and B are read from global memory through arbitrary (row, k) strides, so
// the same kernel serves the forward (X W^T), the input-gradient (dY W) and
// the weight-gradient (dZ^T X, split-K) products of training.  One CTA per SM
// walks 128 x N output tiles (N = 256 or 16) with its warps in three parts:
// one thread keeps a ring of 64-wide K chunks full by TMA, one issues
// tcgen05.mma (M=128, N, K=16, kind::f16, BF16 x BF16 -> F32) into one of two
// TMEM accumulators, and sixteen warps empty the other through the epilogue.
// Operands whose K axis is contiguous come as K-major tiles, operands whose
// row axis is contiguous (the transposed operands of the weight gradients) as
// MN-major ones, both in the 128-byte swizzle; strides that TMA does not take
// are copied by cp.async, others element by element, into the same layouts.
// The epilogue reads TMEM with tcgen05.ld (a warp reads the lanes of quarter
// w % 4), turns 32-column chunks through shared memory so that accesses are
// whole lines, and for GELU' also accumulates the column sums of its output
// (the layer's bias gradient).
// What bounds it: with K = 256 the epilogue's traffic (z and the activation,
// six bytes an output).  84,375 x 256 x 256: bias + GELU 37 us (4.7 TB/s; 88 us
// with one tile per CTA and cp.async), GELU' 42 us (116 us), weight gradient
// 20 us (56 us); at 189,440 rows another 94,720 cost GELU' 35 us, 5.5 TB/s.
// Every mbarrier wait is bounded; on time-out the kernel latches an error
// flag, skips the epilogue, waits (bounded) until the tensor-core work and the
// copies it issued have retired, frees its TMEM and returns.
// gsv_mlp_gemm_test_timeout drives that path: the issuing thread leaves one K
// stage's MMAs and commits out, so the waits on them run out.
// No cluster launch, no multicast.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <climits>

#include "gsv_common.cuh"

namespace {

constexpr int kBM = 128;
constexpr int kBK = 64;
// How the operands come and the outputs go: by TMA and in wide accesses; by TMA
// and element by element; by cp.async or element by element and either.  (One
// kernel for the first two kept GELU''s z in local memory: 45 us for 42.)
enum Mode : int { TMA_WIDE = 0, TMA_NARROW = 1, COPIES = 2 };
// Warps of a CTA: the epilogue's, in column groups of four (a warp reads the TMEM
// lanes of its quarter), the one that issues the MMAs, and the loading ones.
// TMA: one thread issues all copies; GELU' took 51 us with 8 epilogue warps and
// 43 with 16.  Otherwise eight warps copy the operands, a pair to each of the
// four stages.
template <int MODE>
struct Warps {
    static constexpr int kEpi = MODE != COPIES ? 16 : 8;
    static constexpr int kLoad = MODE != COPIES ? 1 : 8;
    static constexpr int kThreads = (kEpi + 1 + kLoad) * 32;
};
constexpr uint32_t kAtom = 1024;      // swizzled 128-byte x 8 block: 8 rows x 64 k, or 64 rows x 8 k
constexpr uint32_t kMnBox = 64 * kBK * 2;  // MN-major: 64 rows x the chunk's 64 k
constexpr int kScratch = 32 * 32 * 4;  // an epilogue warp's 32 x 32 chunk
constexpr long long kWaitLimit = 1ll << 26;

enum Epi : int {
    EPI_F32 = 0,        // out_f32 = acc (+ bias)
    EPI_BIAS_GELU = 1,  // z_f32 = acc + bias; out_bf16 = gelu(z)
    EPI_GELU_GRAD = 2,  // out_bf16 = acc * gelu'(z_f32)
    EPI_ATOMIC_F32 = 3  // atomicAdd(out_f32, acc)   (split-K)
};

struct GemmArgs {
    const __nv_bfloat16* a;
    const __nv_bfloat16* b;
    long long a_sm, a_sk;  // A element (m, k) at a[m*a_sm + k*a_sk]
    long long b_sn, b_sk;  // B element (n, k) at b[n*b_sn + k*b_sk]
    int M, N, K;
    int k_per_split;       // K range per blockIdx.z
    const float* bias;     // [N] or null
    float* out_f32;
    __nv_bfloat16* out_bf16;
    float* z_f32;          // EPI_BIAS_GELU writes it, EPI_GELU_GRAD reads it
    long long c_sm, c_sn;  // C element (m, n) at c[m*c_sm + n*c_sn]
    int epi;
    int a_mode, b_mode;    // Stage: how each operand is copied to shared memory
    int wide;              // rows of C take 32-byte (FP32) and 16-byte (BF16) accesses
    int tiles_m, tiles_n, tiles;
    float* col_sum;        // EPI_GELU_GRAD: += column sums of the BF16 output (or null)
    int* error;
    long long wait_limit;  // polls per mbarrier wait (kWaitLimit unless testing the time-out)
    int skip_stage;        // test hook: K stage whose MMAs and commits are left out (-1: none)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// tcgen05 shared-memory matrix descriptor: 128-byte swizzle, version 1.
// K-major: 8-row blocks 1024 B apart (the leading offset is not used within
// one swizzled row).  MN-major: 8-k blocks 1024 B apart, 64-row blocks kMnBox
// apart.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, bool mn) {
    uint64_t d = 0;
    d |= uint64_t((saddr >> 4) & 0x3FFF);
    d |= uint64_t(mn ? kMnBox >> 4 : 1) << 16;
    d |= uint64_t(kAtom >> 4) << 32;
    d |= uint64_t(1) << 46;  // descriptor version for tcgen05
    d |= uint64_t(2) << 61;  // 128-byte swizzle
    return d;
}
// Bytes from one K = 16 step to the next.
__device__ __forceinline__ uint32_t k16_step(bool mn) { return mn ? 2 * kAtom : 32; }

// Instruction descriptor, kind::f16: D=F32, A=B=BF16, both K-major, M=128.
__host__ __device__ constexpr uint32_t make_idesc(int n) {
    return (1u << 4)                       // D format F32
           | (1u << 7)                     // A format BF16
           | (1u << 10)                    // B format BF16
           | (uint32_t(n >> 3) << 17)      // N / 8
           | (uint32_t(kBM >> 4) << 24);   // M / 16
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long limit) {
    for (long long i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// tcgen05.ld and its wait need the whole warp converged, wherever its lanes come from.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    __syncwarp();
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// GELU in its tanh form (Hendrycks & Gimpel, "Gaussian Error Linear Units",
// 2016): 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3))), with the SFU's
// tanh.approx; its outputs are rounded to BF16, far coarser than the
// approximation.
__device__ __forceinline__ float tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
constexpr float kGeluC0 = 0.7978845608028654f;       // sqrt(2/pi)
constexpr float kGeluC1 = 0.7978845608028654f * 0.044715f;
// Two at a time: with one value at a time the GELU' epilogue issued 35
// instructions per output and warp and took 43 us where this takes 40.
__device__ __forceinline__ float2 splat(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 tanh_inner(float2 x, float2 x2) {  // tanh of sqrt(2/pi) (x + 0.044715 x^3)
    const float2 u = __fmul2_rn(x, __ffma2_rn(splat(kGeluC1), x2, splat(kGeluC0)));
    return make_float2(tanh_approx(u.x), tanh_approx(u.y));
}
__device__ __forceinline__ float2 gelu(float2 x) {
    const float2 t = tanh_inner(x, __fmul2_rn(x, x));
    return __fmul2_rn(__fmul2_rn(splat(0.5f), x), __fadd2_rn(splat(1.0f), t));
}
// 0.5 (1 + t) + 0.5 x (1 - t^2) du, with du the derivative of tanh's argument
__device__ __forceinline__ float2 gelu_grad(float2 x) {
    const float2 x2 = __fmul2_rn(x, x), t = tanh_inner(x, x2);
    const float2 du = __ffma2_rn(splat(3.0f * kGeluC1), x2, splat(kGeluC0));
    const float2 c = __fmul2_rn(__fmul2_rn(splat(-0.5f), x), __ffma2_rn(t, t, splat(-1.0f)));
    return __ffma2_rn(splat(0.5f), __fadd2_rn(splat(1.0f), t), __fmul2_rn(c, du));
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    __syncwarp();
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 16-byte global -> shared copy that bypasses registers (cp.async, L2 only);
// bytes < 16 zero-fills the rest, bytes == 0 reads nothing.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Byte offset of element (r, k) of a staged operand tile in the canonical
// 128-byte-swizzle layouts, which are also what TMA writes: 16-byte piece p of
// 128-byte line l of an atom lies at piece p ^ (l % 8).
//   K-major : line r, piece k / 8
//   MN-major: line k of the 64-row block r / 64, piece r % 64 / 8
__device__ __forceinline__ uint32_t tile_off(int r, int k, bool mn) {
    return mn ? (r >> 6) * kMnBox + k * 128 + ((((r >> 3) ^ k) & 7) << 4) + (r & 7) * 2
              : r * 128 + (((k >> 3) ^ (r & 7)) << 4) + (k & 7) * 2;
}

// TMA: the box at (x, y) of a tensor map to shared memory, counted on `bar`.
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Operand access mode, fixed per GEMM call on the host.
enum Stage : int {
    ST_K_VEC = 0,   // K contiguous (s_k == 1), 16-byte aligned rows: cp.async along K
    ST_MN_VEC = 1,  // rows contiguous (s_r == 1), 16-byte aligned K steps: cp.async along rows
    ST_SCALAR = 2   // anything else: element-wise loads, K-major layout
};

// A loading pair's copies (thread `tid` of 64) of rows [r0, r0 + ROWS) x k [k0, k0 + kn) of one operand
// into the stage at `dst` (kn: the chunk's k range rounded up to the MMA's
// 16), for strides that TMA does not take; out-of-range elements become zero.
// The scalar mode stores synchronously.
template <int ROWS>
__device__ __forceinline__ void stage_operand(unsigned char* dst, const __nv_bfloat16* src, long long s_r,
                                              long long s_k, int mode, int r0, int nrows, int k0, int kend, int kn,
                                              int tid) {
    const uint32_t base = smem_u32(dst);
    if (mode == ST_K_VEC) {
        const int r = tid & 7, k = (tid >> 3) * 8;
        if (k < kn) {
            const uint32_t at = base + tile_off(r, k, false);
            const __nv_bfloat16* p = src + (long long)(r0 + r) * s_r + k0 + k;
#pragma unroll 4
            for (int i = 0; i < ROWS / 8; ++i, p += 8 * s_r) {
                const bool ok = r0 + r + i * 8 < nrows && k0 + k < kend;
                cp_async16(at + i * kAtom, ok ? p : src, ok ? min(16, (kend - k0 - k) * 2) : 0);
            }
        }
    } else if (mode == ST_MN_VEC) {
        const int k = tid & 7;
        for (int r = (tid >> 3) * 8; r < ROWS; r += 64) {
            const uint32_t at = base + tile_off(r, k, true);
            const __nv_bfloat16* p = src + r0 + r + (long long)(k0 + k) * s_k;
#pragma unroll 4
            for (int i = 0; i < kn / 8; ++i, p += 8 * s_k) {
                const bool ok = r0 + r < nrows && k0 + k + i * 8 < kend;
                cp_async16(at + i * kAtom, ok ? p : src, ok ? min(16, (nrows - r0 - r) * 2) : 0);
            }
        }
    } else {
        // threads along the axis with the smaller stride, sixteen loads in flight
        const __nv_bfloat16 zero = __float2bfloat16(0.0f);
        __nv_bfloat16 v[16];
        if (s_k < s_r) {
            const int k = tid;
            const bool k_ok = k0 + k < kend;
            const __nv_bfloat16* p = src + r0 * s_r + (k0 + k) * s_k;
            for (int r = 0; r < ROWS; r += 16, p += 16 * s_r) {
#pragma unroll
                for (int u = 0; u < 16; ++u) v[u] = k_ok && r0 + r + u < nrows ? p[u * s_r] : zero;
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    *reinterpret_cast<__nv_bfloat16*>(dst + r * 128 + tile_off(u, k, false)) = v[u];
            }
        } else {
            constexpr int kAlong = ROWS < 64 ? ROWS : 64, kAcross = 64 / kAlong;
            for (int r = tid % kAlong; r < ROWS; r += kAlong) {
                const int k_end = r0 + r < nrows ? kend - k0 : 0;
                const __nv_bfloat16* p = src + (r0 + r) * s_r + (k0 + tid / kAlong * 16) * s_k;
                for (int k = tid / kAlong * 16; k < kn; k += kAcross * 16) {
#pragma unroll
                    for (int u = 0; u < 16; ++u, p += s_k) v[u] = k + u < k_end ? *p : zero;
                    p += (kAcross - 1) * 16 * s_k;
#pragma unroll
                    for (int h = 0; h < 16; h += 8) {
                        uint32_t w[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            w[u] = uint32_t(__bfloat16_as_ushort(v[h + 2 * u])) |
                                   uint32_t(__bfloat16_as_ushort(v[h + 2 * u + 1])) << 16;
                        *reinterpret_cast<uint4*>(dst + tile_off(r, k + h, false)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        }
    }
}

// One output from its sum x; z is read by the caller.
template <int EPI>
__device__ __forceinline__ void epi_store(const GemmArgs& g, int64_t ci, float x, float bias_n, float z) {
    if constexpr (EPI == EPI_F32) {
        g.out_f32[ci] = x + bias_n;
    } else if constexpr (EPI == EPI_BIAS_GELU) {
        x += bias_n;
        g.z_f32[ci] = x;
        g.out_bf16[ci] = __float2bfloat16(gelu(splat(x)).x);
    } else if constexpr (EPI == EPI_GELU_GRAD) {
        g.out_bf16[ci] = __float2bfloat16(x * gelu_grad(splat(z)).x);
    } else {
        atomicAdd(g.out_f32 + ci, x);
    }
}

__device__ __forceinline__ float bias_of(const GemmArgs& g, int n) {
    return (n < g.N && g.bias && (g.epi == EPI_F32 || g.epi == EPI_BIAS_GELU)) ? g.bias[n] : 0.f;
}

// 32-byte accesses: a whole sector per lane.
__device__ __forceinline__ void ld_v8(const float* p, float2* v) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[2].x), "=f"(v[2].y), "=f"(v[3].x),
                   "=f"(v[3].y)
                 : "l"(p));
}
__device__ __forceinline__ void st_v8(float* p, const float2* v) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0].x), "f"(v[0].y),
                 "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y)
                 : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float2 v) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(v.x, v.y);
    return reinterpret_cast<const uint32_t&>(p);
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void red_v4(float* p, float2 a, float2 b) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y)
                 : "memory");
}

// The epilogue's chunk: 32 rows by CW columns of a warp, turned through 32 x CW
// floats of shared memory from a row per lane (what TMEM gives) to CW / 8
// lanes per row with eight columns each, so that a warp's access is whole
// lines.  A row per lane needs no turning, but its 32-byte accesses touch 32
// lines each: bias + GELU over 84,375 rows took 47 us that way, 20 of them for
// z, and takes 36 this way.
template <int CW>
struct Chunk {
    static constexpr int kLanes = CW / 8;       // lanes per row
    static constexpr int kRows = 32 / kLanes;   // rows per pass
    static constexpr int kPasses = kLanes;
    // byte offset of 16-byte piece p of row r: no two of eight lanes share a bank
    __device__ static __forceinline__ int at(int r, int p) {
        return CW == 32 ? r * 128 + ((p ^ (r & 7)) << 4) : r * 64 + ((p ^ ((r >> 1) & 3)) << 4);
    }
    __device__ static __forceinline__ int row(int pass, int lane) { return pass * kRows + lane / kLanes; }
    __device__ static __forceinline__ int col(int lane) { return lane % kLanes * 8; }
    __device__ static __forceinline__ void put(unsigned char* scr, uint32_t taddr, int lane) {
        float v[CW];
        if constexpr (CW == 32) tmem_ld32(taddr, v);
        else tmem_ld16(taddr, v);  // either begins with a __syncwarp: the previous chunk has been read
#pragma unroll
        for (int p = 0; p < CW / 4; ++p)
            *reinterpret_cast<float4*>(scr + at(lane, p)) = make_float4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
        __syncwarp();
    }
    __device__ static __forceinline__ void get(const unsigned char* scr, int pass, int lane, float2* v) {
        const int r = row(pass, lane), p = lane % kLanes * 2;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 q = *reinterpret_cast<const float4*>(scr + at(r, p + h));
            v[2 * h] = make_float2(q.x, q.y), v[2 * h + 1] = make_float2(q.z, q.w);
        }
    }
    __device__ static __forceinline__ float get1(const unsigned char* scr, int r, int c) {
        return *reinterpret_cast<const float*>(scr + at(r, c >> 2) + (c & 3) * 4);
    }
};

// A chunk of C that does not take wide accesses, element by element: strided
// columns (the rows across the lanes), or rows that are not aligned (the
// columns across the lanes).
template <int EPI, int CW>
__device__ __noinline__ void store_chunk(const GemmArgs& g, uint32_t taddr, unsigned char* scr, int row0, int n0) {
    using C = Chunk<CW>;
    const int lane = threadIdx.x & 31;
    if (g.c_sn != 1) {
#pragma unroll 1
        for (int h = 0; h < CW; h += 16) {
            float v[16], z[16] = {};
            const int64_t at = (row0 + lane) * g.c_sm + (n0 + h) * g.c_sn;
            const bool row_ok = row0 + lane < g.M;
            if (EPI == EPI_GELU_GRAD && row_ok) {
#pragma unroll
                for (int k = 0; k < 16; ++k) z[k] = g.z_f32[at + k * g.c_sn];
            }
            tmem_ld16(taddr + h, v);
            if (row_ok) {
#pragma unroll
                for (int k = 0; k < 16; ++k) epi_store<EPI>(g, at + k * g.c_sn, v[k], bias_of(g, n0 + h + k), z[k]);
            }
        }
        return;
    }
    const int n = n0 + lane % CW;
    constexpr int kStep = 32 / CW, kDeep = 32 / kStep;  // rows between a lane's rows; its rows
    const float b = bias_of(g, n);
    float cs = 0.f, z[kDeep] = {};
    const int left = g.M - row0 - lane / CW;
    const int64_t at = int64_t(row0 + lane / CW) * g.c_sm + n;
    if (EPI == EPI_GELU_GRAD) {
#pragma unroll
        for (int k = 0; k < kDeep; ++k)
            if (k * kStep < left) z[k] = g.z_f32[at + k * kStep * g.c_sm];
    }
    C::put(scr, taddr, lane);
#pragma unroll
    for (int k = 0; k < kDeep; ++k) {
        if (k * kStep >= left) continue;
        const int64_t ci = at + k * kStep * g.c_sm;
        const float x = C::get1(scr, lane / CW + k * kStep, lane % CW);
        if constexpr (EPI == EPI_GELU_GRAD) {
            const __nv_bfloat16 o = __float2bfloat16(x * gelu_grad(splat(z[k])).x);
            g.out_bf16[ci] = o;
            cs += __bfloat162float(o);
        } else {
            epi_store<EPI>(g, ci, x, b, 0.f);
        }
    }
    if (EPI == EPI_GELU_GRAD && g.col_sum) atomicAdd(g.col_sum + n, cs);
}

// The epilogue of one warp: all its tiles' rows of TMEM quarter q and columns
// [cbeg, cend) of each tile.
template <int BN, int EPI, int MODE>
__device__ __forceinline__ bool epilogue(const GemmArgs& g, uint32_t tmem, uint32_t acc_cols, const uint64_t* acc_full,
                                         const uint64_t* acc_empty, unsigned char* scr, int q, int cbeg, int cend) {
    constexpr int CW = (BN < 32) ? BN : 32;   // columns read at a time
    using C = Chunk<CW>;
    const int lane = threadIdx.x & 31;
    const int chunks = (cend - cbeg) / CW;
    // GELU': z of the chunk to come is on its way while this one is worked on
    float2 z[EPI == EPI_GELU_GRAD ? C::kPasses * 4 : 1];
    auto load_z = [&](int pass, int row0, int n) {
        const int row = row0 + C::row(pass, lane);
        if (row < g.M) ld_v8(g.z_f32 + int64_t(row) * g.c_sm + n + C::col(lane), z + pass * 4);
    };
    if constexpr (EPI == EPI_GELU_GRAD) {
#pragma unroll
        for (int i = 0; i < C::kPasses * 4; ++i) z[i] = make_float2(0.f, 0.f);
        const int t = blockIdx.x;
        if (g.wide && chunks > 0 && t < g.tiles) {
#pragma unroll
            for (int pass = 0; pass < C::kPasses; ++pass)
                load_z(pass, t % g.tiles_m * kBM + q * 32, t / g.tiles_m % g.tiles_n * BN + cbeg);
        }
    }
    int i = 0;
    for (int t = blockIdx.x; t < g.tiles; t += gridDim.x, ++i) {
        const int row0 = t % g.tiles_m * kBM + q * 32, n0 = t / g.tiles_m % g.tiles_n * BN;
        const int split = t / (g.tiles_m * g.tiles_n);
        const int acc = i & 1, use = i >> 1;
        if (!__all_sync(~0u, mbar_wait(smem_u32(&acc_full[acc]), uint32_t(use & 1), g.wait_limit))) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + acc * acc_cols + (uint32_t(q * 32) << 16);
        for (int ch = 0; ch < chunks; ++ch) {
            // the splits of one tile begin at different columns, so that their sums
            // do not arrive at one address together
            const int c0 = cbeg + (EPI == EPI_ATOMIC_F32 ? (ch + split) % chunks : ch) * CW;
            if constexpr (MODE != TMA_WIDE) {
                if (MODE == TMA_NARROW || !g.wide) {
                    store_chunk<EPI, CW>(g, taddr + c0, scr, row0, n0 + c0);
                    continue;
                }
            }
            C::put(scr, taddr + c0, lane);
            const int n = n0 + c0 + C::col(lane);
            float2 b[4] = {}, cs[4] = {};
            if ((EPI == EPI_F32 || EPI == EPI_BIAS_GELU) && g.bias) {
                const float4 u = __ldg(reinterpret_cast<const float4*>(g.bias + n));
                const float4 w = __ldg(reinterpret_cast<const float4*>(g.bias + n) + 1);
                b[0] = make_float2(u.x, u.y), b[1] = make_float2(u.z, u.w);
                b[2] = make_float2(w.x, w.y), b[3] = make_float2(w.z, w.w);
            }
#pragma unroll
            for (int pass = 0; pass < C::kPasses; ++pass) {
                const int row = row0 + C::row(pass, lane);
                const bool row_ok = row < g.M;
                const int64_t at = int64_t(row) * g.c_sm + n;
                float2 v[4];
                C::get(scr, pass, lane, v);
                if constexpr (EPI == EPI_ATOMIC_F32) {
                    if (row_ok) {
                        red_v4(g.out_f32 + at, v[0], v[1]);
                        red_v4(g.out_f32 + at + 4, v[2], v[3]);
                    }
                    continue;
                }
                if constexpr (EPI != EPI_GELU_GRAD) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[k] = __fadd2_rn(v[k], b[k]);
                    if (row_ok) st_v8((EPI == EPI_F32 ? g.out_f32 : g.z_f32) + at, v);
                    if constexpr (EPI == EPI_F32) continue;
                }
                uint32_t o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if constexpr (EPI == EPI_GELU_GRAD) o[k] = pack_bf16(__fmul2_rn(v[k], gelu_grad(z[pass * 4 + k])));
                    else o[k] = pack_bf16(gelu(v[k]));
                }
                if (row_ok) *reinterpret_cast<uint4*>(g.out_bf16 + at) = make_uint4(o[0], o[1], o[2], o[3]);
                if constexpr (EPI == EPI_GELU_GRAD) {
                    if (row_ok) {  // sums of the stored values
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            cs[k] = __fadd2_rn(cs[k], make_float2(__uint_as_float(o[k] << 16),
                                                                  __uint_as_float(o[k] & 0xffff0000u)));
                    }
                    const int tn = t + gridDim.x;
                    if (ch + 1 < chunks) load_z(pass, row0, n0 + c0 + CW);
                    else if (tn < g.tiles)
                        load_z(pass, tn % g.tiles_m * kBM + q * 32, tn / g.tiles_m % g.tiles_n * BN + cbeg);
                }
            }
            if constexpr (EPI == EPI_GELU_GRAD) {
                if (g.col_sum) {
                    // over the lanes with the same eight columns, halving the columns at
                    // each of the first three exchanges
                    float c[8] = {cs[0].x, cs[0].y, cs[1].x, cs[1].y, cs[2].x, cs[2].y, cs[3].x, cs[3].y};
#pragma unroll
                    for (int h = 4; h >= 1; h >>= 1) {
                        const bool up = lane & (4 * h);
#pragma unroll
                        for (int k = 0; k < h; ++k) {
                            const float give = up ? c[k] : c[k + h];
                            c[k] = (up ? c[k + h] : c[k]) + __shfl_xor_sync(~0u, give, 4 * h);
                        }
                    }
                    if (CW == 16) c[0] += __shfl_xor_sync(~0u, c[0], 2);
                    if (CW == 32 || !(lane & 2)) atomicAdd(g.col_sum + n + ((lane >> 2) & 7), c[0]);
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
    }
    return true;
}

// Ring: 3 x 48 KB, or 6 x 24 KB for 16 columns, beside the chunks of 16 epilogue
// warps (64 KB); 4 x 48 or 8 x 24 beside those of 8.
constexpr int stages(int bn, int mode) { return (bn == 256 ? 1 : 2) * (mode != COPIES ? 3 : 4); }

// A CTA walks 128 x BN output tiles (of one K split each), a grid apart.  One
// thread keeps the ring of stages full with TMA copies, another issues the
// MMAs and commits them to the stage's `empty` barrier and, after a tile's
// last stage, to the accumulator's; the epilogue warps empty one of the
// two accumulators while the next tile is summed in the other.  Operands that
// TMA does not take are copied by pairs of warps.
// What bounds it: the copies.  With cp.async a 48 KB stage took 1.7 us, on an
// idle GPU too (an SM keeps about 24 KB of such copies in flight), while its
// MMAs take 0.4 us.
template <int BN, int EPI, int MODE>
__global__ void __launch_bounds__(Warps<MODE>::kThreads, 1)
    k_gemm_tcgen05(const __grid_constant__ GemmArgs g, const __grid_constant__ CUtensorMap map_a,
                   const __grid_constant__ CUtensorMap map_b) {
    constexpr int kATile = kBM * kBK * 2;   // 16 KB
    constexpr int kBTile = (BN < 64 ? 64 : BN) * kBK * 2;  // an MN-major box has 64 rows
    constexpr int kStage = kATile + kBTile;
    constexpr int kEpiWarps = Warps<MODE>::kEpi, kLoadWarps = Warps<MODE>::kLoad;
    constexpr int STAGES = stages(BN, MODE);
    constexpr uint32_t kAccCols = BN < 32 ? 32 : BN;
    constexpr uint32_t kTmemCols = 2 * kAccCols;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], drain;
    __shared__ uint32_t tmem_base_holder;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == kEpiWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_base_holder)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full[s]), MODE != COPIES ? 1 : 2);
            mbar_init(smem_u32(&empty[s]), 1);
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);
            mbar_init(smem_u32(&acc_empty[b]), kEpiWarps);
        }
        mbar_init(smem_u32(&drain), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_holder;

    bool ok = true;
    int issued = 0;  // TMA: stages filled by this thread
    const bool a_mn = g.a_mode == ST_MN_VEC, b_mn = g.b_mode == ST_MN_VEC;
    if (MODE != COPIES && warp > kEpiWarps) {
        if (threadIdx.x == (kEpiWarps + 1) * 32) {
            constexpr int kBoxesA = kBM / 64, kBoxesB = BN < 64 ? 1 : BN / 64;  // MN-major: 64 rows each
            const uint32_t bytes = kATile + (b_mn ? kBoxesB * kMnBox : BN * kBK * 2);
            for (int t = blockIdx.x; ok && t < g.tiles; t += gridDim.x) {
                const int m0 = t % g.tiles_m * kBM, n0 = t / g.tiles_m % g.tiles_n * BN;
                const int kb = t / (g.tiles_m * g.tiles_n) * g.k_per_split;
                const int ke = min(g.K, kb + g.k_per_split);
                for (int k0 = kb; k0 < ke; k0 += kBK, ++issued) {
                    const int s = issued % STAGES, round = issued / STAGES;
                    if (round > 0) ok = mbar_wait(smem_u32(&empty[s]), uint32_t((round - 1) & 1), g.wait_limit);
                    if (!ok) break;
                    const uint32_t st_a = smem_u32(smem + s * kStage), st_b = st_a + kATile, bar = smem_u32(&full[s]);
                    mbar_expect(bar, bytes);
                    if (a_mn) {
#pragma unroll
                        for (int b = 0; b < kBoxesA; ++b) tma_load(st_a + b * kMnBox, &map_a, m0 + b * 64, k0, bar);
                    } else {
                        tma_load(st_a, &map_a, k0, m0, bar);
                    }
                    if (b_mn) {
#pragma unroll
                        for (int b = 0; b < kBoxesB; ++b) tma_load(st_b + b * kMnBox, &map_b, n0 + b * 64, k0, bar);
                    } else {
                        tma_load(st_b, &map_b, k0, n0, bar);
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp > kEpiWarps) {
        // A pair owns its stages, so the phase it waits for is the one after the last
        // it saw: with a stage filled by several pairs in turn the parity would not
        // tell a phase from the one two before it.
        static_assert(MODE != COPIES || STAGES % (kLoadWarps / 2) == 0, "a loading pair owns its stages");
        constexpr int kPairs = kLoadWarps > 1 ? kLoadWarps / 2 : 1;
        const int mine = (warp - kEpiWarps - 1) / 2, tid = (threadIdx.x - (kEpiWarps + 1) * 32) & 63;
        int c = 0;  // stages filled so far by all pairs
        for (int t = blockIdx.x; ok && t < g.tiles; t += gridDim.x) {
            const int m0 = t % g.tiles_m * kBM, n0 = t / g.tiles_m % g.tiles_n * BN;
            const int kb = t / (g.tiles_m * g.tiles_n) * g.k_per_split;
            const int ke = min(g.K, kb + g.k_per_split);
            for (int k0 = kb; k0 < ke; k0 += kBK, ++c) {
                if (c % kPairs != mine) continue;
                const int s = c % STAGES, round = c / STAGES;
                if (round > 0) {
                    ok = mbar_wait(smem_u32(&empty[s]), uint32_t((round - 1) & 1), g.wait_limit);
                    ok = __all_sync(~0u, ok);
                    if (!ok) break;
                }
                unsigned char* st = smem + s * kStage;
                const int kn = min(kBK, (ke - k0 + 15) & ~15);
                stage_operand<kBM>(st, g.a, g.a_sm, g.a_sk, g.a_mode, m0, g.M, k0, ke, kn, tid);
                stage_operand<BN>(st + kATile, g.b, g.b_sn, g.b_sk, g.b_mode, n0, g.N, k0, ke, kn, tid);
                cp_async_wait_all();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&full[s]));
            }
        }
    } else if (warp == kEpiWarps) {
        if (lane == 0) {
            const uint32_t idesc = make_idesc(BN) | (uint32_t(a_mn) << 15) | (uint32_t(b_mn) << 16);
            int c = 0, i = 0;
            for (int t = blockIdx.x; ok && t < g.tiles; t += gridDim.x, ++i) {
                const int kb = t / (g.tiles_m * g.tiles_n) * g.k_per_split;
                const int ke = min(g.K, kb + g.k_per_split);
                const int acc = i & 1, use = i >> 1;
                if (use > 0) ok = mbar_wait(smem_u32(&acc_empty[acc]), uint32_t((use - 1) & 1), g.wait_limit);
                bool skipped = false;
                for (int k0 = kb; ok && k0 < ke; k0 += kBK, ++c) {
                    const int s = c % STAGES;
                    ok = mbar_wait(smem_u32(&full[s]), uint32_t((c / STAGES) & 1), g.wait_limit);
                    if (!ok) break;
                    if ((k0 - kb) / kBK == g.skip_stage) {
                        skipped = true;
                        continue;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_base = smem_u32(smem + s * kStage), b_base = a_base + kATile;
                    const int steps = (min(kBK, ke - k0) + 15) / 16;
                    for (int j = 0; j < steps; ++j)
                        mma_bf16(tmem + acc * kAccCols, make_desc(a_base + j * k16_step(a_mn), a_mn),
                                 make_desc(b_base + j * k16_step(b_mn), b_mn), idesc, (k0 > kb || j > 0) ? 1u : 0u);
                    mma_commit(smem_u32(&empty[s]));
                }
                if (ok && !skipped) mma_commit(smem_u32(&acc_full[acc]));
            }
        }
        __syncwarp();
    } else {
        // warp w: the TMEM lanes of quarter w % 4 (the rows it may access), column group w / 4
        constexpr int kGroups = kEpiWarps / 4;
        constexpr int GC = (BN / kGroups >= 16) ? BN / kGroups : BN;
        const int q = warp & 3, cbeg = (warp >> 2) * GC;
        ok = epilogue<BN, EPI, MODE>(g, tmem, kAccCols, acc_full, acc_empty,
                               smem + STAGES * kStage + warp * kScratch, q, cbeg, cbeg < BN ? cbeg + GC : cbeg);
    }
    if (!__syncthreads_and(ok)) {
        if (threadIdx.x == kEpiWarps * 32) {
            atomicOr(g.error, 1);
            // A wait ran out, so MMAs committed earlier may not have been waited
            // for: one more commit arrives on the drain barrier once every
            // tcgen05 operation this thread issued has completed; TMEM is freed
            // only after that (or after the bounded wait on it gives up).
            mma_commit(smem_u32(&drain));
            mbar_wait(smem_u32(&drain), 0u, kWaitLimit);
        }
        // ... nor the copies in flight, which write this CTA's shared memory
        for (int c = max(0, issued - STAGES); c < issued; ++c)
            mbar_wait(smem_u32(&full[c % STAGES]), uint32_t((c / STAGES) & 1), kWaitLimit);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kEpiWarps)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// The driver's tensor map encoder, or null where the driver has none.
PFN_cuTensorMapEncodeTiled tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &found) !=
                cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(f);
    }();
    return fn;
}

// Tensor map of one operand (`rows` x K, its contiguous axis given by `mode`)
// in boxes of 64 elements of that axis by `lines` of the other, 128-byte
// swizzle, zeros outside.  False where TMA does not take it: element-wise
// operands, rows that overlap or run backwards, strides of 2^40 bytes.
bool encode_operand(CUtensorMap* map, const void* p, long long s_r, long long s_k, int mode, int rows, int K,
                    int lines) {
    if (mode == ST_SCALAR) return false;
    const bool mn = mode == ST_MN_VEC;
    const long long inner = mn ? rows : K, outer = mn ? K : rows, stride = mn ? s_k : s_r;
    if (stride < inner || stride >= (1ll << 39)) return false;
    const PFN_cuTensorMapEncodeTiled encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[2] = {cuuint64_t(inner), cuuint64_t(outer)}, strides[1] = {cuuint64_t(stride) * 2};
    const cuuint32_t box[2] = {64, cuuint32_t(lines)}, steps[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, steps,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int EPI, int MODE>
int launch_kernel(const GemmArgs& g, const CUtensorMap& map_a, const CUtensorMap& map_b, int ctas, cudaStream_t st) {
    constexpr int kSmem = stages(BN, MODE) * (kBM + (BN < 64 ? 64 : BN)) * kBK * 2 + Warps<MODE>::kEpi * kScratch;
    GSV_CUDA_TRY(cudaFuncSetAttribute(k_gemm_tcgen05<BN, EPI, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kSmem));
    k_gemm_tcgen05<BN, EPI, MODE><<<ctas, Warps<MODE>::kThreads, kSmem, st>>>(g, map_a, map_b);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

// One CTA per SM: the ring, the epilogue warps' chunks and both accumulators
// (all 512 TMEM columns for 256) fill it.
template <int BN, int EPI>
int launch_tiles(const GemmArgs& g, cudaStream_t st) {
    int dev = 0, sms = 0;
    GSV_CUDA_TRY(cudaGetDevice(&dev));
    GSV_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int ctas = g.tiles < sms ? g.tiles : sms;
    CUtensorMap map_a{}, map_b{};
    if (encode_operand(&map_a, g.a, g.a_sm, g.a_sk, g.a_mode, g.M, g.K, g.a_mode == ST_MN_VEC ? kBK : kBM) &&
        encode_operand(&map_b, g.b, g.b_sn, g.b_sk, g.b_mode, g.N, g.K, g.b_mode == ST_MN_VEC ? kBK : BN))
        return g.wide ? launch_kernel<BN, EPI, TMA_WIDE>(g, map_a, map_b, ctas, st)
                      : launch_kernel<BN, EPI, TMA_NARROW>(g, map_a, map_b, ctas, st);
    return launch_kernel<BN, EPI, COPIES>(g, map_a, map_b, ctas, st);
}

template <int EPI>
int launch_gemm(const GemmArgs& g, int bn, cudaStream_t st) {
    return bn == 256 ? launch_tiles<256, EPI>(g, st) : launch_tiles<16, EPI>(g, st);
}

// Operand copy mode: 16-byte cp.async needs a 16-byte aligned base and a
// contiguous axis whose neighbours sit a multiple of 8 elements apart.
int stage_mode(const void* p, long long s_r, long long s_k) {
    const bool aligned = (reinterpret_cast<uintptr_t>(p) & 15) == 0;
    if (aligned && s_k == 1 && s_r % 8 == 0) return ST_K_VEC;
    if (aligned && s_r == 1 && s_k % 8 == 0) return ST_MN_VEC;
    return ST_SCALAR;
}

int mlp_gemm(const void* a, long long a_sm, long long a_sk, const void* b, long long b_sn, long long b_sk, int M,
             int N, int K, int splits, const float* bias, float* out_f32, void* out_bf16, float* z_f32,
             long long c_sm, long long c_sn, int epi, float* col_sum, int* error, void* stream,
             long long wait_limit, int skip_stage) {
    if (!a || !b || !error || M <= 0 || N <= 0 || K <= 0 || (N % 16) != 0 || splits <= 0) return GSV_ERR_INVALID_ARGUMENT;
    if (epi < EPI_F32 || epi > EPI_ATOMIC_F32) return GSV_ERR_INVALID_ARGUMENT;
    if (splits > 1 && epi != EPI_ATOMIC_F32) return GSV_ERR_INVALID_ARGUMENT;
    if ((epi == EPI_F32 || epi == EPI_ATOMIC_F32) && !out_f32) return GSV_ERR_INVALID_ARGUMENT;
    if ((epi == EPI_BIAS_GELU || epi == EPI_GELU_GRAD) && (!out_bf16 || !z_f32)) return GSV_ERR_INVALID_ARGUMENT;
    if (col_sum && (epi != EPI_GELU_GRAD || c_sn != 1)) return GSV_ERR_INVALID_ARGUMENT;
    GemmArgs g{};
    g.a = static_cast<const __nv_bfloat16*>(a);
    g.b = static_cast<const __nv_bfloat16*>(b);
    g.a_sm = a_sm; g.a_sk = a_sk; g.b_sn = b_sn; g.b_sk = b_sk;
    g.M = M; g.N = N; g.K = K;
    const int kchunks = (K + kBK - 1) / kBK;
    const int per = (kchunks + splits - 1) / splits;
    g.k_per_split = per * kBK;
    const int zs = (K + g.k_per_split - 1) / g.k_per_split;
    g.bias = bias; g.out_f32 = out_f32; g.out_bf16 = static_cast<__nv_bfloat16*>(out_bf16); g.z_f32 = z_f32;
    g.c_sm = c_sm; g.c_sn = c_sn; g.epi = epi; g.col_sum = col_sum; g.error = error;
    g.wait_limit = wait_limit; g.skip_stage = skip_stage;
    g.a_mode = stage_mode(a, a_sm, a_sk);
    g.b_mode = stage_mode(b, b_sn, b_sk);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int bn = (N % 256 == 0) ? 256 : 16;
    g.tiles_m = (M + kBM - 1) / kBM;
    g.tiles_n = N / bn;
    const long long tiles = (long long)g.tiles_m * g.tiles_n * zs;
    if (tiles > INT_MAX - 65536) return GSV_ERR_INVALID_ARGUMENT;
    g.tiles = int(tiles);
    auto aligned = [](const void* p, unsigned bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; };
    g.wide = c_sn == 1 && c_sm % 8 == 0 && aligned(out_f32, 32) && aligned(out_bf16, 16) && aligned(z_f32, 32) &&
             aligned(bias, 16);
    int rc = GSV_OK;
    switch (epi) {
        case EPI_F32: rc = launch_gemm<EPI_F32>(g, bn, st); break;
        case EPI_BIAS_GELU: rc = launch_gemm<EPI_BIAS_GELU>(g, bn, st); break;
        case EPI_GELU_GRAD: rc = launch_gemm<EPI_GELU_GRAD>(g, bn, st); break;
        default: rc = launch_gemm<EPI_ATOMIC_F32>(g, bn, st); break;
    }
    return rc;
}

}  // namespace

extern "C" {

int gsv_mlp_gemm(const void* a, long long a_sm, long long a_sk, const void* b, long long b_sn,
                         long long b_sk, int M, int N, int K, int splits, const float* bias, float* out_f32,
                         void* out_bf16, float* z_f32, long long c_sm, long long c_sn, int epi, float* col_sum,
                         int* error, void* stream) {
    return mlp_gemm(a, a_sm, a_sk, b, b_sn, b_sk, M, N, K, splits, bias, out_f32, out_bf16, z_f32, c_sm, c_sn, epi,
                    col_sum, error, stream, kWaitLimit, -1);
}

int gsv_mlp_gemm_test_timeout(const void* a, const void* b, int M, int N, int K, float* out_f32, int skip_stage,
                              long long wait_limit, int* error, void* stream) {
    if (skip_stage < 0 || skip_stage >= (K + kBK - 1) / kBK) return GSV_ERR_INVALID_ARGUMENT;
    if (wait_limit <= 0 || wait_limit > kWaitLimit) return GSV_ERR_INVALID_ARGUMENT;
    return mlp_gemm(a, K, 1, b, K, 1, M, N, K, 1, nullptr, out_f32, nullptr, nullptr, N, 1, EPI_F32, nullptr, error,
                    stream, wait_limit, skip_stage);
}

}  // extern "C"
