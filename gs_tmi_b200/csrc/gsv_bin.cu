// gsv_bin.cu -- preprocess and tile binning (counting sort or device radix sort), sm_100a.
//
// Binning is bit-exact with build_tile_pairs (3DGS/3dgsVC/gaussian/
// tile_voxelizer.py:87-162): the FP32 center/radius follow :284-286 op for
// op, the voxel box uses floor/ceil + clamp (:97-105), the tile box integer
// division + clamp (:107-114), pairs are generated Gaussian-major in
// (d,h,w) raster order (:126-145) and stably sorted by tile id, so each
// tile's list is in ascending Gaussian id; empty tiles keep range (0,0)
// (:151-161).  Unlike the reference there is no host synchronisation unless
// the caller asks for the pair total.
#include <cub/cub.cuh>

#include <cstdio>
#include <cstring>

#include "gsv_common.cuh"

using namespace gsv;

namespace {

thread_local char g_last_error[512] = {0};

constexpr int kMaxTilesPerAxis = 65535;  // box packing: 16 bits per field

struct ShapeInfo {
    int32_t d, h, w, ts, ntd, nth, ntw;
    int64_t ntiles;
    bool ok;
};

ShapeInfo shape_info(gsv_shape s) {
    ShapeInfo r{};
    r.ok = s.d > 0 && s.h > 0 && s.w > 0 && s.tile_size > 0 && s.d < (1 << 24) && s.h < (1 << 24) &&
           s.w < (1 << 24);
    if (!r.ok) return r;
    r.d = s.d; r.h = s.h; r.w = s.w; r.ts = s.tile_size;
    r.ntd = (s.d + s.tile_size - 1) / s.tile_size;
    r.nth = (s.h + s.tile_size - 1) / s.tile_size;
    r.ntw = (s.w + s.tile_size - 1) / s.tile_size;
    r.ok = r.ntd <= kMaxTilesPerAxis && r.nth <= kMaxTilesPerAxis && r.ntw <= kMaxTilesPerAxis;
    r.ntiles = int64_t(r.ntd) * r.nth * r.ntw;
    r.ok = r.ok && r.ntiles < (int64_t(1) << 30);
    return r;
}

int sort_end_bit(int64_t ntiles) {
    // keys are tile ids in [0, ntiles]; ntiles is the padding sentinel.
    int bits = 1;
    while ((int64_t(1) << bits) <= ntiles) ++bits;
    return bits;
}

// The preprocess scans the per-Gaussian pair counts in one pass (decoupled
// look-back): blocks of kPrepThreads Gaussians, one 64-bit look-back word per
// block after the Status struct, all cleared by the one memset of the status
// region that starts every preprocess.
constexpr int kPrepThreads = 256;
__host__ __device__ inline int64_t prep_blocks(int64_t n) { return (n + 1 + kPrepThreads - 1) / kPrepThreads; }

// Counting-sort binning, used unless the tile grid is large for the pairs (cs_pays).  The pairs'
// final order is fixed by two facts: a tile's list holds its Gaussians in
// ascending id, and Gaussians are handled in rows of consecutive ids.  The
// kernel that counts the pairs, or k_count_rows, also writes, per row, how many of the row's
// pairs fall in each tile (rows x tiles 16-bit counts, "cs_mat", rows padded
// to whole words); k_colscan writes, per row and tile, the position of the
// row's first pair of that tile in the sorted output ("cs_pos": the column's
// exclusive prefix plus the tile's start, from a single-pass scan of the tile
// totals) and the tile ranges; k_scatter places each row's pairs.  The result
// equals the stable radix sort's, which larger problems keep.  The counts
// stay intact and k_scatter clears k_colscan's scan state, so binning may be
// repeated after one preprocess (e.g. with a larger capacity).
//
// A row is 64 Gaussians, which gives k_scatter many short blocks, while there
// are no more rows than tiles (a column of k_colscan grows with the rows, a
// block of k_scatter with the tiles), few row counts and at most 4096 tiles (4845:
// 50,000 Gaussians 52.1 and 49.6); otherwise 256 (a block of the counting kernel).
// Preprocess and binning with rows of 64, of 256 and the radix sort, us:
//   tiles  Gaussians (pairs each)   64    256   radix
//     512    20,000 (15)           28.5   30.9   55.4
//     512    60,000 (11)           40.3   37.3
//     512   200,000 (6)            65.0   52.7   79.2
//    1728   120,000 (15)           59.2   56.7
//    3072    50,000 (36)           48.9   54.6   87.4
//    3072    75,000 (11)           50.0   46.5
//    3072    85,000 (11)           55.7   53.3
//    3072    85,000 (38)           68.7   71.8
//    3072   200,000 (16)           92.8   79.5  126
//    3072   500,000 (10)          210    140    182
//    3072   800,000 (8)                  198    228
//    3072 1,300,000 (6)                  297    298
//    3456     2,000 (11)           27.7   32.9
//    3456    20,000 (38)           40.8   46.0
//    3456    40,000 (77)           61.4   74.2
//    3456    50,000 (12)           42.5   45.1
//    3456    64,000 (12)           43.2   42.1
//    3840    50,000 (39)           54.4   60.2
//    4096    50,000 (39)           54.9   60.9
//    4096    60,000 (39)           60.3   61.1
//    9216   154,793 (36)                 130    159
//    9216   400,000 (20)                 251    224
//   13824    40,000 (139)                133    179
//   13824   300,000 (35)                 248    247
//   18432   230,000 (45)                 253    245
// k_scatter's lanes per Gaussian, by the row's mean pairs a Gaussian: up to 12 eight, up to 24 sixteen, above a
// warp.  k_scatter with 8, 16 and 32 lanes, us: 10 pairs 59, 64, 88; 15 pairs 8.1, 7.4, 8.4; 36 pairs 20.6, 17.4,
// 16.3; 139 pairs 130, 95, 84.
constexpr int64_t kCsNarrow8 = 12, kCsNarrow16 = 24;
constexpr int kCsSub = 64;  // Gaussians k_scatter places at a time: a bit each in a tile's word
constexpr int64_t kCsShortTiles = 4096;                // 64-Gaussian rows up to here: four rows of counters
constexpr int64_t kCsShortCells = 3500000;             // ... and up to this many row counts
constexpr int64_t kCsSmallTiles = 3072;                // up to here always the counting sort (cs_pays), with
constexpr int64_t kCsMaxTiles = 18432;                 // 12 bytes per tile in k_scatter's shared memory (227 KB)
constexpr int64_t kCsMaxCells = int64_t(1) << 23;      // ... twice these 16 MB of counts and 32 MB of positions
constexpr int kCsCols = 32, kCsRowGroups = 32;         // k_colscan block: 32 columns x 32 row groups
__host__ __device__ inline int64_t cs_row_len(int64_t n, int64_t ntiles) {
    const int64_t rows = prep_blocks(n) * (kPrepThreads / kCsSub);
    return ntiles <= kCsShortTiles && rows <= ntiles && rows * ntiles <= kCsShortCells ? kCsSub : kPrepThreads;
}
__host__ __device__ inline int64_t cs_rows(int64_t n, int64_t ntiles) {
    return prep_blocks(n) * (kPrepThreads / cs_row_len(n, ntiles));
}
__host__ __device__ inline int64_t cs_col_blocks(int64_t ntiles) { return (ntiles + kCsCols - 1) / kCsCols; }
__host__ __device__ inline int64_t cs_mstride(int64_t ntiles) { return (ntiles + 1) & ~int64_t(1); }  // counts per row
inline bool cs_eligible(int64_t n, int64_t ntiles) {
    return n > 0 && ntiles <= kCsMaxTiles &&
           cs_rows(n, ntiles) * ntiles <= (ntiles <= kCsSmallTiles ? 2 * kCsMaxCells : kCsMaxCells);
}
// Up to kCsSmallTiles tiles the counting sort is the faster one from 50 Gaussians to a million.  On larger grids
// its row counts have to pay: their filling and scanning grow with rows x tiles (7 us a million), the radix sort
// with the pairs (20 us a million more than 50, where one block cannot sort them; its buffers are the
// capacity's size).  Where the Gaussians alone decide for the counting sort (each has a pair at least), the
// kernel that counts a Gaussian's pairs fills its rows of cs_mat at once; elsewhere gsv_bin decides, and only
// then are the rows counted, by a kernel of their own (3 us more).  Preprocess and binning, us:
//   tiles  Gaussians  row counts    pairs   counting   radix
//    3456        50     0.003 M       163     18.8      16.5
//   18432       500     0.04 M      1,551     33.7      18.2
//    3456     2,000     0.03 M      6,199     25.0      48.8
//   18432     5,000     0.4 M      15,967     36.7      50.4
//    9120   100,000     3.6 M     320,000     54.1      58.8
//    4096   300,000     4.8 M     946,000     72.9      79.5
//   13824   100,000     5.4 M     319,000     73.5      57.9
//   18432   100,000     7.2 M     320,000     83.9      56.9
//    6000   300,000     7.0 M     948,000     93.8      77.5
//   13824   100,000     5.4 M   2,440,000      101      95.4
//   18432   100,000     7.2 M   2,460,000      116      97.7
//    9216   154,793     5.6 M   5,570,000      130       159
constexpr int64_t kCsFewPairs = 4096, kCsFreeCells = 3900000;
inline int64_t cs_cells(int64_t n, int64_t ntiles) { return cs_rows(n, ntiles) * ntiles; }
inline bool cs_pays(int64_t n, int64_t ntiles, int64_t pairs) {
    return ntiles <= kCsSmallTiles || (pairs > kCsFewPairs && cs_cells(n, ntiles) < kCsFreeCells + pairs);
}
inline bool cs_fused(int64_t n, int64_t ntiles) { return cs_pays(n, ntiles, n); }

// Status region: the Status word, the preprocess's look-back words (one per
// block), then k_colscan's (one per column block).  Status::pad[1] and
// pad[2] are the two launches' block-ticket counters.
__host__ __device__ inline size_t status_bytes(int64_t n, int64_t ntiles) {
    return sizeof(Status) + size_t(prep_blocks(n) + cs_col_blocks(ntiles)) * sizeof(unsigned long long);
}

GaussLayout gauss_layout(int64_t n, const ShapeInfo& si) {
    GaussLayout L{};
    size_t o = 0;
    L.rec = o;      o = align_up(o + size_t(n) * sizeof(Rec));
    L.ext = o;      o = align_up(o + size_t(n) * sizeof(float4));
    L.box = o;      o = align_up(o + size_t(n) * sizeof(int4));
    L.offsets = o;  o = align_up(o + size_t(n + 1) * sizeof(int64_t));
    L.ranges = o;   o = align_up(o + size_t(si.ntiles) * sizeof(int2));
    L.accum = o;    o = align_up(o + size_t(n) * kMomStride * sizeof(float));
    L.status = o;   o = align_up(o + status_bytes(n, si.ntiles));
    L.cs = cs_eligible(n, si.ntiles);
    L.cs_mat = o;   o = align_up(o + (L.cs ? size_t(cs_rows(n, si.ntiles) * cs_mstride(si.ntiles)) * sizeof(uint16_t) : 0));
    L.cs_pos = o;   o = align_up(o + (L.cs ? size_t(cs_rows(n, si.ntiles) * si.ntiles) * sizeof(int32_t) : 0));
    L.total = o;
    return L;
}

PairLayout pair_layout(int64_t cap, const ShapeInfo& si, int flags) {
    PairLayout L{};
    size_t sort_bytes = 0;
    const int end_bit = sort_end_bit(si.ntiles);
    cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (const int32_t*)nullptr, (int32_t*)nullptr,
                                    (const int32_t*)nullptr, (int32_t*)nullptr, int(cap > 0 ? cap : 1),
                                    0, end_bit);
    L.sort_tmp_bytes = sort_bytes;
    size_t o = 0;
    const size_t c = size_t(cap > 0 ? cap : 1);
    L.keys_in = o;  o = align_up(o + c * sizeof(int32_t));
    L.vals_in = o;  o = align_up(o + c * sizeof(int32_t));
    L.keys_out = o; o = align_up(o + c * sizeof(int32_t));
    L.vals_out = o; o = align_up(o + c * sizeof(int32_t));
    L.sort_tmp = o; o = align_up(o + sort_bytes);
    L.partials = o;
    if (flags & GSV_BACKWARD_DETERMINISTIC) o = align_up(o + c * kMomStride * sizeof(float));
    L.total = o;
    return L;
}

template <typename T>
T* at(void* base, size_t off) {
    return reinterpret_cast<T*>(static_cast<char*>(base) + off);
}
template <typename T>
const T* at(const void* base, size_t off) {
    return reinterpret_cast<const T*>(static_cast<const char*>(base) + off);
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

struct DevShape {
    int32_t size[3];
    int32_t nt[3];
    int32_t ts;
    float shape_f[3];
    float hs[3];
    float ih[3];
};

DevShape dev_shape(const ShapeInfo& si) {
    DevShape s{};
    s.size[0] = si.d; s.size[1] = si.h; s.size[2] = si.w;
    s.nt[0] = si.ntd; s.nt[1] = si.nth; s.nt[2] = si.ntw;
    s.ts = si.ts;
    for (int a = 0; a < 3; ++a) {
        s.shape_f[a] = float(s.size[a]);
        s.hs[a] = s.shape_f[a] * 0.5f;
        s.ih[a] = 1.0f / s.hs[a];  // host IEEE division, same as the device __fdiv_rn
    }
    return s;
}

// Tile box of one Gaussian; returns the tile count (<= 0 for an empty box).
__device__ __forceinline__ int64_t tile_box(const DevShape& s, const float c[3], float r, int4* box) {
    int32_t tlo[3], na[3];
    int64_t cnt = 1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // (center_vox - r3).floor().int() / (center_vox + r3).ceil().int(), clamp (:97-105)
        int32_t lo = __float2int_rz(floorf(__fsub_rn(c[a], r)));
        int32_t hi = __float2int_rz(ceilf(__fadd_rn(c[a], r)));
        lo = min(max(lo, 0), s.size[a] - 1);
        hi = min(max(hi, 0), s.size[a] - 1);
        // // tile_size, clamp (:107-114); lo, hi >= 0 here so C division == floor division
        int32_t t0 = min(max(lo / s.ts, 0), s.nt[a] - 1);
        int32_t t1 = min(max(hi / s.ts, 0), s.nt[a] - 1);
        tlo[a] = t0;
        na[a] = t1 - t0 + 1;
        if (na[a] <= 0) cnt = 0;
        else cnt *= na[a];
    }
    box->x = tlo[0] | (tlo[1] << 16);
    box->y = tlo[2] | (max(na[0], 0) << 16);
    box->z = max(na[1], 0) | (max(na[2], 0) << 16);
    box->w = int32_t(cnt);
    return cnt;
}

// Look-back word of a block: flag in the top two bits, an int64 pair count
// below.  kLbAgg: the block's own total; kLbPre: the total of every block up
// to and including it.
constexpr unsigned long long kLbAgg = 1ull << 62, kLbPre = 2ull << 62, kLbVal = (1ull << 62) - 1;
constexpr int kLbSpinLimit = 1 << 22;  // polls of one predecessor's word before giving up

__device__ __forceinline__ unsigned long long lb_load(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void lb_store(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Decoupled look-back of scan block `bid`, run by all 32 lanes of one warp:
// publishes the block's total, walks back over the predecessors' words and
// returns the sum of every earlier block's total (the same in all lanes),
// after publishing its own inclusive prefix.  Lane l reads the word of block
// j - l, so one step covers 32 predecessors; the nearest inclusive prefix
// (kLbPre) in the window ends the walk, and every word in front of it must
// be published (flag set) before the window is summed, else the step is
// retried.  Block ids come from a ticket counter, so every block waited for
// has started.  Each retry is bounded: on time-out GSV_FLAG_SCAN_STALLED is
// latched and the block publishes what it has, so no later block waits the
// full limit again.
// A word carries all that is passed on, so it needs no ordering against other
// accesses: acquire and release, which wait for the block's record stores,
// cost 50,000 Gaussians 2 us (k_prepare and k_colscan) and 2M 11 us.  Two to
// eight windows in flight a step measured the same or slower (2M: 172 to 187 us
// against 161): they only poll more.
__device__ int64_t lookback(unsigned long long* lb, int64_t bid, int64_t block_tot, Status* status, int lane) {
    if (bid == 0) {
        if (lane == 0) lb_store(&lb[0], kLbPre | (unsigned long long)block_tot);
        return 0;
    }
    if (lane == 0) lb_store(&lb[bid], kLbAgg | (unsigned long long)block_tot);
    int64_t base = 0;
    int64_t j = bid - 1;  // the window's nearest predecessor
    int spins = 0;
    while (true) {
        const int64_t idx = j - lane;
        // before block 0 there is nothing: an inclusive prefix of zero
        const unsigned long long v = idx >= 0 ? lb_load(&lb[idx]) : kLbPre;
        const unsigned long long f = v & ~kLbVal;
        const unsigned pre = __ballot_sync(0xffffffffu, f == kLbPre);
        const int first = pre ? __ffs(pre) - 1 : 31;  // last lane of this step
        const unsigned upto = first == 31 ? 0xffffffffu : (2u << first) - 1u;
        const unsigned missing = __ballot_sync(0xffffffffu, f == 0) & upto;
        if (missing) {
            if (++spins > kLbSpinLimit) {
                if (lane == 0) atomicOr(&status->flags, GSV_FLAG_SCAN_STALLED);
                break;
            }
            continue;
        }
        spins = 0;
        int64_t part = ((upto >> lane) & 1u) ? int64_t(v & kLbVal) : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        base += part;
        if (pre) break;
        j -= 32;
    }
    if (lane == 0) lb_store(&lb[bid], kLbPre | (unsigned long long)(base + block_tot));
    return base;
}

// Tile id of pair `c` (0-based, raster order) of a Gaussian's packed tile box,
// for the counting sort, where the pair index and both box extents are at most
// the tile count (<= kCsMaxTiles): the two integer divisions become
// trunc((x + 0.5) * rcp(n)) in IEEE single precision, a few instructions
// instead of about twenty each.  Exact: (x + 0.5) / n lies at least 0.5 / n from
// an integer, and the two roundings move it by at most 1.2e-7 (x + 0.5) / n, less
// than that for x below four million.  r1, r2: __frcp_rn of the box's n1, n2.
__device__ __forceinline__ int32_t small_div(int32_t x, float rcp_n) {
    return __float2int_rz(__fmul_rn(__fadd_rn(float(x), 0.5f), rcp_n));
}
__device__ __forceinline__ int32_t box_tile_small(const DevShape& s, int bx, int by, int bz, float r1, float r2,
                                                  int32_t c) {
    const int32_t t0 = bx & 0xffff, t1 = (bx >> 16) & 0xffff, t2 = by & 0xffff;
    const int32_t n1 = bz & 0xffff, n2 = (bz >> 16) & 0xffff;
    const int32_t r = small_div(c, r2), k = c - r * n2;
    const int32_t i = small_div(r, r1), jj = r - i * n1;
    return ((t0 + i) * s.nt[1] + (t1 + jj)) * s.nt[2] + (t2 + k);
}
__device__ __forceinline__ float box_rcp(int field) { return __frcp_rn(float(max(field & 0xffff, 1))); }

// The exclusive scan of the Gaussians' pair counts into `offsets`
// (offsets[n] = pair total, also in Status::total), inside the kernel that
// counts them, a thread per Gaussian.  Blocks take their position in the scan
// from a counter in the status region, so every block a block waits for has
// already started.
__device__ __forceinline__ int64_t scan_ticket(Status* status) {
    __shared__ int bid_s;
    if (threadIdx.x == 0) bid_s = atomicAdd(&status->pad[1], 1);
    __syncthreads();
    return bid_s;
}

struct PairScan {
    int64_t first;     // this Gaussian's first pair, counted within the block
    int64_t warp_end;  // one past the warp's last
};

__device__ __forceinline__ PairScan scan_counts(int64_t cnt, int64_t n, int64_t bid, int64_t* __restrict__ offsets,
                                                Status* status) {
    __shared__ int64_t warp_tot[kPrepThreads / 32];
    __shared__ int64_t block_base;
    const int64_t g = bid * kPrepThreads + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int64_t warp_base = 0, block_tot = 0;
#pragma unroll
    for (int w = 0; w < kPrepThreads / 32; ++w) {
        if (w < warp) warp_base += warp_tot[w];
        block_tot += warp_tot[w];
    }
    if (warp == 0) {
        const int64_t base = lookback(reinterpret_cast<unsigned long long*>(status + 1), bid, block_tot, status, lane);
        if (lane == 0) block_base = base;
    }
    __syncthreads();
    const int64_t first = warp_base + incl - cnt;
    if (g <= n) offsets[g] = block_base + first;
    if (g == n) status->total = block_base + first;
    return PairScan{first, warp_base + warp_tot[warp]};
}

// A block's rows of cs_mat (`row_len` Gaussians each): their pairs per tile.  A row
// has at most row_len pairs in a tile, so the counters are 16-bit, two to a word,
// in shared memory (dynamic: ceil(ntiles / 2) words a row) and in cs_mat alike: the
// rows go out as the same words.  A warp whose Gaussians have many tiles takes
// them one after the other, its lanes a Gaussian's tiles; otherwise its lanes
// stride over its pairs, the block-local range [o of lane 0, warp_end), lane l's
// Gaussian the part starting at o, and find each pair's Gaussian by a shuffle
// search over the 32 starts (zero-count lanes share their successor's start
// and are never chosen).  The first costs little more with more pairs, the second a search for each: they cross
// at 16 pairs a Gaussian.  k_prepare, first and second way, us: 20,000 Gaussians with 6 pairs 16.3 and
// 13.5, 15 pairs 16.1 and 16.1, 24 pairs 16.6 and 19.0; 100,000 with 11 pairs 25.0 and 22.8, 16 pairs 24.7
// and 24.5, 18 pairs 25.3 and 25.9, 27 pairs 26.2 and 29.7.
constexpr int kCountWide = 16;
__device__ __forceinline__ void count_rows(const DevShape& s, int4 box, const PairScan& sc, int64_t bid, int row_len,
                                           uint16_t* __restrict__ cs_mat, int32_t ntiles) {
    constexpr unsigned kAll = 0xffffffffu;
    static_assert(kPrepThreads < 65536, "16-bit counters");
    extern __shared__ uint32_t cs_hist[];  // [rows][words]: counter of tile t in word t / 2
    const int lane = threadIdx.x & 31;
    const int words = (ntiles + 1) >> 1, all = words * (kPrepThreads / row_len);
    for (int i = threadIdx.x; i < all; i += kPrepThreads) cs_hist[i] = 0u;
    __syncthreads();
    uint32_t* row = cs_hist + (threadIdx.x / row_len) * words;  // warp-uniform: row_len is a multiple of 32
    const long long o = sc.first;
    const long long wstart = __shfl_sync(kAll, o, 0);
    const long long wend = sc.warp_end;
    const float rcp1 = box_rcp(box.z), rcp2 = box_rcp(box.z >> 16);
    if (wend - wstart >= 32 * kCountWide) {
        for (int j = 0; j < 32; ++j) {
            const int cnt = __shfl_sync(kAll, box.w, j);
            const int bx = __shfl_sync(kAll, box.x, j), by = __shfl_sync(kAll, box.y, j), bz = __shfl_sync(kAll, box.z, j);
            const float r1 = __shfl_sync(kAll, rcp1, j), r2 = __shfl_sync(kAll, rcp2, j);
            for (int c = lane; c < cnt; c += 32) {
                const int32_t t = box_tile_small(s, bx, by, bz, r1, r2, c);
                atomicAdd(&row[t >> 1], 1u << ((t & 1) * 16));
            }
        }
    } else {
        for (long long base = wstart; base < wend; base += 32) {
            const long long p = base + lane;
            int j = 0;  // largest j with o_j <= p
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const long long oj = __shfl_sync(kAll, o, j + step);
                if (oj <= p) j += step;
            }
            const long long oj = __shfl_sync(kAll, o, j);
            const int bx = __shfl_sync(kAll, box.x, j), by = __shfl_sync(kAll, box.y, j), bz = __shfl_sync(kAll, box.z, j);
            const float r1 = __shfl_sync(kAll, rcp1, j), r2 = __shfl_sync(kAll, rcp2, j);
            if (p < wend) {
                const int32_t t = box_tile_small(s, bx, by, bz, r1, r2, int32_t(p - oj));
                atomicAdd(&row[t >> 1], 1u << ((t & 1) * 16));
            }
        }
    }
    __syncthreads();
    // tile t's count is half t & 1 of its word (little-endian)
    uint32_t* dst = reinterpret_cast<uint32_t*>(cs_mat + bid * (kPrepThreads / row_len) * cs_mstride(ntiles));
    for (int i = threadIdx.x; i < all; i += kPrepThreads) dst[i] = cs_hist[i];
}

// Preprocess (center, radius, quadratic-form coefficients, tight extent, tile
// box) of one Gaussian per thread, the clearing of its backward moment
// accumulators, and the exclusive scan of the Gaussians'
// pair counts into `offsets` in the same launch (scan_counts).  With `cs_mat` the block
// also counts its pairs per tile (count_rows).
__global__ void __launch_bounds__(kPrepThreads) k_prepare(const float* __restrict__ pos,
                                                          const float* __restrict__ scl,
                                                          const float* __restrict__ rot,
                                                          const float* __restrict__ dr,
                                                          const float* __restrict__ di, int64_t dstride, int64_t n,
                                                          const int32_t* __restrict__ live, DevShape s,
                                                          Rec* __restrict__ recs, float4* __restrict__ ext,
                                                          int4* __restrict__ boxes,
                                                          int64_t* __restrict__ offsets, Status* status,
                                                          uint16_t* __restrict__ cs_mat, int32_t row_len,
                                                          int32_t ntiles, float* __restrict__ accum) {
    const int64_t bid = scan_ticket(status);
    const int64_t g = bid * kPrepThreads + threadIdx.x;
    int64_t cnt = 0;
    int4 box = make_int4(0, 0, 0, 0);
    if (g < n) {  // the backward's moment accumulators start from zero
        float4* acc4 = reinterpret_cast<float4*>(accum + g * kMomStride);
        acc4[0] = acc4[1] = acc4[2] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (g < n && live && g >= int64_t(*live)) {  // parked row: no tiles, no contribution
        recs[g] = Rec{};
        ext[g] = make_float4(0.f, 0.f, 0.f, 0.f);
        boxes[g] = make_int4(0, 0, 0, 0);
    } else if (g < n) {
        float p[3], sc[3], q[4];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            p[a] = pos[g * 3 + a];
            sc[a] = scl[g * 3 + a];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = rot[g * 4 + k];
        float c[3], sv[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            // center_vox = (positions + 1.0) * 0.5 * shape - 0.5   (:284)
            c[a] = __fsub_rn(__fmul_rn(__fmul_rn(__fadd_rn(p[a], 1.0f), 0.5f), s.shape_f[a]), 0.5f);
            sv[a] = __fmul_rn(sc[a], s.hs[a]);  // scale_vox (:285)
        }
        const float r = __fmul_rn(nanmax3(sv[0], sv[1], sv[2]), 3.0f);  // radius_vox (:286)
        float qc[6];
        qcoef_from_params(sc, q, s.ih, qc);
        Rec R;
        R.c0 = c[0]; R.c1 = c[1]; R.c2 = c[2];
        R.q00 = qc[0]; R.q01x2 = qc[1]; R.q02x2 = qc[2]; R.q11 = qc[3]; R.q12x2 = qc[4]; R.q22 = qc[5];
        R.rho_r = dr[g * dstride]; R.rho_i = di[g * dstride]; R.pad = 0.0f;
        recs[g] = R;
        ext[g] = tight_extent(qc);
        cnt = tile_box(s, c, r, &box);
        if (cnt <= 0) {
            atomicOr(&status->flags, GSV_FLAG_EMPTY_BOX);
            cnt = 0;
            box.w = 0;
        }
        boxes[g] = box;
    }
    const PairScan sc = scan_counts(cnt, n, bid, offsets, status);
    if (cs_mat != nullptr) count_rows(s, box, sc, bid, row_len, cs_mat, ntiles);  // block-uniform
}

// Tile boxes, pair counts and their scan for the reference-signature binning.
__global__ void __launch_bounds__(kPrepThreads) k_count_compat(const float* __restrict__ center,
                                                               const float* __restrict__ radius, int64_t n,
                                                               DevShape s, int4* __restrict__ boxes,
                                                               int64_t* __restrict__ offsets, Status* status,
                                                               uint16_t* __restrict__ cs_mat, int32_t row_len, int32_t ntiles) {
    const int64_t bid = scan_ticket(status);
    const int64_t g = bid * kPrepThreads + threadIdx.x;
    int64_t cnt = 0;
    int4 box = make_int4(0, 0, 0, 0);
    if (g < n) {
        float c[3] = {center[g * 3], center[g * 3 + 1], center[g * 3 + 2]};
        cnt = tile_box(s, c, radius[g], &box);
        if (cnt <= 0) {
            atomicOr(&status->flags, GSV_FLAG_EMPTY_BOX);
            cnt = 0;
            box.w = 0;
        }
        boxes[g] = box;
    }
    const PairScan sc = scan_counts(cnt, n, bid, offsets, status);
    if (cs_mat != nullptr) count_rows(s, box, sc, bid, row_len, cs_mat, ntiles);  // block-uniform
}

// count_rows from the tile boxes of an earlier launch (where not cs_fused).
__global__ void __launch_bounds__(kPrepThreads) k_count_rows(const int4* __restrict__ boxes, int64_t n, DevShape s,
                                                             uint16_t* __restrict__ cs_mat, int32_t row_len, int32_t ntiles) {
    const int64_t bid = blockIdx.x, g = bid * kPrepThreads + threadIdx.x;
    const int4 box = g < n ? boxes[g] : make_int4(0, 0, 0, 0);
    int64_t incl = box.w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((threadIdx.x & 31) >= o) incl += y;
    }
    count_rows(s, box, PairScan{incl - box.w, __shfl_sync(0xffffffffu, incl, 31)}, bid, row_len, cs_mat, ntiles);
}

// Emission of the pairs in Gaussian-major (d,h,w) raster order
// (tile_voxelizer.py:126-145), plus the two fills the sort and the range
// pass need: the tile ranges cleared to (0,0) and the sort padding past the
// pair total (keys = ntiles, after every real tile) -- one launch.
// A warp owns 32 consecutive Gaussians and writes their pairs as one
// contiguous range: lane l takes pairs base + l, base + 32 + l, ... and finds
// its Gaussian by a shuffle binary search over the warp's first indices.
// Bound by the shuffles and the tile arithmetic: indices are relative to the
// warp's first pair (one shuffle a step instead of two) and the divisions are
// small_div's where every pair index is below its limit.  2M Gaussians with
// 23 M pairs: 72 us, against 120 with 64-bit indices and integer division.
constexpr int64_t kSmallDivMax = 4000000;
__global__ void __launch_bounds__(128) k_emit(const int4* __restrict__ boxes,
                                              const int64_t* __restrict__ offsets, int64_t n,
                                              DevShape s, int64_t cap, int32_t* __restrict__ keys,
                                              int32_t* __restrict__ vals, int2* __restrict__ ranges,
                                              int64_t ntiles, Status* status) {
    constexpr unsigned kAll = 0xffffffffu;
    const int64_t g = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    const int lane = threadIdx.x & 31;
    const int64_t total = offsets[n];
    if (g == 0) {
        if (total > cap) atomicOr(&status->flags, GSV_FLAG_CAPACITY_OVERFLOW);
        if (total > int64_t(INT32_MAX)) atomicOr(&status->flags, GSV_FLAG_TOO_MANY_PAIRS);
    }
    for (int64_t t = g; t < ntiles; t += stride) ranges[t] = make_int2(0, 0);
    for (int64_t i = total + g; i < cap; i += stride) {
        keys[i] = int32_t(ntiles);
        vals[i] = 0;
    }
    const int64_t g0 = g - lane;  // first Gaussian of this warp (warp-uniform)
    if (g0 >= n) return;
    const int m = int(min(int64_t(32), n - g0));
    const int64_t start = offsets[g0];
    // The warp's pairs from `start` on: 32 tile boxes can hold more than 2^31 pairs, but those past the
    // capacity (itself below 2^31) are not written.
    const unsigned end = unsigned(max(min(offsets[g0 + m], cap) - start, int64_t(0)));
    int4 b = make_int4(0, 0, 0, 0);
    unsigned o = UINT32_MAX;  // lanes past the last Gaussian never match
    if (lane < m) {
        b = boxes[g];
        o = unsigned(min(offsets[g] - start, int64_t(UINT32_MAX)));
    }
    const bool small = ntiles <= kSmallDivMax;
    const float r1 = box_rcp(b.z), r2 = box_rcp(b.z >> 16);
    for (unsigned base = 0; base < end; base += 32) {
        const unsigned p = base + lane;
        int j = 0;  // largest j with o_j <= p
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const unsigned oj = __shfl_sync(kAll, o, j + step);
            if (oj <= p) j += step;
        }
        const int32_t c = int32_t(p - __shfl_sync(kAll, o, j));
        const int bx = __shfl_sync(kAll, b.x, j), by = __shfl_sync(kAll, b.y, j), bz = __shfl_sync(kAll, b.z, j);
        const float q1 = __shfl_sync(kAll, r1, j), q2 = __shfl_sync(kAll, r2, j);
        if (p >= end) continue;
        int32_t tile;
        if (small) {
            tile = box_tile_small(s, bx, by, bz, q1, q2, c);
        } else {
            const int32_t t0 = bx & 0xffff, t1 = (bx >> 16) & 0xffff, t2 = by & 0xffff;
            const int32_t n1 = bz & 0xffff, n2 = (bz >> 16) & 0xffff;
            const int32_t k = c % n2, r = c / n2;
            tile = ((t0 + r / n1) * s.nt[1] + (t1 + r % n1)) * s.nt[2] + (t2 + k);
        }
        keys[start + p] = tile;
        vals[start + p] = int32_t(g0 + j);
    }
}

// Tile ranges from the sorted keys; empty tiles stay (0,0).  Bound by the
// keys' bytes: four to a load, the neighbours' from the lanes beside (a key
// and both neighbours per thread: 98 us for 23 M keys, 93 MB; now 30).
__global__ void __launch_bounds__(256) k_ranges(const int32_t* __restrict__ keys,
                                                const int64_t* __restrict__ offsets, int64_t n, int64_t cap,
                                                int64_t ntiles, int2* __restrict__ ranges) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t total = min(offsets[n], cap);
    const int64_t step = int64_t(gridDim.x) * blockDim.x * 4;
    // the warp's first key; warps stay whole for the shuffles
    for (int64_t w = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x - lane) * 4; w < total; w += step) {
        const int64_t i = w + lane * 4;
        int32_t k[6];  // the key before, the four, the one after; -1 outside
        if (i + 3 < total) {
            const int4 q = *reinterpret_cast<const int4*>(keys + i);
            k[1] = q.x, k[2] = q.y, k[3] = q.z, k[4] = q.w;
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) k[1 + u] = i + u < total ? keys[i + u] : -1;
        }
        k[0] = __shfl_up_sync(kAll, k[4], 1);
        k[5] = __shfl_down_sync(kAll, k[1], 1);
        if (lane == 0) k[0] = i > 0 ? keys[i - 1] : -1;
        if (lane == 31) k[5] = i + 4 < total ? keys[i + 4] : -1;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int32_t key = k[1 + u];
            if (key < 0 || key >= ntiles) continue;
            if (k[u] != key) ranges[key].x = int32_t(i + u);
            if (k[2 + u] != key) ranges[key].y = int32_t(i + u + 1);
        }
    }
}

// Column pass of the counting sort: one block per kCsCols tiles (dynamic
// block id from Status::pad[2]), 32 row groups per column.  cs_pos[r][t] =
// start(t) + the pairs of rows < r in tile t, where start(t) = the pairs in
// tiles < t, from a single-pass look-back over the blocks' tile totals.
// Writes every tile's range, (0,0) for an empty tile, clamped to `cap` (so a
// truncated list never reaches past the pair buffer).
__global__ void __launch_bounds__(kCsCols * kCsRowGroups) k_colscan(const uint16_t* __restrict__ mat,
                                                                    int32_t* __restrict__ pos, int64_t rows,
                                                                    int32_t ntiles, int64_t cap,
                                                                    int2* __restrict__ ranges, Status* status,
                                                                    unsigned long long* lb) {
    __shared__ int bid_s;
    __shared__ int64_t part[kCsRowGroups][kCsCols];  // a row group's sum, then its exclusive prefix
    __shared__ int64_t start_s[kCsCols], tot_s[kCsCols];
    if (threadIdx.x == 0) bid_s = atomicAdd(&status->pad[2], 1);
    __syncthreads();
    const int64_t bid = bid_s;
    const int c = threadIdx.x % kCsCols, rg = threadIdx.x / kCsCols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t = bid * kCsCols + c;
    const bool col_ok = t < ntiles;
    const int64_t per = (rows + kCsRowGroups - 1) / kCsRowGroups;
    const int64_t r0 = min(rows, rg * per), r1 = min(rows, r0 + per);
    int64_t sum = 0;
    if (col_ok) {
#pragma unroll 8
        for (int64_t r = r0; r < r1; ++r) sum += mat[r * cs_mstride(ntiles) + t];
    }
    part[rg][c] = sum;
    __syncthreads();
    if (warp == 0) {  // lane = column of this block
        int64_t run = 0;
        for (int k = 0; k < kCsRowGroups; ++k) {
            const int64_t v = part[k][lane];
            part[k][lane] = run;
            run += v;
        }
        tot_s[lane] = run;
        int64_t incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const int64_t block_tot = __shfl_sync(0xffffffffu, incl, 31);
        const int64_t base = lookback(lb, bid, block_tot, status, lane);
        start_s[lane] = base + incl - run;
    }
    __syncthreads();
    if (!col_ok) return;
    int64_t at_r = start_s[c] + part[rg][c];
    for (int64_t r = r0; r < r1; ++r) {
        pos[r * ntiles + t] = int32_t(min(at_r, cap));
        at_r += mat[r * cs_mstride(ntiles) + t];
    }
    if (rg == 0) {
        const int64_t st = start_s[c], tt = tot_s[c];
        ranges[t] = tt > 0 ? make_int2(int32_t(min(st, cap)), int32_t(min(st + tt, cap))) : make_int2(0, 0);
    }
}

// Placement pass of the counting sort: one block per row, kCsSub Gaussians of it
// at a time.  A pair's place is its tile's current position plus the number of
// earlier Gaussians of the kCsSub in that tile.  Every tile has a word with a
// bit per Gaussian: all pairs set their bits (in any order), then read the bits
// below their own, so no pair waits for another; a sweep over the tiles then
// advances the positions.  (A warp that walked the Gaussians in id order
// instead took 19 us for 500 Gaussians and 27 us for 50,000 on 3072 tiles.)  A
// group of lanes takes a Gaussian, each lane some of its tiles; how many lanes
// follows from the row's mean (kCsNarrow8, kCsNarrow16).
// Positions at or past `cap` are dropped (the overflow flag says so).  Block 0
// also latches the capacity flags and clears k_colscan's ticket counter and
// look-back words (k_colscan has finished: stream order).
__global__ void __launch_bounds__(1024) k_scatter(const int32_t* __restrict__ pos_in, const int4* __restrict__ boxes,
                                                  const int64_t* __restrict__ offsets, int64_t n, int row_len,
                                                  int32_t ntiles, DevShape s, int64_t cap, int32_t* __restrict__ pair_ids,
                                                  Status* status, unsigned long long* lb, int64_t lb_words) {
    static_assert(kCsSub == 64, "a tile's word has 64 bits");
    __shared__ int4 box_s[kPrepThreads];
    __shared__ float2 rcp_s[kPrepThreads];
    extern __shared__ uint2 cs_bits[];  // [ntiles], then the tiles' positions
    int32_t* at_t = reinterpret_cast<int32_t*>(cs_bits + ntiles);
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            const int64_t total = offsets[n];
            if (total > cap) atomicOr(&status->flags, GSV_FLAG_CAPACITY_OVERFLOW);
            if (total > int64_t(INT32_MAX)) atomicOr(&status->flags, GSV_FLAG_TOO_MANY_PAIRS);
            status->pad[2] = 0;
        }
        for (int64_t i = threadIdx.x; i < lb_words; i += blockDim.x) lb[i] = 0ull;
    }
    const int64_t row = blockIdx.x, g0 = row * row_len;
    if (g0 >= n) return;  // block-uniform
    const int m = int(min(int64_t(row_len), n - g0));
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int4 b = boxes[g0 + i];
        box_s[i] = b;
        rcp_s[i] = make_float2(box_rcp(b.z), box_rcp(b.z >> 16));
    }
    for (int t0 = threadIdx.x; t0 < ntiles; t0 += 4 * blockDim.x) {  // four loads in flight
        int32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = t0 + i * blockDim.x;
            v[i] = t < ntiles ? __ldg(pos_in + row * ntiles + t) : 0;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = t0 + i * blockDim.x;
            if (t < ntiles) {
                cs_bits[t] = make_uint2(0u, 0u);
                at_t[t] = v[i];
            }
        }
    }
    // lanes per Gaussian
    const int64_t pairs = offsets[g0 + m] - offsets[g0];
    const int log_g = pairs <= kCsNarrow8 * m ? 3 : pairs <= kCsNarrow16 * m ? 4 : 5;
    const int slot = threadIdx.x >> log_g, slots = blockDim.x >> log_g, in = threadIdx.x & ((1 << log_g) - 1);
    __syncthreads();
    for (int h = 0; h < m; h += kCsSub) {  // block-uniform
        const int mh = min(kCsSub, m - h);
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            for (int j = slot; j < mh; j += slots) {
                const int4 b = box_s[h + j];
                const uint32_t bit = 1u << (j & 31);
                const float2 rcp = rcp_s[h + j];
                for (int c = in; c < b.w; c += 1 << log_g) {
                    const int32_t t = box_tile_small(s, b.x, b.y, b.z, rcp.x, rcp.y, c);
                    if (pass == 0) {
                        atomicOr(j < 32 ? &cs_bits[t].x : &cs_bits[t].y, bit);
                    } else {
                        const uint2 w = cs_bits[t];
                        const int before = j < 32 ? __popc(w.x & (bit - 1u)) : __popc(w.x) + __popc(w.y & (bit - 1u));
                        const int64_t p = int64_t(at_t[t]) + before;
                        if (p < cap) pair_ids[p] = int32_t(g0 + h + j);
                    }
                }
            }
            __syncthreads();
        }
        if (h + kCsSub >= m) break;  // the last ones
        for (int t = threadIdx.x; t < ntiles; t += blockDim.x) {
            const uint2 w = cs_bits[t];
            if (w.x | w.y) {
                at_t[t] = int32_t(min(int64_t(at_t[t]) + __popc(w.x) + __popc(w.y), cap));
                cs_bits[t] = make_uint2(0u, 0u);
            }
        }
        __syncthreads();
    }
}

int grid_for(int64_t items, int block) {
    int64_t g = (items + block - 1) / block;
    if (g < 1) g = 1;
    if (g > (int64_t(1) << 30)) g = int64_t(1) << 30;
    return int(g);
}

// Flags and pair total of the last count, in one copy; synchronises the stream.
int read_status(const GaussLayout& L, const void* ws, int64_t* total, int32_t* flags, cudaStream_t st) {
    Status s{};
    GSV_CUDA_TRY(cudaMemcpyAsync(&s, at<Status>(ws, L.status), sizeof(Status), cudaMemcpyDeviceToHost, st));
    GSV_CUDA_TRY(cudaStreamSynchronize(st));
    if (total) *total = s.total;
    if (flags) *flags = s.flags;
    return GSV_OK;
}

// Dynamic shared memory of the counting kernels' row counters (at most 36 KB, the default allows it)
// and of k_scatter's words and positions.
int cs_count_smem_bytes(int64_t n, int64_t ntiles) {
    return int(kPrepThreads / cs_row_len(n, ntiles) * ((ntiles + 1) / 2) * int64_t(sizeof(uint32_t)));
}
int cs_scatter_smem_bytes(int64_t ntiles) { return int(ntiles * int64_t(sizeof(uint2) + sizeof(int32_t))); }
constexpr int kScatterStatic = kPrepThreads * int(sizeof(int4) + sizeof(float2));
static_assert((kCsMaxTiles + 1) / 2 * 4 <= 40 * 1024 && kPrepThreads / kCsSub * (kCsShortTiles + 1) / 2 * 4 <= 40 * 1024,
              "the row counters leave no room for the static words");
static_assert(kCsMaxTiles * (sizeof(uint2) + sizeof(int32_t)) + kScatterStatic <= 227 * 1024,
              "k_scatter's words, positions and boxes exceed an SM's shared memory");

// Shared tail of both binning flavours.  Counting sort (k_colscan,
// k_scatter) where it applies (the counting kernels wrote the per-row tile
// counts) and `mode` allows it; otherwise emit, radix sort, ranges.
int bin_common(const ShapeInfo& si, int64_t n, void* ws_gauss, void* ws_pairs, size_t ws_pairs_bytes,
               int64_t cap, int32_t* vals_out_override, int mode, cudaStream_t st) {
    if (cap < 0 || cap > int64_t(INT32_MAX)) return GSV_ERR_INVALID_ARGUMENT;
    if (mode != GSV_BIN_AUTO && mode != GSV_BIN_RADIX && mode != GSV_BIN_COUNTING) return GSV_ERR_INVALID_ARGUMENT;
    const GaussLayout G = gauss_layout(n, si);
    const PairLayout P = pair_layout(cap, si, 0);
    if (ws_pairs_bytes < P.total || !ws_pairs) return GSV_ERR_INVALID_ARGUMENT;
    DevShape s = dev_shape(si);
    Status* status = at<Status>(ws_gauss, G.status);
    const int64_t* offsets = at<int64_t>(ws_gauss, G.offsets);
    int32_t* keys_in = at<int32_t>(ws_pairs, P.keys_in);
    int32_t* vals_in = at<int32_t>(ws_pairs, P.vals_in);
    int32_t* keys_out = at<int32_t>(ws_pairs, P.keys_out);
    int32_t* vals_out = vals_out_override ? vals_out_override : at<int32_t>(ws_pairs, P.vals_out);
    int2* ranges = at<int2>(ws_gauss, G.ranges);
    if (mode == GSV_BIN_COUNTING && !G.cs) return GSV_ERR_INVALID_ARGUMENT;
    if (cap == 0) {
        GSV_CUDA_TRY(cudaMemsetAsync(ranges, 0, size_t(si.ntiles) * sizeof(int2), st));
        return GSV_OK;
    }
    if (G.cs && (mode == GSV_BIN_COUNTING || (mode == GSV_BIN_AUTO && cs_pays(n, si.ntiles, cap)))) {
        unsigned long long* lb_cs = reinterpret_cast<unsigned long long*>(status + 1) + prep_blocks(n);
        const int64_t rows = cs_rows(n, si.ntiles), row_len = cs_row_len(n, si.ntiles);
        const int32_t T = int32_t(si.ntiles);
        if (!cs_fused(n, T)) {
            k_count_rows<<<unsigned(prep_blocks(n)), kPrepThreads, cs_count_smem_bytes(n, T), st>>>(
                at<int4>(ws_gauss, G.box), n, s, at<uint16_t>(ws_gauss, G.cs_mat), int32_t(row_len), T);
            GSV_LAUNCH_CHECK();
        }
        k_colscan<<<unsigned(cs_col_blocks(T)), kCsCols * kCsRowGroups, 0, st>>>(
            at<uint16_t>(ws_gauss, G.cs_mat), at<int32_t>(ws_gauss, G.cs_pos), rows, T, cap, ranges, status, lb_cs);
        GSV_LAUNCH_CHECK();
        // Short rows of many blocks take 512 threads, with which more blocks fit on an SM; more threads shorten the
        // sweeps over many tiles, of which one block fits from 9088 on.  Binning with 512 and 1024, us: 3072 tiles,
        // 50,000 Gaussians 22 and 25, 200,000 42 and 48; 4096 tiles 26 and 26, 45 and 51; 8832 tiles, 20,000 36 and
        // 34, 100,000 49 and 47; 9384 tiles 37 and 33, 61 and 52; 17576 tiles 51 and 44, 103 and 90.  Between 4096
        // and 9088 either may be the faster: 5760 tiles, 200,000 75 and 81; 6336 tiles, 100,000 44 and 42.
        const int smem = cs_scatter_smem_bytes(T);
        const int threads = T <= 4096 ? 512 : 1024;
        // The limit belongs to the function, for every thread and captured launch: always the largest
        // grid's, so that no call lowers it under another's launch.
        if (smem + kScatterStatic > 48 * 1024)
            GSV_CUDA_TRY(cudaFuncSetAttribute(k_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              cs_scatter_smem_bytes(kCsMaxTiles)));
        k_scatter<<<unsigned(rows), threads, smem, st>>>(at<int32_t>(ws_gauss, G.cs_pos), at<int4>(ws_gauss, G.box),
                                                         offsets, n, int(row_len), T, s, cap, vals_out, status, lb_cs,
                                                         cs_col_blocks(T));
        GSV_LAUNCH_CHECK();
        return GSV_OK;
    }
    // enough CTAs for the emission (one thread per Gaussian) and for the fills
    const int fill_grid = grid_for(cap > si.ntiles ? cap : si.ntiles, 128);
    const int emit_grid = grid_for(n, 128);
    const int grid = emit_grid > (fill_grid < 1184 ? fill_grid : 1184) ? emit_grid : (fill_grid < 1184 ? fill_grid : 1184);
    k_emit<<<grid, 128, 0, st>>>(at<int4>(ws_gauss, G.box), offsets, n, s, cap, keys_in, vals_in, ranges,
                                 si.ntiles, status);
    GSV_LAUNCH_CHECK();
    size_t sort_bytes = P.sort_tmp_bytes;
    GSV_CUDA_TRY(cub::DeviceRadixSort::SortPairs(at<void>(ws_pairs, P.sort_tmp), sort_bytes, keys_in,
                                                 keys_out, vals_in, vals_out, int(cap), 0,
                                                 sort_end_bit(si.ntiles), st));
    const int range_grid = grid_for((cap + 3) / 4, 256);
    k_ranges<<<range_grid < 1184 ? range_grid : 1184, 256, 0, st>>>(keys_out, offsets, n, cap, si.ntiles, ranges);
    GSV_LAUNCH_CHECK();
    return GSV_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// C entry points
// ---------------------------------------------------------------------------

void gsv_detail_set_error(cudaError_t e, const char* what, const char* file, int line) {
    snprintf(g_last_error, sizeof(g_last_error), "%s (%s) at %s:%d: %s", cudaGetErrorName(e), what,
             file, line, cudaGetErrorString(e));
}

extern "C" {

const char* gsv_last_error(void) { return g_last_error; }

int gsv_abi_version(void) { return GSV_ABI_VERSION; }

const char* gsv_status_string(int status) {
    switch (status) {
        case GSV_OK: return "ok";
        case GSV_ERR_INVALID_ARGUMENT: return "invalid argument";
        case GSV_ERR_CAPACITY: return "pair capacity exceeded";
        case GSV_ERR_CUDA: return "CUDA error";
        case GSV_ERR_EMPTY_BOX: return "empty tile box (negative radius)";
        case GSV_ERR_TOO_MANY_PAIRS: return "more than INT32_MAX tile pairs";
        default: return "unknown status";
    }
}

int64_t gsv_num_tiles(gsv_shape shape) {
    ShapeInfo si = shape_info(shape);
    return si.ok ? si.ntiles : -1;
}

size_t gsv_gauss_workspace_bytes(int64_t n, gsv_shape shape) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || n < 0 || n >= int64_t(INT32_MAX)) return 0;
    return gauss_layout(n, si).total;
}

size_t gsv_pair_workspace_bytes(int64_t capacity, gsv_shape shape, int flags) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || capacity < 0 || capacity > int64_t(INT32_MAX)) return 0;
    return pair_layout(capacity, si, flags).total;
}

static int prepare_impl(const gsv_params* p, int64_t density_stride, const int32_t* live, gsv_shape shape,
                        void* ws_gauss, size_t ws_gauss_bytes, int64_t* total_pairs_host, int32_t* flags_host,
                        void* stream) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || !p || p->n < 0 || p->n >= int64_t(INT32_MAX) || !ws_gauss) return GSV_ERR_INVALID_ARGUMENT;
    const int64_t n = p->n;
    if (n > 0 && (!p->positions || !p->scales || !p->rotations || !p->density_r || !p->density_i))
        return GSV_ERR_INVALID_ARGUMENT;
    const GaussLayout L = gauss_layout(n, si);
    if (ws_gauss_bytes < L.total) return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Status* status = at<Status>(ws_gauss, L.status);
    // status flags, the block counters and the scans' look-back words
    GSV_CUDA_TRY(cudaMemsetAsync(status, 0, status_bytes(n, si.ntiles), st));
    const bool count = L.cs && cs_fused(n, si.ntiles);
    const int smem = count ? cs_count_smem_bytes(n, si.ntiles) : 0;
    k_prepare<<<unsigned(prep_blocks(n)), kPrepThreads, smem, st>>>(
        p->positions, p->scales, p->rotations, p->density_r, p->density_i, density_stride, n, live, dev_shape(si),
        at<Rec>(ws_gauss, L.rec), at<float4>(ws_gauss, L.ext), at<int4>(ws_gauss, L.box),
        at<int64_t>(ws_gauss, L.offsets), status, count ? at<uint16_t>(ws_gauss, L.cs_mat) : nullptr,
        int32_t(cs_row_len(n, si.ntiles)), int32_t(si.ntiles), at<float>(ws_gauss, L.accum));
    GSV_LAUNCH_CHECK();
    if (total_pairs_host) return read_status(L, ws_gauss, total_pairs_host, flags_host, st);
    return GSV_OK;
}

int gsv_prepare(const gsv_params* p, gsv_shape shape, void* ws_gauss, size_t ws_gauss_bytes,
                int64_t* total_pairs_host, void* stream) {
    return prepare_impl(p, 1, nullptr, shape, ws_gauss, ws_gauss_bytes, total_pairs_host, nullptr, stream);
}

int gsv_prepare_live(const gsv_params* p, const int32_t* live, gsv_shape shape, void* ws_gauss,
                     size_t ws_gauss_bytes, int64_t* total_pairs_host, void* stream) {
    if (!live) return GSV_ERR_INVALID_ARGUMENT;
    return prepare_impl(p, 1, live, shape, ws_gauss, ws_gauss_bytes, total_pairs_host, nullptr, stream);
}

int gsv_prepare_strided(const gsv_params* p, int64_t density_stride, const int32_t* live, gsv_shape shape,
                        void* ws_gauss, size_t ws_gauss_bytes, int64_t* total_pairs_host, int32_t* flags_host,
                        void* stream) {
    if (density_stride < 1) return GSV_ERR_INVALID_ARGUMENT;
    return prepare_impl(p, density_stride, live, shape, ws_gauss, ws_gauss_bytes, total_pairs_host, flags_host, stream);
}

int gsv_bin_ex(gsv_shape shape, int64_t n, void* ws_gauss, void* ws_pairs, size_t ws_pairs_bytes,
               int64_t capacity, int mode, void* stream) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || n < 0 || !ws_gauss) return GSV_ERR_INVALID_ARGUMENT;
    return bin_common(si, n, ws_gauss, ws_pairs, ws_pairs_bytes, capacity, nullptr, mode,
                      static_cast<cudaStream_t>(stream));
}

int gsv_bin(gsv_shape shape, int64_t n, void* ws_gauss, void* ws_pairs, size_t ws_pairs_bytes,
            int64_t capacity, void* stream) {
    return gsv_bin_ex(shape, n, ws_gauss, ws_pairs, ws_pairs_bytes, capacity, GSV_BIN_AUTO, stream);
}

int gsv_bin_views(gsv_shape shape, int64_t n, void* ws_gauss, void* ws_pairs, int64_t capacity,
                  int32_t** tile_ranges, int32_t** pair_ids) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || n < 0 || !ws_gauss || !ws_pairs) return GSV_ERR_INVALID_ARGUMENT;
    if (tile_ranges) *tile_ranges = at<int32_t>(ws_gauss, gauss_layout(n, si).ranges);
    if (pair_ids) *pair_ids = at<int32_t>(ws_pairs, pair_layout(capacity, si, 0).vals_out);
    return GSV_OK;
}

int gsv_status_views(gsv_shape shape, int64_t n, void* ws_gauss, int32_t** flags, int64_t** total_pairs) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || n < 0 || !ws_gauss) return GSV_ERR_INVALID_ARGUMENT;
    const GaussLayout L = gauss_layout(n, si);
    if (flags) *flags = &at<Status>(ws_gauss, L.status)->flags;
    if (total_pairs) *total_pairs = &at<Status>(ws_gauss, L.status)->total;
    return GSV_OK;
}

int gsv_read_status(gsv_shape shape, int64_t n, const void* ws_gauss, int64_t* total_pairs,
                    int32_t* flags, void* stream) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || n < 0 || !ws_gauss) return GSV_ERR_INVALID_ARGUMENT;
    const GaussLayout L = gauss_layout(n, si);
    return read_status(L, ws_gauss, total_pairs, flags, static_cast<cudaStream_t>(stream));
}

int gsv_build_tile_pairs_count(const float* center_vox, const float* radius_vox, int64_t n,
                               gsv_shape shape, void* ws_gauss, size_t ws_gauss_bytes,
                               int64_t* total_pairs_host, void* stream) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || n < 0 || n >= int64_t(INT32_MAX) || !ws_gauss) return GSV_ERR_INVALID_ARGUMENT;
    if (n > 0 && (!center_vox || !radius_vox)) return GSV_ERR_INVALID_ARGUMENT;
    const GaussLayout L = gauss_layout(n, si);
    if (ws_gauss_bytes < L.total) return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Status* status = at<Status>(ws_gauss, L.status);
    GSV_CUDA_TRY(cudaMemsetAsync(status, 0, status_bytes(n, si.ntiles), st));
    const bool count = L.cs && cs_fused(n, si.ntiles);
    k_count_compat<<<unsigned(prep_blocks(n)), kPrepThreads, count ? cs_count_smem_bytes(n, si.ntiles) : 0, st>>>(
        center_vox, radius_vox, n, dev_shape(si), at<int4>(ws_gauss, L.box), at<int64_t>(ws_gauss, L.offsets), status,
        count ? at<uint16_t>(ws_gauss, L.cs_mat) : nullptr, int32_t(cs_row_len(n, si.ntiles)), int32_t(si.ntiles));
    GSV_LAUNCH_CHECK();
    if (total_pairs_host) return read_status(L, ws_gauss, total_pairs_host, nullptr, st);
    return GSV_OK;
}

int gsv_build_tile_pairs_fill(gsv_shape shape, int64_t n, void* ws_gauss, void* ws_pairs,
                              size_t ws_pairs_bytes, int64_t capacity, int32_t* tile_ranges,
                              int32_t* pair_ids, void* stream) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || n < 0 || !ws_gauss || !tile_ranges || (capacity > 0 && !pair_ids))
        return GSV_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc = bin_common(si, n, ws_gauss, ws_pairs, ws_pairs_bytes, capacity, pair_ids, GSV_BIN_AUTO, st);
    if (rc != GSV_OK) return rc;
    const GaussLayout L = gauss_layout(n, si);
    GSV_CUDA_TRY(cudaMemcpyAsync(tile_ranges, at<int2>(ws_gauss, L.ranges), size_t(si.ntiles) * sizeof(int2),
                                 cudaMemcpyDeviceToDevice, st));
    return GSV_OK;
}

}  // extern "C"

// Internal accessors for the render translation unit.
namespace gsv {
int layout_for(gsv_shape shape, int64_t n, int64_t cap, int flags, GaussLayout* G, PairLayout* P,
               int64_t* ntiles) {
    ShapeInfo si = shape_info(shape);
    if (!si.ok || n < 0) return GSV_ERR_INVALID_ARGUMENT;
    if (G) *G = gauss_layout(n, si);
    if (P) *P = pair_layout(cap, si, flags);
    if (ntiles) *ntiles = si.ntiles;
    return GSV_OK;
}
}  // namespace gsv
