// Exact 2-NN of u8 SIFT descriptors on sm_100a: one persistent, warp-
// specialised kernel computes q.b on the 5th-generation tensor cores
// (tcgen05.mma kind::i8, u8 x u8 -> s32, accumulators in TMEM, operands
// staged by TMA) and reduces every accumulator tile to a per-query top-2 in
// the epilogue, so the queries x base distance matrix never reaches HBM.
//
// Replaces the reference's GEMM + scan pairs:
//   cublasHgemm / cublasGemmEx   src/knn_brute.cu:244, :592   (dist = -2 q.r to HBM)
//   find_matches / min_dist_f    src/knn_brute.cu:340-448, :726-796 (scan of dist)
//   sqrEuclidianDist             src/knn_brute.cu:671-691     (full squared L2)
//
// Ranking key. For query q and base row b the kernel ranks by
//     key(b) = norm(b) - 2 q.b        (norm(b) = |b|^2 for kMetricL2, 0 for kMetricDot)
// which orders candidates exactly like |q - b|^2 = |q|^2 + key (resp. -2 q.b).
// All values are exact integers: |key| <= 2 * 128 * 255^2 < 2^25.
// Ties are broken by the lower base index (lexicographic (key, index) order),
// which is the order of the reference's host_brute (src/knn_brute.cu:816-831).
//
// Work decomposition. A CTA holds kQT = 4 query tiles (512 queries) in shared
// memory and streams base tiles of kBN = 128 rows; a unit = (query group,
// base tile). Units are split evenly over a persistent grid of one CTA per SM.
//
// Warp roles (kThreads = 576):
//   warp 0       TMA producer: the query tiles of the current group and a
//                kStages ring of base tiles
//   warp 1       TMEM allocator + single-thread MMA issuer: per base tile one
//                128 x 128 x 128 product per query tile into that tile's
//                TMEM slot (4 slots x 128 columns)
//   warps 2..17  epilogue: warp w owns query tile (w - 2) / 4 and TMEM lane
//                quarter w % 4, i.e. 32 query rows, one thread per row
//
// Epilogue pruning. Per 8-row subgroup of base rows a thread takes the largest
// dot product m of its query row; with n_min the smallest norm of the subgroup
// (precomputed), n_min - 2 m is a lower bound of every key in it. A group of
// 32 rows (four subgroups, one vote) whose four bounds all exceed the thread's
// threshold is skipped (~0.8 instruction per element); otherwise only the
// passing subgroups form exact keys. The threshold is the thread's own
// second-best key and an upper bound of the final second-best key that the
// CTAs splitting the same query group share through global memory (atomicMin).
#include <cfloat>
#include <climits>
#include <algorithm>
#include <cuda_fp16.h>
#include "exact2nn.cuh"
#include "launch.cuh"
#include "ptx.cuh"
#include "epilogue.cuh"

namespace sift {

namespace {

constexpr int kQTileBytes = kBM * kDim;           // 16 KB: one query tile (u8)
constexpr int kBTileBytes = kBN * kDim;           // 16 KB: one base tile (u8)
constexpr int kRecBytes = kRecInts * 4;           // 640 B: norms record of one base tile

struct __align__(8) SmemCtl {
    uint64_t full[kStages];    // base tile + norms record landed (TMA)
    uint64_t empty[kStages];   // MMAs reading the base tile done (tcgen05.commit)
    uint64_t nempty[kStages];  // all epilogue warps done with the norms record
    uint64_t qfull, qempty;
    uint64_t tfull[kQT], tempty[kQT];
    uint64_t drain;
    uint32_t tmem_base;
    int abort_flag;
    int no_abort;
};

constexpr size_t kSmemBytes =
    1024 + kQT * kQTileBytes + kStages * kBTileBytes + kStages * kRecBytes + sizeof(SmemCtl);

// 16 consecutive elements of a row.
__device__ __forceinline__ uint4 load16_u8(const uint8_t* x, int row, int sub) {
    return reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * kDim)[sub];
}
__global__ void __launch_bounds__(256) row_norms_kernel(const uint8_t* __restrict__ x, int n, int n_pad,
                                                        int metric, int32_t* __restrict__ norm,
                                                        int32_t* __restrict__ rec,
                                                        int32_t* __restrict__ thresh) {
    launch_next();
    // 32 rows per block, 8 threads per row, 16 elements per thread.
    const int row = blockIdx.x * 32 + (threadIdx.x >> 3);
    const int sub = threadIdx.x & 7;
    uint32_t s = 0;
    if (row < n) {
        const uint4 w = load16_u8(x, row, sub);
        s = __dp4a(w.x, w.x, 0u);
        s = __dp4a(w.y, w.y, s);
        s = __dp4a(w.z, w.z, s);
        s = __dp4a(w.w, w.w, s);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    const int32_t v = row < n ? (metric == kMetricL2 ? static_cast<int32_t>(s) : 0) : kKeyPad;
    __shared__ int32_t nrm[32];
    // Record of base tile (row / kBN): [0, 128) norms, [128, 144) 8-row minima.
    int32_t* r = rec ? rec + static_cast<size_t>(blockIdx.x / 4) * kRecInts : nullptr;
    const int part = blockIdx.x & 3;  // which 32-row quarter of the tile
    if (sub == 0) {
        nrm[threadIdx.x >> 3] = v;
        if (norm) norm[row] = v;
        if (r) r[part * 32 + (threadIdx.x >> 3)] = v;
        if (thresh) thresh[row] = thresh[static_cast<size_t>(n_pad) + row] = INT_MAX;
    }
    __syncthreads();
    if (threadIdx.x < 4 && r) {
        int m = nrm[8 * threadIdx.x];
        #pragma unroll
        for (int i = 1; i < 8; ++i) m = min(m, nrm[8 * threadIdx.x + i]);
        r[128 + part * 4 + threadIdx.x] = m;
    }
}

// Norm folding (the fold variant of the u8 pair kernel). A fifth MMA per tile
// product multiplies a constant query-side row a[32] (u8) with 32 signed
// digits d[32] per base row (s8) so that the accumulator holds
// q.b - c with c = min(ceil(|b|^2 / 2), kFoldMax) and a.d = -c:
//   a = {1, 16, 255 x 30}, c = 255 h + l (0 <= l < 255),
//   d[0] = -(l & 15), d[1] = -(l >> 4), d[2..31] = -h in parts of at most 128.
// The key |b|^2 - 2 q.b = r - 2 acc with the residual r = |b|^2 - 2 c >= -1,
// so every key of a row set is at least -1 - 2 max(acc): one max tree per
// row set bounds its keys exactly up to that 1 (rows whose c was clamped
// only make the bound looser). Records hold the residuals.
//
// fold[] layout: per base tile, per half of 64 rows, 2048 bytes in the
// tensor cores' no-swizzle K-major layout (8-row groups of 256 bytes, two
// 16-byte K chunks of 128 bytes each, 16 bytes per row), so one 2-D TMA box
// of 8 x 256 bytes lands a half tile ready as an MMA operand.
//
// One block per base tile: 8 threads per row, the 4 rows of a thread's
// 32-row parts loaded up front (64 bytes in flight per thread), then per row
// the norm, the folded half-norm c, its digits and the residual. Blocks past the
// base tiles take 128 query rows each: norms and cleared bounds (a launch of
// their own cost 2.5 us of every search).
__global__ void __launch_bounds__(256)
    fold_records_kernel(const uint8_t* __restrict__ x, int n, int n_pad, int metric, int32_t* __restrict__ rec,
                        uint32_t* __restrict__ fold, const uint8_t* __restrict__ q, int q_n, int q_pad,
                        int32_t* __restrict__ qnorm, int32_t* __restrict__ thresh) {
    launch_next();
    const int tiles = n_pad / kBN;
    const bool is_base = static_cast<int>(blockIdx.x) < tiles;
    const int t = is_base ? blockIdx.x : blockIdx.x - tiles;
    const int sub = threadIdx.x & 7;
    const int lrow = threadIdx.x >> 3;
    uint4 w[4];
    #pragma unroll
    for (int part = 0; part < 4; ++part) {
        const int row = t * kBN + part * 32 + lrow;
        w[part] = row < (is_base ? n : q_n) ? load16_u8(is_base ? x : q, row, sub) : make_uint4(0u, 0u, 0u, 0u);
    }
    int32_t* r = rec + static_cast<size_t>(t) * kRecInts;
    #pragma unroll
    for (int part = 0; part < 4; ++part) {
        const int wr = part * 32 + lrow;  // row within the tile
        const bool live = t * kBN + wr < n;
        uint32_t s = __dp4a(w[part].x, w[part].x, 0u);
        s = __dp4a(w[part].y, w[part].y, s);
        s = __dp4a(w[part].z, w[part].z, s);
        s = __dp4a(w[part].w, w[part].w, s);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        if (!is_base) {
            const int row = t * kBN + wr;
            if (sub == 0 && row < q_pad) {
                qnorm[row] = static_cast<int32_t>(s);
                thresh[row] = thresh[static_cast<size_t>(q_pad) + row] = INT_MAX;
            }
            continue;
        }
        const int32_t norm = live ? (metric == kMetricL2 ? static_cast<int32_t>(s) : 0) : kKeyPad;
        const int32_t c = live ? min((norm + 1) >> 1, kFoldMax) : 0;
        const int32_t resid = norm - 2 * c;
        // This thread's 4 digits k = 4 sub .. 4 sub + 3.
        const int l = c % 255, h = c / 255;
        uint32_t word = 0;
        #pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int k = 4 * sub + b;
            const int d = k == 0 ? -(l & 15) : (k == 1 ? -(l >> 4) : -min(128, max(0, h - 128 * (k - 2))));
            word |= (static_cast<uint32_t>(d) & 0xFFu) << (8 * b);
        }
        const size_t off = (static_cast<size_t>(t) * 2 + (wr >> 6)) * kFoldHalfBytes + ((wr & 63) >> 3) * 256 +
                           (sub >> 2) * 128 + (wr & 7) * 16 + 4 * (sub & 3);
        fold[off / 4] = word;
        if (sub == 0) r[wr] = resid;
    }
}

// 16 consecutive elements of a row as floats.
__device__ __forceinline__ void load16_f32(const __half* x, int row, int sub, float (&f)[16]) {
    const uint4* p = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * kDim) + 2 * sub;
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4 v = p[h];
        const __half2* hv = reinterpret_cast<const __half2*>(&v);
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 a = __half22float2(hv[k]);
            f[8 * h + 2 * k] = a.x;
            f[8 * h + 2 * k + 1] = a.y;
        }
    }
}

// Squared norms of general (non-integer) half rows, in FP32, stored as float bit patterns in the int32 slots of the integer path (norm,
// record norms and 8-row minima); padding rows get kFloatKeyPad. thresh is set
// to INT_MAX (the largest ordered key, see float_key).
__global__ void __launch_bounds__(256) row_norms_float_kernel(const __half* __restrict__ x, int n, int n_pad,
                                                              int metric, int32_t* __restrict__ norm,
                                                              int32_t* __restrict__ rec,
                                                              int32_t* __restrict__ thresh) {
    launch_next();
    const int row = blockIdx.x * 32 + (threadIdx.x >> 3);
    const int sub = threadIdx.x & 7;
    float s = 0.0f;
    if (row < n) {
        float f[16];
        load16_f32(x, row, sub, f);
        #pragma unroll
        for (int i = 0; i < 16; ++i) s = fmaf(f[i], f[i], s);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    const float v = row < n ? (metric == kMetricL2 ? s : 0.0f) : kFloatKeyPad;
    __shared__ float nrm[32];
    int32_t* r = rec ? rec + static_cast<size_t>(blockIdx.x / 4) * kRecInts : nullptr;
    const int part = blockIdx.x & 3;
    if (sub == 0) {
        nrm[threadIdx.x >> 3] = v;
        if (norm) norm[row] = __float_as_int(v);
        if (r) r[part * 32 + (threadIdx.x >> 3)] = __float_as_int(v);
        if (thresh) thresh[row] = thresh[static_cast<size_t>(n_pad) + row] = INT_MAX;
    }
    __syncthreads();
    if (threadIdx.x < 4 && r) {
        float m = nrm[8 * threadIdx.x];
        #pragma unroll
        for (int i = 1; i < 8; ++i) m = fminf(m, nrm[8 * threadIdx.x + i]);
        r[128 + part * 4 + threadIdx.x] = __float_as_int(m);
    }
}

// Largest k with key(items[k]) <= v over a non-decreasing key; empty
// problems share the key of the problem after them, so the match is the
// problem that owns v.
template <typename F>
__device__ __forceinline__ int find_item(int n_items, long long v, F key) {
    int lo = 0, hi = n_items - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (key(mid) <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Norms of a batch in one launch, one block per 128 rows with four 16-byte row
// loads in flight per thread. Blocks [0, tiles): the base-tile records of the
// packed epilogue, K[col] = 127 - col - 128 |b|^2 (epilogue.cuh; the record
// belongs to the problem whose record range holds it, rows of its base set past
// n_b get 0). The blocks after them: query norms and cleared bounds. HBM-bound:
// 128 bytes read per row, 4-8 written.
__global__ void __launch_bounds__(256)
    batch_prep_kernel(const uint8_t* __restrict__ base, const WorkItem* __restrict__ items, int n_items,
                      const WorkItem single, int tiles, int32_t* __restrict__ rec, const uint8_t* __restrict__ q, int q_n, int q_pad,
                      int32_t* __restrict__ qnorm, int32_t* __restrict__ thresh) {
    launch_next();
    const int sub = threadIdx.x & 7, lrow = threadIdx.x >> 3;
    const bool is_base = static_cast<int>(blockIdx.x) < tiles;
    const uint8_t* x = q;
    int first = (blockIdx.x - tiles) * kBN, n = q_n;  // rows [first, first + 128) of x, valid below n
    if (is_base) {
        const int T = blockIdx.x;
        // 32 probes per step instead of one: the largest p with rec_off <= T.
        int lo = 0, hi = n_items;  // rec_off[lo] <= T < rec_off[hi]; no list: the single problem
        while (items && hi - lo > 1) {
            const int step = (hi - lo + 31) / 32;
            const int at = lo + (threadIdx.x & 31) * step;
            const bool le = at < hi && items[at].rec_off <= T;
            const int k = __popc(__ballot_sync(0xffffffffu, le)) - 1;  // rec_off is non-decreasing
            hi = min(hi, lo + (k + 1) * step);
            lo += k * step;
        }
        const WorkItem it = items ? items[lo] : single;
        x = base + static_cast<size_t>(it.b_off) * kDim;
        first = (T - it.rec_off) * kBN;
        n = it.n_b;
    }
    uint4 w[4];
    #pragma unroll
    for (int part = 0; part < 4; ++part) {
        const int row = first + part * 32 + lrow;
        w[part] = row < n ? load16_u8(x, row, sub) : make_uint4(0u, 0u, 0u, 0u);
    }
    #pragma unroll
    for (int part = 0; part < 4; ++part) {
        uint32_t s = __dp4a(w[part].x, w[part].x, 0u);
        s = __dp4a(w[part].y, w[part].y, s);
        s = __dp4a(w[part].z, w[part].z, s);
        s = __dp4a(w[part].w, w[part].w, s);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        const int col = part * 32 + lrow, row = first + col;
        if (sub != 0) continue;
        if (is_base) {
            rec[static_cast<size_t>(blockIdx.x) * kRecInts + col] =
                row < n ? 127 - col - 128 * static_cast<int32_t>(s) : 0;
        } else if (row < q_pad) {
            qnorm[row] = static_cast<int32_t>(s);
            thresh[row] = INT_MAX;
        }
    }
}

__global__ void __launch_bounds__(kThreads, 1)
    exact2nn_u8_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap bmap,
                       const int32_t* __restrict__ brec, const ExactPlan plan, int4* __restrict__ partial,
                       int32_t* __restrict__ thresh, int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment for the 128-byte swizzle atoms.
    const uint32_t raw_u32 = ptx::smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (raw_u32 & 1023u)) & 1023u);
    uint8_t* q_smem = smem;
    uint8_t* b_smem = smem + kQT * kQTileBytes;
    int32_t* r_smem = reinterpret_cast<int32_t*>(b_smem + kStages * kBTileBytes);
    SmemCtl* ctl = reinterpret_cast<SmemCtl*>(r_smem + kStages * kRecInts);
    const uint32_t q_s = ptx::smem_u32(q_smem);
    const uint32_t b_s = ptx::smem_u32(b_smem);
    const uint32_t r_s = ptx::smem_u32(r_smem);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const long long W = plan.units;
    const long long G = plan.grid;
    const long long w_begin = plan_w0(blockIdx.x, W, G);
    const int n_units = static_cast<int>(plan_w0(blockIdx.x + 1, W, G) - w_begin);
    const int BT = plan.base_tiles;
    const int g_begin = static_cast<int>(w_begin / BT);
    const int j_begin = static_cast<int>(w_begin - static_cast<long long>(g_begin) * BT);

    const uint32_t bar_full = ptx::smem_u32(&ctl->full[0]);
    const uint32_t bar_empty = ptx::smem_u32(&ctl->empty[0]);
    const uint32_t bar_nempty = ptx::smem_u32(&ctl->nempty[0]);
    const uint32_t bar_qfull = ptx::smem_u32(&ctl->qfull);
    const uint32_t bar_qempty = ptx::smem_u32(&ctl->qempty);
    const uint32_t bar_tfull = ptx::smem_u32(&ctl->tfull[0]);
    const uint32_t bar_tempty = ptx::smem_u32(&ctl->tempty[0]);
    const uint32_t bar_drain = ptx::smem_u32(&ctl->drain);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            ptx::mbar_init(bar_full + 8 * s, 1);
            ptx::mbar_init(bar_empty + 8 * s, 1);
            ptx::mbar_init(bar_nempty + 8 * s, kEpiWarps);
        }
        ptx::mbar_init(bar_qfull, 1);
        ptx::mbar_init(bar_qempty, 1);
        for (int i = 0; i < kQT; ++i) {
            ptx::mbar_init(bar_tfull + 8 * i, 1);
            ptx::mbar_init(bar_tempty + 8 * i, 4);  // the four lane-quarter warps of tile i
        }
        ptx::mbar_init(bar_drain, 1);
        ctl->abort_flag = 0;
        ctl->no_abort = 0;
        ptx::fence_mbar_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), kTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    volatile int* abort_flag = &ctl->abort_flag;
    volatile int* never = &ctl->no_abort;  // drain waits: time-bounded, never aborted early

    if (warp == 0) {
        if (lane == 0) {
            // ------------------------------------------------ TMA producer
            ptx::tma_prefetch_desc(&qmap);
            ptx::tma_prefetch_desc(&bmap);
            int cur_g = -1, ngroups = 0;
            int g = g_begin, j = j_begin;
            int n = 0;
            for (; n < n_units; ++n) {
                if (g != cur_g) {
                    if (ngroups > 0 &&
                        !ptx::mbar_wait(bar_qempty, (ngroups - 1) & 1, abort_flag, err, kErrWaitQuery))
                        break;
                    const int t0 = g * kQT;
                    const int nqt = min(kQT, plan.q_tiles - t0);
                    ptx::mbar_arrive_expect_tx(bar_qfull, nqt * kQTileBytes);
                    for (int t = 0; t < nqt; ++t)
                        ptx::tma_load_2d(q_s + t * kQTileBytes, &qmap, 0, (t0 + t) * kBM, bar_qfull);
                    cur_g = g;
                    ++ngroups;
                }
                const int s = n % kStages;
                const uint32_t par = ((n / kStages) & 1) ^ 1;
                if (!ptx::mbar_wait(bar_empty + 8 * s, par, abort_flag, err, kErrWaitProducer)) break;
                if (!ptx::mbar_wait(bar_nempty + 8 * s, par, abort_flag, err, kErrWaitProducer)) break;
                ptx::mbar_arrive_expect_tx(bar_full + 8 * s, kBTileBytes + kRecBytes);
                ptx::tma_load_2d(b_s + s * kBTileBytes, &bmap, 0, j * kBN, bar_full + 8 * s);
                ptx::bulk_load(r_s + s * kRecBytes, brec + static_cast<size_t>(j) * kRecInts, kRecBytes,
                               bar_full + 8 * s);
                if (++j == BT) { j = 0; ++g; }
            }
            // Drain: every issued copy lands before the CTA may exit.
            for (int k = (n > kStages ? n - kStages : 0); k < n; ++k)
                ptx::mbar_wait(bar_full + 8 * (k % kStages), (k / kStages) & 1, never, err, kErrWaitDrain);
            if (ngroups > 0) ptx::mbar_wait(bar_qfull, (ngroups - 1) & 1, never, err, kErrWaitDrain);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            // -------------------------------------------------- MMA issuer
            constexpr uint32_t idesc = ptx::idesc_make(2 /*S32*/, 0 /*u8*/, 0 /*u8*/, kBM, kBN);
            int cur_g = -1, ngroups = 0, nqt = 0;
            int g = g_begin, j = j_begin;
            uint32_t use_parity = 0;  // bit t: parity of the accumulator uses of tile t so far
            bool ok = true;
            for (int n = 0; n < n_units && ok; ++n) {
                if (g != cur_g) {
                    if (!ptx::mbar_wait(bar_qfull, ngroups & 1, abort_flag, err, kErrWaitQuery)) break;
                    cur_g = g;
                    ++ngroups;
                    nqt = min(kQT, plan.q_tiles - g * kQT);
                }
                const int s = n % kStages;
                if (!ptx::mbar_wait(bar_full + 8 * s, (n / kStages) & 1, abort_flag, err, kErrWaitMmaFull)) break;
                ptx::tc_fence_after();
                const uint32_t b0 = b_s + s * kBTileBytes;
                #pragma unroll
                for (int t = 0; t < kQT; ++t) {
                    if (t < nqt && ok) {
                        if (!ptx::mbar_wait(bar_tempty + 8 * t, ((use_parity >> t) & 1) ^ 1, abort_flag, err,
                                            kErrWaitMmaTmem)) {
                            ok = false;
                        } else {
                            ptx::tc_fence_after();
                            const uint32_t d = tmem + t * kBN;
                            const uint32_t a0 = q_s + t * kQTileBytes;
                            #pragma unroll
                            for (int kk = 0; kk < kDim / 32; ++kk)
                                ptx::mma_i8(d, ptx::sdesc_sw128(a0 + kk * 32), ptx::sdesc_sw128(b0 + kk * 32), idesc,
                                            kk > 0 ? 1u : 0u);
                            ptx::tc_commit(bar_tfull + 8 * t);
                            use_parity ^= 1u << t;
                        }
                    }
                }
                if (!ok) break;
                ptx::tc_commit(bar_empty + 8 * s);
                const bool last_of_group = (n + 1 == n_units) || (j + 1 == BT);
                if (last_of_group) ptx::tc_commit(bar_qempty);
                if (++j == BT) { j = 0; ++g; }
            }
            // Drain: all issued MMAs complete before TMEM is released.
            ptx::tc_commit(bar_drain);
            ptx::mbar_wait(bar_drain, 0, never, err, kErrWaitDrain);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------ epilogue
        const int e = warp - 2;
        const int t = e >> 2;          // query tile of this warp
        const int quarter = warp & 3;  // TMEM lane quarter this warp may access
        const uint32_t taddr0 = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + t * kBN;
        Top2 st{INT_MAX, -1, INT_MAX, -1, INT_MAX};
        int published = INT_MAX;
        int cur_g = -1, nqt = 0, split = 0, q = 0;
        int g = g_begin, j = j_begin;
        uint32_t use = 0;

        for (int n = 0; n < n_units; ++n) {
            if (g != cur_g) {
                if (cur_g >= 0 && t < nqt)
                    partial[static_cast<size_t>(split) * plan.q_pad + q] = make_int4(st.k1, st.i1, st.k2, st.i2);
                st = Top2{INT_MAX, -1, INT_MAX, -1, INT_MAX};
                published = INT_MAX;
                cur_g = g;
                nqt = min(kQT, plan.q_tiles - g * kQT);
                split = static_cast<int>(blockIdx.x) - plan_cta_of(static_cast<long long>(g) * BT, W, G);
                q = (g * kQT + t) * kBM + quarter * 32 + lane;
            }
            const bool active = t < nqt;
            // Bound shared with the other CTAs that scan this query's group;
            // loaded before the waits so its latency hides behind them.
            const int shared_thr = active ? __ldcg(thresh + q) : INT_MAX;
            const int s = n % kStages;
            bool waited = ptx::mbar_wait(bar_full + 8 * s, (n / kStages) & 1, abort_flag, err, kErrWaitEpilogue);
            if (active && waited)
                waited = ptx::mbar_wait(bar_tfull + 8 * t, use & 1, abort_flag, err, kErrWaitEpilogue);
            if (!__all_sync(0xffffffffu, waited)) break;
            if (active) {
                ++use;
                ptx::tc_fence_after();
                st.thr = min(st.thr, shared_thr);
                const int32_t* rec = r_smem + s * kRecInts;
                const int row0 = j * kBN;
                uint32_t va[32];
                ptx::tmem_ld32(taddr0, va);
                ptx::tmem_ld_wait(va);
                scan_group(va, row0, rec, rec + 128, st);
                ptx::tmem_ld32(taddr0 + 32, va);
                ptx::tmem_ld_wait(va);
                scan_group(va, row0 + 32, rec + 32, rec + 132, st);
                ptx::tmem_ld32(taddr0 + 64, va);
                ptx::tmem_ld_wait(va);
                scan_group(va, row0 + 64, rec + 64, rec + 136, st);
                ptx::tmem_ld32(taddr0 + 96, va);
                ptx::tmem_ld_wait(va);
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar_tempty + 8 * t);
                scan_group(va, row0 + 96, rec + 96, rec + 140, st);
                if (st.k2 < published) {
                    atomicMin(thresh + q, st.k2);
                    published = st.k2;
                }
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar_nempty + 8 * s);
            if (++j == BT) { j = 0; ++g; }
        }
        if (cur_g >= 0 && t < nqt)
            partial[static_cast<size_t>(split) * plan.q_pad + q] = make_int4(st.k1, st.i1, st.k2, st.i2);
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, kTmemCols);
    }
}

__device__ __forceinline__ bool lex_less(int ka, int ia, int kb, int ib) {
    return ka < kb || (ka == kb && ia < ib);
}

// Lexicographic (key, index) top-2 of one query row while its partial lists
// are merged. Every base row is in exactly one list and (key, index) is a total
// order, so the result does not depend on the order of the pushes.
struct MergeTop2 {
    int k1 = INT_MAX, i1 = -1, k2 = INT_MAX, i2 = -1;
    __device__ __forceinline__ void push(int k, int i) {
        if (i < 0) return;
        if (lex_less(k, i, k1, i1) || i1 < 0) {
            k2 = k1; i2 = i1;
            k1 = k; i1 = i;
        } else if (lex_less(k, i, k2, i2) || i2 < 0) {
            k2 = k; i2 = i;
        }
    }
    __device__ __forceinline__ void push(const int4& p) {
        push(p.x, p.y);
        push(p.z, p.w);
    }
};

struct MergeOut {
    uint32_t* matches;
    float4* sorted;
    int32_t* nn_idx;
    float* nn_dist;
    float qmul = 0.0f;
};

// Distances, ratio test and outputs of query row q. Rows past the problem's
// base set (index >= n_b) are padding: they may hold another problem's rows,
// but only enter a top-2 when fewer real rows exist. FLOATKEY: the keys are
// ordered images of float keys (float_key) and qn is a float bit pattern (the
// general float path); else integers.
template <bool FLOATKEY>
__device__ __forceinline__ void merge_finish(const MergeTop2& t, int q, int n_b, const int32_t* qnorm,
                                             int metric, float thr, float dscale, const MergeOut& out) {
    // out.qmul (FP16 rows holding integers): query norms are floats, the integers divided by it.
    bool v1, v2;
    float d1, d2;
    if constexpr (FLOATKEY) {
        // Squared distances |b|^2 - 2 q.b + |q|^2 can round a little below
        // zero for (near-)identical rows: clamped at 0.
        v1 = t.i1 >= 0 && t.i1 < n_b;
        v2 = t.i2 >= 0 && t.i2 < n_b;
        const float qn = metric == kMetricL2 ? __int_as_float(qnorm[q]) : 0.0f;
        const float lo = metric == kMetricL2 ? 0.0f : -FLT_MAX;
        d1 = v1 ? fmaxf((key_float(t.k1) + qn) * dscale, lo) : FLT_MAX;
        d2 = v2 ? fmaxf((key_float(t.k2) + qn) * dscale, lo) : FLT_MAX;
    } else {
        v1 = t.i1 >= 0 && t.i1 < n_b && t.k1 < kKeyPad;
        v2 = t.i2 >= 0 && t.i2 < n_b && t.k2 < kKeyPad;
        int qn = metric == kMetricL2 ? qnorm[q] : 0;
        if (out.qmul > 0.0f) qn = __float2int_rn(__int_as_float(qn) * out.qmul);
        d1 = v1 ? static_cast<float>(t.k1 + qn) * dscale : FLT_MAX;
        d2 = v2 ? static_cast<float>(t.k2 + qn) * dscale : FLT_MAX;
    }
    if (out.matches) {
        bool pass = false;
        if (v1) {
            float f1, f2;
            if (metric == kMetricL2) {
                f1 = sqrtf(d1);
                f2 = v2 ? sqrtf(d2) : INFINITY;
            } else {
                f1 = sqrtf(d1 + 2.0f);
                f2 = v2 ? sqrtf(d2 + 2.0f) : INFINITY;
            }
            pass = (f1 / f2) < thr;
        }
        out.matches[q] = pass ? static_cast<uint32_t>(t.i1) : UINT32_MAX;
    }
    if (out.sorted)
        out.sorted[q] =
            make_float4(d1, d2, v1 ? static_cast<float>(t.i1) : FLT_MAX, v2 ? static_cast<float>(t.i2) : FLT_MAX);
    if (out.nn_idx) {
        out.nn_idx[2 * static_cast<size_t>(q)] = v1 ? t.i1 : -1;
        out.nn_idx[2 * static_cast<size_t>(q) + 1] = v2 ? t.i2 : -1;
    }
    if (out.nn_dist) {
        out.nn_dist[2 * static_cast<size_t>(q)] = d1;
        out.nn_dist[2 * static_cast<size_t>(q) + 1] = d2;
    }
}

// Merge of the partial lists of one search or a batch. A query row has
// (workers of its group) x parts lists: 76 at 1,000 x 10,000, ~10 at
// 10,000 x 1,000,000, 2-4 in a batch. What bounds it is the chain of dependent
// loads per row, so a block of LANES warps owns 32 query rows: warp w reads
// every LANES-th list of all 32 rows (512 consecutive bytes per list, four
// lists in flight), the partial top-2s cross through shared memory so that
// LANES consecutive threads hold one row's, and shuffles merge them. LANES = 1
// (a thread per row, 256 rows per block) for the few lists of a batch.
// launch_merge has the rule. Measured (whole match() call): 1,000 x 10,000
// 56.5 -> 33.8 us, FP16 2,561 x 500,003 435 -> 427 us against one thread per row.
constexpr int kMergeRows = 32;
template <int LANES>
constexpr int kMergeThreads = LANES == 1 ? 256 : kMergeRows * LANES;

// All LANES threads of the block's row (threadIdx.x / LANES) return its top-2.
template <int LANES>
__device__ __forceinline__ MergeTop2 merge_lists_of_rows(const MergeTop2& mine) {
    __shared__ int4 s_top[LANES][kMergeRows + 1];
    s_top[threadIdx.x / kMergeRows][threadIdx.x % kMergeRows] = make_int4(mine.k1, mine.i1, mine.k2, mine.i2);
    __syncthreads();
    const int4 p = s_top[threadIdx.x % LANES][threadIdx.x / LANES];
    MergeTop2 t{p.x, p.y, p.z, p.w};
    #pragma unroll
    for (int off = 1; off < LANES; off <<= 1) {
        const int4 o = make_int4(__shfl_xor_sync(0xffffffffu, t.k1, off), __shfl_xor_sync(0xffffffffu, t.i1, off),
                                 __shfl_xor_sync(0xffffffffu, t.k2, off), __shfl_xor_sync(0xffffffffu, t.i2, off));
        t.push(o);
    }
    return t;
}

// Lists sub, sub + step, ... < n of a row (list s at p + s * stride).
__device__ __forceinline__ void merge_lists(MergeTop2& t, const int4* p, size_t stride, int sub, int n,
                                            int step) {
    int s = sub;
    for (; s + 3 * step < n; s += 4 * step) {
        int4 v[4];
        #pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = p[static_cast<size_t>(s + k * step) * stride];
        #pragma unroll
        for (int k = 0; k < 4; ++k) t.push(v[k]);
    }
    for (; s < n; s += step) t.push(p[static_cast<size_t>(s) * stride]);
}

template <bool FLOATKEY, int LANES>
__global__ void __launch_bounds__(kMergeThreads<LANES>)
    merge2nn_kernel(const int4* partial, const ExactPlan plan, const WorkItem* items,
                    int n_items, const WorkItem single, int group_rows, int total_q, const int32_t* qnorm,
                    int metric, float thr, float dscale, const MergeOut out) {
    wait_previous();
    const int row0 = blockIdx.x * (kMergeThreads<LANES> / LANES);
    int q = row0 + (LANES == 1 ? threadIdx.x : threadIdx.x % kMergeRows);
    const long long W = plan.weight > 0 ? plan.weight : plan.units, G = plan.grid;
    auto item_of = [&](int row) {
        return items ? items[find_item(n_items, row, [&](int k) { return static_cast<long long>(items[k].a_off); })]
                     : single;
    };
    MergeTop2 t;
    if (LANES == 1 && q >= total_q) return;
    int n_b = 0;
    if (q < total_q) {
        const WorkItem it = item_of(q);
        n_b = it.n_b;
        // No base rows: no CTA scanned this query and every neighbour is absent.
        if (W > 0 && it.tiles > 0) {
            const int g = (q - it.a_off) / group_rows;
            long long first = it.u_begin + static_cast<long long>(g) * it.tiles, last = first + it.tiles - 1;
            if (plan.weight > 0) {
                first = unit_weight_begin(it, group_rows, g, 0);
                last = unit_weight_begin(it, group_rows, g, it.tiles - 1);
            }
            const int c0 = plan_cta_of(first, W, G);
            const int c1 = plan_cta_of(last, W, G);
            merge_lists(t, partial + q, plan.q_pad, LANES == 1 ? 0 : threadIdx.x / kMergeRows,
                        (c1 - c0 + 1) * plan.parts, LANES);
        }
    }
    if constexpr (LANES > 1) {
        t = merge_lists_of_rows<LANES>(t);
        q = row0 + threadIdx.x / LANES;
        if (threadIdx.x % LANES != 0 || q >= total_q) return;
        n_b = item_of(q).n_b;
    }
    merge_finish<FLOATKEY>(t, q, n_b, qnorm, metric, thr, dscale, out);
}

// Merge of a search split over base chunks (indices already global): ~75 lists
// per query row for 10,000 x 1,000,000 in 8 chunks, read as merge2nn_kernel
// reads them.
constexpr int kMergeChunkLanes = 8;
__global__ void __launch_bounds__(kMergeThreads<kMergeChunkLanes>)
    merge2nn_chunks_kernel(const int4* __restrict__ partial, const ChunkSet cs, int q_n,
                           const int32_t* __restrict__ qnorm, int metric, float thr, float dscale,
                           const MergeOut out) {
    constexpr int LANES = kMergeChunkLanes;
    int q = blockIdx.x * kMergeRows + threadIdx.x % kMergeRows;
    const int sub = threadIdx.x / kMergeRows;
    MergeTop2 t;
    if (q < q_n) {
        const int g = q / (kQT * kBM);
        int done = 0;  // lists of the earlier chunks
        for (int c = 0; c < cs.n; ++c) {
            if (cs.W[c] <= 0 || cs.tiles[c] <= 0) continue;
            const long long first = static_cast<long long>(g) * cs.tiles[c];
            const int c0 = plan_cta_of(first, cs.W[c], cs.G[c]);
            const int c1 = plan_cta_of(first + cs.tiles[c] - 1, cs.W[c], cs.G[c]);
            const int n_lists = (c1 - c0 + 1) * cs.parts;
            merge_lists(t, partial + c * cs.slot_stride + q, cs.q_pad, (sub - done % LANES + LANES) % LANES, n_lists,
                        LANES);
            done += n_lists;
        }
    }
    t = merge_lists_of_rows<LANES>(t);
    q = blockIdx.x * kMergeRows + threadIdx.x / LANES;
    if (threadIdx.x % LANES != 0 || q >= q_n) return;
    merge_finish<false>(t, q, cs.r_n, qnorm, metric, thr, dscale, out);
}

}  // namespace

cudaError_t launch_merge2nn_chunks(const int4* partial, const ChunkSet& cs, int q_n, const int32_t* qnorm, int metric,
                                   float threshold, float dist_scale, uint32_t* matches, float4* sorted,
                                   int32_t* nn_idx, float* nn_dist, cudaStream_t stream) {
    if (q_n <= 0) return cudaSuccess;
    merge2nn_chunks_kernel<<<(q_n + kMergeRows - 1) / kMergeRows, kMergeThreads<kMergeChunkLanes>, 0, stream>>>(
        partial, cs, q_n, qnorm, metric, threshold, dist_scale, MergeOut{matches, sorted, nn_idx, nn_dist});
    return cudaGetLastError();
}

ExactPlan make_exact_plan(int q_n, int r_n, int num_sms, int parts, int group_tiles) {
    ExactPlan p{};
    p.parts = parts;
    p.q_n = q_n;
    p.r_n = r_n;
    p.q_tiles = (q_n + kBM - 1) / kBM;
    p.q_groups = (p.q_tiles + group_tiles - 1) / group_tiles;
    p.q_pad = p.q_tiles * kBM;
    p.base_tiles = (r_n + kBN - 1) / kBN;
    p.r_pad = p.base_tiles * kBN;
    p.units = static_cast<long long>(p.q_groups) * p.base_tiles;
    p.grid = static_cast<int>(std::min<long long>(num_sms, p.units));
    int ms = 1;
    if (p.grid > 0) {
        for (int g = 0; g < p.q_groups; ++g) {
            const long long BT = p.base_tiles;
            const int c0 = plan_cta_of(g * BT, p.units, p.grid);
            const int c1 = plan_cta_of((g + 1) * BT - 1, p.units, p.grid);
            ms = std::max(ms, c1 - c0 + 1);
        }
    }
    p.max_splits = ms;
    return p;
}

size_t exact2nn_smem_bytes() { return kSmemBytes; }

cudaError_t launch_row_norms_u8(const uint8_t* x, int n, int n_pad, int metric, int32_t* norm, int32_t* rec,
                                int32_t* thresh, cudaStream_t stream) {
    if (n_pad <= 0) return cudaSuccess;
    row_norms_kernel<<<n_pad / 32, 256, 0, stream>>>(x, n, n_pad, metric, norm, rec, thresh);
    return cudaGetLastError();
}

cudaError_t launch_fold_records_u8(const uint8_t* x, int n, int n_pad, int metric, int32_t* rec, uint32_t* fold,
                                   const uint8_t* q, int q_n, int q_pad, int32_t* qnorm, int32_t* thresh,
                                   cudaStream_t stream) {
    const int blocks = n_pad / kBN + (q_pad + kBN - 1) / kBN;
    if (blocks <= 0) return cudaSuccess;
    fold_records_kernel<<<blocks, 256, 0, stream>>>(x, n, n_pad, metric, rec, fold, q, q_n, q_pad, qnorm, thresh);
    return cudaGetLastError();
}

cudaError_t launch_row_norms_float(const void* x, int n, int n_pad, int metric, int32_t* norm, int32_t* rec,
                                   int32_t* thresh, cudaStream_t stream) {
    if (n_pad <= 0) return cudaSuccess;
    row_norms_float_kernel<<<n_pad / 32, 256, 0, stream>>>(static_cast<const __half*>(x), n, n_pad, metric, norm, rec,
                                                           thresh);
    return cudaGetLastError();
}

cudaError_t launch_exact2nn_u8(const CUtensorMap& qmap, const CUtensorMap& bmap, const int32_t* brec,
                               const ExactPlan& plan, int4* partial, int32_t* thresh, int* err, cudaStream_t stream) {
    // The shared-memory opt-in is per device; the host API serialises calls per device.
    static bool attr_set[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(exact2nn_u8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kSmemBytes));
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    if (plan.grid <= 0) return cudaSuccess;
    exact2nn_u8_kernel<<<plan.grid, kThreads, kSmemBytes, stream>>>(qmap, bmap, brec, plan, partial, thresh, err);
    return cudaGetLastError();
}

// The launch of merge2nn_kernel with as many warps per 32 rows as the longest
// row has lists to share out, in steps of 1, 8 and 32 (one list per thread up
// to 32 lists, three at the 76 of 1,000 x 10,000; at 2-4 lists the exchange
// through shared memory would cost more than the second load it saves).
template <bool FLOATKEY>
cudaError_t launch_merge(const int4* partial, const ExactPlan& plan, const WorkItem* items, int n_items,
                         const WorkItem& single, int group_rows, int total_q, const int32_t* qnorm, int metric,
                         float threshold, float dist_scale, const MergeOut& out, cudaStream_t stream) {
    if (total_q <= 0) return cudaSuccess;
    const int lists = plan.max_splits * plan.parts;
    const int blocks = (total_q + kMergeRows - 1) / kMergeRows;
    if (lists <= 4)
        return launch_after(merge2nn_kernel<FLOATKEY, 1>, (total_q + 255) / 256, kMergeThreads<1>, 0, stream,
            partial, plan, items, n_items, single, group_rows, total_q, qnorm, metric, threshold, dist_scale, out);
    if (lists <= 32)
        return launch_after(merge2nn_kernel<FLOATKEY, 8>, blocks, kMergeThreads<8>, 0, stream,
            partial, plan, items, n_items, single, group_rows, total_q, qnorm, metric, threshold, dist_scale, out);
    return launch_after(merge2nn_kernel<FLOATKEY, 32>, blocks, kMergeThreads<32>, 0, stream,
            partial, plan, items, n_items, single, group_rows, total_q, qnorm, metric, threshold, dist_scale, out);
}

WorkItem merge_item(const ExactPlan& plan) {
    WorkItem single{};
    single.n_a = plan.q_n;
    single.n_b = plan.r_n;
    single.groups = plan.q_groups;
    single.tiles = plan.base_tiles;
    return single;
}

cudaError_t launch_merge2nn(const int4* partial, const ExactPlan& plan, const int32_t* qnorm, int metric,
                            float threshold, float dist_scale, uint32_t* matches, float4* sorted, int32_t* nn_idx,
                            float* nn_dist, cudaStream_t stream, float qnorm_mul) {
    return launch_merge<false>(partial, plan, nullptr, 1, merge_item(plan), kQT * kBM, plan.q_n, qnorm, metric,
                               threshold, dist_scale, MergeOut{matches, sorted, nn_idx, nn_dist, qnorm_mul}, stream);
}

cudaError_t launch_merge2nn_float(const int4* partial, const ExactPlan& plan, int group_rows, const int32_t* qnorm,
                                  int metric, float threshold, float dist_scale, uint32_t* matches, float4* sorted,
                                  int32_t* nn_idx, float* nn_dist, cudaStream_t stream) {
    return launch_merge<true>(partial, plan, nullptr, 1, merge_item(plan), group_rows, plan.q_n, qnorm, metric,
                              threshold, dist_scale, MergeOut{matches, sorted, nn_idx, nn_dist}, stream);
}

cudaError_t launch_merge2nn_batch(const int4* partial, const BatchPlan& bp, int total_queries, const int32_t* qnorm,
                                  int metric, float threshold, float dist_scale, uint32_t* matches, float4* sorted,
                                  int32_t* nn_idx, float* nn_dist, cudaStream_t stream) {
    return launch_merge<false>(partial, bp.plan, bp.items, bp.n_items, WorkItem{}, bp.group_rows, total_queries, qnorm,
                               metric, threshold, dist_scale, MergeOut{matches, sorted, nn_idx, nn_dist}, stream);
}

cudaError_t launch_batch_prep(const uint8_t* base, const uint8_t* q, int q_n, const BatchPlan& bp, int32_t* rec,
                              int32_t* qnorm, int32_t* thresh, cudaStream_t stream) {
    const int blocks = bp.total_tiles + bp.plan.q_tiles;
    if (blocks <= 0) return cudaSuccess;
    WorkItem single{};
    single.n_b = bp.plan.r_n;
    batch_prep_kernel<<<blocks, 256, 0, stream>>>(base, bp.items, bp.n_items, single, bp.total_tiles, rec, q, q_n,
                                                  bp.plan.q_pad, qnorm, thresh);
    return cudaGetLastError();
}

long long make_batch_items(int n_items, const int* n_a, const int* n_b, const int* b_off, int group_rows,
                           WorkItem* items, int* total_tiles, int* total_queries) {
    long long u = 0, w = 0;
    int a = 0, rec = 0;
    for (int p = 0; p < n_items; ++p) {
        WorkItem& it = items[p];
        it = WorkItem{};
        it.a_off = a;
        it.n_a = n_a[p];
        it.b_off = b_off[p];
        it.n_b = n_b[p];
        it.groups = (n_a[p] + group_rows - 1) / group_rows;
        it.tiles = (n_b[p] + kBN - 1) / kBN;
        it.u_begin = u;
        it.w_begin = w;
        it.rec_off = rec;
        if (it.groups > 0) w = unit_weight_begin(it, group_rows, it.groups - 1, it.tiles);
        u += static_cast<long long>(it.groups) * it.tiles;
        rec += it.tiles;
        a += n_a[p];
    }
    if (total_tiles) *total_tiles = rec;
    if (total_queries) *total_queries = a;
    return u;
}

constexpr int kMinWeightedUnits = 8;  // per worker: they weigh at least 32, a dense unit 6
ExactPlan make_batch_plan(const WorkItem* items, int n_items, int group_rows, long long units, int total_queries,
                          int num_workers, int parts) {
    ExactPlan p{};
    p.parts = parts;
    p.q_n = total_queries;
    p.r_n = 0;
    p.q_tiles = (total_queries + kBM - 1) / kBM;
    p.q_pad = p.q_tiles * kBM;
    p.units = units;
    p.grid = static_cast<int>(std::min<long long>(num_workers, units));
    int ms = 1;
    // A share of at least one dense unit's weight holds a unit: no worker of a
    // group's range is without one, so every list that the merge reads is written.
    if (units >= kMinWeightedUnits * static_cast<long long>(p.grid) && n_items > 0) {
        const WorkItem& it = items[n_items - 1];
        p.weight = it.groups > 0 ? unit_weight_begin(it, group_rows, it.groups - 1, it.tiles) : it.w_begin;
    }
    const long long W = p.weight > 0 ? p.weight : units;
    if (p.grid > 0) {
        for (int k = 0; k < n_items; ++k) {
            const WorkItem& it = items[k];
            for (int g = 0; g < it.groups && it.tiles > 0; ++g) {
                long long first = it.u_begin + static_cast<long long>(g) * it.tiles, last = first + it.tiles - 1;
                if (p.weight > 0) {
                    first = unit_weight_begin(it, group_rows, g, 0);
                    last = unit_weight_begin(it, group_rows, g, it.tiles - 1);
                }
                const int c0 = plan_cta_of(first, W, p.grid);
                const int c1 = plan_cta_of(last, W, p.grid);
                ms = std::max(ms, c1 - c0 + 1);
            }
        }
    }
    p.max_splits = ms;
    return p;
}

}  // namespace sift
