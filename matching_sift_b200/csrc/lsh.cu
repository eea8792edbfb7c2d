// Random-hyperplane LSH for u8 SIFT descriptors on sm_100a.
//
// Replaces the reference's LSH pipeline (src/lsh_h.cu):
//   hash GEMM cublasHgemm(H, X)            :909, :914   -> lsh_hash_kernel (tcgen05 kind::i8)
//   set_bit_h sign packing                 :265-317     -> fused into lsh_hash_kernel's epilogue
//   thrust::sort by code + host run-length :565-629     -> bucket histogram / scan / scatter kernels
//   host merge-join of Q and R buckets     :657-681     -> the query code indexes the bucket table
//   brute_2nn_h + atomic_min2_update       :441-562     -> lsh_scan_kernel (warp or block per query)
//
// Codes. Table t of L uses k hyperplanes; bit j of a point's code is set when
// its dot product with hyperplane j is negative (set_bit_h, src/lsh_h.cu:302-309).
// Hyperplanes are int8, so the dot products are exact integers computed on
// the tensor cores (u8 x s8 -> s32), and a code is a pure function of the
// point and the hyperplanes.
//
// Buckets. Per table, base points are grouped by the top B = min(k, 16) bits
// of their code (counting sort: histogram, exclusive scan, scatter). A query
// scans the group of its own top bits and keeps the members whose full code
// equals its own, so every table contributes exactly the bucket of the
// query's code (the reference scans sorted positions starting at a point id
// instead, src/lsh_h.cu:599,617 vs :469,482, which is not the bucket).
//
// Candidate scan. One warp or one block per query over its L buckets (L x P
// with P probe codes per table: multi-probe); candidate rows are fetched by
// groups of 8 lanes with coalesced 16-byte loads (4 rows per warp-wide load)
// and scored as the exact |q - b|^2 (dp4a); the per-query top-2 is
// lexicographic in (distance, index) and counts a base point found in several
// tables once.
#include <algorithm>
#include <climits>
#include <cfloat>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>
#include "lsh.cuh"
#include "ptx.cuh"

namespace sift {
namespace {

// ------------------------------------------------------------ hash kernel
constexpr int kHStages = 6;
constexpr int kHTileBytes = 128 * 128;  // 128 points x 128 u8
constexpr int kHThreads = 64 + 4 * 32;  // producer, MMA, 4 epilogue warps

struct __align__(8) HashCtl {
    uint64_t full[kHStages], empty[kHStages];
    uint64_t pfull;
    uint64_t tfull[4], tempty[4];
    uint64_t drain;
    uint32_t tmem_base;
    int abort_flag, no_abort;
};

__host__ __device__ constexpr size_t hash_smem_bytes(int P) {
    return 1024 + static_cast<size_t>(P) * 128 + kHStages * kHTileBytes + sizeof(HashCtl);
}

// P = number of hyperplane rows padded to a multiple of 32 (<= 256). TMEM:
// nbuf accumulator buffers of slot_cols columns (P rounded up to a power of
// two; nbuf = 4 for P <= 128, else 2), so the MMA of tile i + nbuf - 1 can run
// while the epilogue still reads tile i.
__global__ void __launch_bounds__(kHThreads, 1)
    lsh_hash_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap pmap, int n, int P,
                    int L, int k, int nbuf, uint32_t slot_cols, uint32_t* __restrict__ codes,
                    float* __restrict__ z, int* __restrict__ err) {
    const uint32_t tmem_cols = static_cast<uint32_t>(nbuf) * slot_cols;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = ptx::smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
    uint8_t* p_smem = smem;                                   // P x 128 planes (s8)
    uint8_t* x_smem = smem + static_cast<size_t>(P) * 128;    // point tile ring (P*128 is a multiple of 1024)
    HashCtl* ctl = reinterpret_cast<HashCtl*>(x_smem + kHStages * kHTileBytes);
    const uint32_t p_s = ptx::smem_u32(p_smem), x_s = ptx::smem_u32(x_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = (n + 127) / 128;
    const int my_tiles = blockIdx.x < tiles ? (tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;

    const uint32_t bar_full = ptx::smem_u32(&ctl->full[0]), bar_empty = ptx::smem_u32(&ctl->empty[0]);
    const uint32_t bar_pfull = ptx::smem_u32(&ctl->pfull), bar_drain = ptx::smem_u32(&ctl->drain);
    const uint32_t bar_tfull = ptx::smem_u32(&ctl->tfull[0]), bar_tempty = ptx::smem_u32(&ctl->tempty[0]);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kHStages; ++s) {
            ptx::mbar_init(bar_full + 8 * s, 1);
            ptx::mbar_init(bar_empty + 8 * s, 1);
        }
        ptx::mbar_init(bar_pfull, 1);
        for (int b = 0; b < nbuf; ++b) {
            ptx::mbar_init(bar_tfull + 8 * b, 1);
            ptx::mbar_init(bar_tempty + 8 * b, 4);
        }
        ptx::mbar_init(bar_drain, 1);
        ctl->abort_flag = 0;
        ctl->no_abort = 0;
        ptx::fence_mbar_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), tmem_cols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    volatile int* abort_flag = &ctl->abort_flag;
    volatile int* never = &ctl->no_abort;

    if (warp == 0) {
        if (lane == 0) {
            ptx::tma_prefetch_desc(&xmap);
            ptx::tma_prefetch_desc(&pmap);
            // One box of all P hyperplane rows (the map's box is P rows, P <= 256).
            ptx::mbar_arrive_expect_tx(bar_pfull, P * 128);
            ptx::tma_load_2d(p_s, &pmap, 0, 0, bar_pfull);
            int i = 0;
            for (; i < my_tiles; ++i) {
                const int s = i % kHStages;
                if (!ptx::mbar_wait(bar_empty + 8 * s, ((i / kHStages) & 1) ^ 1, abort_flag, err, kErrWaitProducer))
                    break;
                ptx::mbar_arrive_expect_tx(bar_full + 8 * s, kHTileBytes);
                ptx::tma_load_2d(x_s + s * kHTileBytes, &xmap, 0, (blockIdx.x + i * gridDim.x) * 128, bar_full + 8 * s);
            }
            for (int kk = (i > kHStages ? i - kHStages : 0); kk < i; ++kk)
                ptx::mbar_wait(bar_full + 8 * (kk % kHStages), (kk / kHStages) & 1, never, err, kErrWaitDrain);
            ptx::mbar_wait(bar_pfull, 0, never, err, kErrWaitDrain);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            // u8 points (A) x s8 hyperplanes (B) -> s32, in MMAs of at most
            // 128 hyperplane columns: P > 128 is split into two equal chunks
            // of P/2 columns (a multiple of 16; each chunk starts on a
            // 1024-byte swizzle atom) written to adjacent TMEM columns.
            const int nchunk = (P + 127) / 128;
            const uint32_t nc = static_cast<uint32_t>(P / nchunk);
            const uint32_t idesc = ptx::idesc_make(2 /*S32*/, 0 /*u8*/, 1 /*s8*/, 128, nc);
            bool ok = ptx::mbar_wait(bar_pfull, 0, abort_flag, err, kErrWaitMmaFull);
            for (int i = 0; i < my_tiles && ok; ++i) {
                const int s = i % kHStages, b = i % nbuf;
                if (!ptx::mbar_wait(bar_full + 8 * s, (i / kHStages) & 1, abort_flag, err, kErrWaitMmaFull)) break;
                if (!ptx::mbar_wait(bar_tempty + 8 * b, ((i / nbuf) & 1) ^ 1, abort_flag, err, kErrWaitMmaTmem))
                    break;
                ptx::tc_fence_after();
                const uint32_t d = tmem + b * slot_cols;
                for (int ch = 0; ch < nchunk; ++ch) {
                    #pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        ptx::mma_i8(d + ch * nc, ptx::sdesc_sw128(x_s + s * kHTileBytes + kk * 32),
                                    ptx::sdesc_sw128(p_s + ch * nc * 128 + kk * 32), idesc, kk > 0 ? 1u : 0u);
                }
                ptx::tc_commit(bar_tfull + 8 * b);
                ptx::tc_commit(bar_empty + 8 * s);
            }
            ptx::tc_commit(bar_drain);
            ptx::mbar_wait(bar_drain, 0, never, err, kErrWaitDrain);
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3;
        for (int i = 0; i < my_tiles; ++i) {
            const int b = i % nbuf;
            const bool waited = ptx::mbar_wait(bar_tfull + 8 * b, (i / nbuf) & 1, abort_flag, err, kErrWaitEpilogue);
            if (!__all_sync(0xffffffffu, waited)) break;
            ptx::tc_fence_after();
            const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + b * slot_cols;
            const int point = (blockIdx.x + i * gridDim.x) * 128 + quarter * 32 + lane;
            uint32_t mask[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            // Up to 4 loads of 32 columns in flight per wait (one TMEM round
            // trip for P <= 128 hyperplanes instead of one per 32 columns).
            #pragma unroll
            for (int w0 = 0; w0 < 8; w0 += 4) {
                if (w0 * 32 < P) {
                    uint32_t v[4][32];
                    #pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if ((w0 + u) * 32 < P) ptx::tmem_ld32(taddr + (w0 + u) * 32, v[u]);
                    ptx::tmem_ld_wait(v[0]);
                    ptx::tmem_ld_wait(v[1]);
                    ptx::tmem_ld_wait(v[2]);
                    ptx::tmem_ld_wait(v[3]);
                    #pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int w = w0 + u;
                        if (w * 32 < P) {
                            uint32_t m = 0;
                            #pragma unroll
                            for (int c = 0; c < 32; ++c) m |= (v[u][c] >> 31) << c;
                            mask[w] = m;
                            if (z && point < n) {
                                // Dot products of the point with each hyperplane (multi-probe margins).
                                #pragma unroll
                                for (int c = 0; c < 32; ++c) {
                                    const int col = w * 32 + c;
                                    if (col < L * k)
                                        z[(static_cast<size_t>(col / k) * n + point) * k + col % k] =
                                            static_cast<float>(static_cast<int>(v[u][c]));
                                }
                            }
                        }
                    }
                }
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar_tempty + 8 * b);
            if (point < n) {
                for (int t = 0; t < L; ++t) {
                    const int bit0 = t * k;
                    const int w = bit0 >> 5, sh = bit0 & 31;
                    // mask[w], mask[w + 1] by selects (register-resident, no indexed access)
                    uint32_t lo = mask[0], hi = mask[1];
                    #pragma unroll
                    for (int u = 1; u < 8; ++u) {
                        lo = w == u ? mask[u] : lo;
                        hi = w + 1 == u ? mask[u] : hi;
                    }
                    if (w + 1 >= 8) hi = 0;
                    const uint64_t pair = static_cast<uint64_t>(lo) | (static_cast<uint64_t>(hi) << 32);
                    const uint32_t code = static_cast<uint32_t>(pair >> sh) & (k == 32 ? 0xffffffffu : ((1u << k) - 1));
                    codes[static_cast<size_t>(t) * n + point] = code;
                }
            }
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, tmem_cols);
    }
}

// --------------------------------------------------------------- buckets
// Counting sort of a table's points by the top bits of their codes, in three
// launches: counts, exclusive scan, scatter. Codes crowd (a bin can hold several
// percent of all points), and one global atomic per point serialises on such a
// bin, so a block takes a chunk of 8,192 points, ranks them within their bins by
// shared-memory atomics on 16-bit counters (128 KB for 65,536 bins), and the
// first point of each bin moves the global counter once for all of them.
// 1M points in the skewed codes of a learned hash: counts + scan + scatter
// 74 + 117 + 80 us with a global atomic per point and one block for the scan,
// 9 + 14 + 22 us now.
constexpr int kChunkThreads = 1024;
constexpr int kChunkPer = 8;
constexpr int kChunkPoints = kChunkThreads * kChunkPer;

// Chunks of n points (n up to 2^31 - 1: the rounded sum needs 64 bits).
__host__ __device__ constexpr int bucket_chunks(int n) {
    return static_cast<int>((static_cast<long long>(n) + kChunkPoints - 1) / kChunkPoints);
}

size_t bucket_smem_bytes(int nbins, bool scatter) {
    return ((static_cast<size_t>(nbins) * 2 + 15) & ~static_cast<size_t>(15)) + (scatter ? kChunkPoints * 4 : 0);
}

// COUNT: hist[bin] += points. SCATTER: order[pos] = point id, ocode[pos] = its
// code, pos counted down from the end of the bin (hist is consumed).
template <bool SCATTER>
__global__ void __launch_bounds__(kChunkThreads, 1)
    lsh_bucket_kernel(const uint32_t* __restrict__ codes, int n, int shift, int nbins, const int* __restrict__ start,
                      int* __restrict__ hist, int* __restrict__ order, uint32_t* __restrict__ ocode) {
    extern __shared__ __align__(16) uint32_t s_words[];
    uint16_t* s_cnt = reinterpret_cast<uint16_t*>(s_words);  // [nbins]: points of the chunk, then their leader
    int* s_base = reinterpret_cast<int*>(reinterpret_cast<char*>(s_words) + ((nbins * 2 + 15) & ~15));
    const size_t t = blockIdx.y;
    codes += t * n;
    hist += t * nbins;
    if constexpr (SCATTER) {
        start += t * (nbins + 1);
        order += t * n;
        ocode += t * n;
    }
    const int tid = threadIdx.x;
    for (int i = tid; i < (nbins + 1) / 2; i += kChunkThreads) s_words[i] = 0;
    const int chunks = bucket_chunks(n);
    for (int c = blockIdx.x; c < chunks; c += gridDim.x) {
        __syncthreads();  // counters are zero
        uint32_t code[kChunkPer];
        int rank[kChunkPer];
        #pragma unroll
        for (int j = 0; j < kChunkPer; ++j) {
            const long long i = static_cast<long long>(c) * kChunkPoints + j * kChunkThreads + tid;
            rank[j] = -1;
            code[j] = i < n ? codes[i] : 0u;
            if (i < n) rank[j] = 0;
        }
        #pragma unroll
        for (int j = 0; j < kChunkPer; ++j) {
            if (rank[j] < 0) continue;
            const uint32_t bin = code[j] >> shift, half = 16 * (bin & 1u);
            rank[j] = static_cast<int>((atomicAdd(&s_words[bin >> 1], 1u << half) >> half) & 0xffffu);
        }
        __syncthreads();
        #pragma unroll
        for (int j = 0; j < kChunkPer; ++j) {
            if (rank[j] != 0) continue;
            const uint32_t bin = code[j] >> shift;
            const int cnt = s_cnt[bin];
            if constexpr (SCATTER) {
                s_base[j * kChunkThreads + tid] = start[bin] + atomicSub(&hist[bin], cnt) - cnt;
                s_cnt[bin] = static_cast<uint16_t>(j * kChunkThreads + tid);
            } else {
                atomicAdd(&hist[bin], cnt);
            }
        }
        __syncthreads();
        if constexpr (SCATTER) {
            #pragma unroll
            for (int j = 0; j < kChunkPer; ++j) {
                if (rank[j] < 0) continue;
                const int pos = s_base[s_cnt[code[j] >> shift]] + rank[j];
                order[pos] = c * kChunkPoints + j * kChunkThreads + tid;
                ocode[pos] = code[j];
            }
            __syncthreads();
        }
        #pragma unroll
        for (int j = 0; j < kChunkPer; ++j)
            if (rank[j] >= 0) s_cnt[code[j] >> shift] = 0;
    }
}

// Exclusive scan of hist[t][0..nbins) into start[t][0..nbins]: a block per 1,024
// bins, which sums the bins before its own itself (at most 256 KB from L2).
constexpr int kScanBinsThreads = 256;
__global__ void __launch_bounds__(kScanBinsThreads)
    lsh_scan_bins_kernel(const int* __restrict__ hist, int nbins, int n, int* __restrict__ start) {
    __shared__ int warp_sums[kScanBinsThreads / 32];
    __shared__ int warp_before[kScanBinsThreads / 32];
    const int* h = hist + static_cast<size_t>(blockIdx.y) * nbins;
    int* st = start + static_cast<size_t>(blockIdx.y) * (nbins + 1);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int before = 0;  // blocks past the first exist only when nbins is a multiple of 1,024
    #pragma unroll 8
    for (int i = tid; i < static_cast<int>(blockIdx.x) * kScanBinsThreads; i += kScanBinsThreads) {
        const int4 v = reinterpret_cast<const int4*>(h)[i];
        before += v.x + v.y + v.z + v.w;
    }
    const int b0 = (blockIdx.x * kScanBinsThreads + tid) * 4;
    int v[4], local = 0;
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
        v[e] = b0 + e < nbins ? h[b0 + e] : 0;
        local += v[e];
    }
    before = __reduce_add_sync(0xffffffffu, before);
    int incl = local;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) {
        warp_sums[w] = incl;
        warp_before[w] = before;
    }
    __syncthreads();
    int run = incl - local;
    #pragma unroll
    for (int k = 0; k < kScanBinsThreads / 32; ++k) run += warp_before[k] + (k < w ? warp_sums[k] : 0);
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (b0 + e < nbins) st[b0 + e] = run;
        run += v[e];
    }
    if (blockIdx.x == 0 && tid == 0) st[nbins] = n;
}

// ---------------------------------------------------------- candidate scan
__device__ __forceinline__ bool lex_lt(int da, int ia, int db, int ib) { return da < db || (da == db && ia < ib); }

__device__ __forceinline__ void push_dedup(int d, int i, int& d1, int& i1, int& d2, int& i2) {
    if (i < 0 || i == i1 || i == i2) return;
    if (i1 < 0 || lex_lt(d, i, d1, i1)) {
        d2 = d1; i2 = i1;
        d1 = d; i1 = i;
    } else if (i2 < 0 || lex_lt(d, i, d2, i2)) {
        d2 = d; i2 = i;
    }
}

// NW warps per query. The query's probed buckets (L x P entries: table and
// code) are laid out in shared memory as runs of 32 positions ("chunks"), and
// every warp walks its equal share of the chunks: the ids (and, when a group
// holds several codes, the codes) of a chunk are one coalesced 128-byte load
// each, the next chunk's fetched while the current one is used. Members whose
// full code matches are appended to the warp's queue, and every 32 of them are
// scored together: 8 lanes fetch one row with coalesced 16-byte loads (8 loads,
// 32 rows in flight per warp), each lane sums b.b - 2 q.b over its 16 bytes
// by dp4a (|q - b|^2 = |q|^2 + that, exact integers), and 7 shuffles leave one
// row's distance in each lane. Every lane keeps a lexicographic (distance,
// index) top-2 of its rows; the lists are merged at the end, and a base row
// found in several tables (or probes) is compared each time but enters a list
// once.
//
// What bounds it: the random 128-byte rows of the candidates (L2 and DRAM).
// Candidates per query vary by a factor of 20 (8,788 to 163,868 at 1M rows, 8
// tables of 16 bits, 16 probes), so with one warp per query the last warps ran
// alone (70% of the SM cycles active), and the scoring took ~3x the
// instructions (byte differences, 3 shuffles per 4 rows, chunks of short
// buckets scored half empty). scan_warps has the rule for NW. Measured: that
// search 13.4 -> 3.2 ms (25-30 GB of candidate rows and ids: 8 TB/s, part of it
// from L2), the learned-hash match of 4,096 queries and 8 probes 4.87 -> 1.26 ms.
constexpr int kScanThreads = 256;
constexpr int kScanWarps = kScanThreads / 32;

struct ScanEntry {
    int pos, end;   // positions of the bucket in its table's order
    uint32_t code;
    int chunk0;     // first chunk of the entry among the query's chunks
};

__host__ __device__ constexpr size_t scan_smem_bytes(int entries, int nw) {
    return static_cast<size_t>(kScanWarps / nw) * (entries + 1) * sizeof(ScanEntry);
}

struct ScanTop2 {
    int d1 = INT_MAX, i1 = -1, d2 = INT_MAX, i2 = -1;
    __device__ __forceinline__ void push(int d, int i) { push_dedup(d, i, d1, i1, d2, i2); }
    __device__ __forceinline__ void merge_xor(int o) {
        const int od1 = __shfl_xor_sync(0xffffffffu, d1, o), oi1 = __shfl_xor_sync(0xffffffffu, i1, o);
        const int od2 = __shfl_xor_sync(0xffffffffu, d2, o), oi2 = __shfl_xor_sync(0xffffffffu, i2, o);
        push(od1, oi1);
        push(od2, oi2);
    }
};

// Scores the first 32 ids of a warp's queue (-1: none) against the query row
// chunk qv of lane part `lane & 7`, |q|^2 = qn.
__device__ __forceinline__ void score32(const uint8_t* __restrict__ r, const int* queue, const uint4& qv, int qn,
                                        int lane, ScanTop2& top) {
    const int sub = lane >> 3, part = lane & 7;  // rows 8 sub .. 8 sub + 7 of the queue, 16-byte chunk of the row
    const int4 ida = reinterpret_cast<const int4*>(queue)[2 * sub], idb = reinterpret_cast<const int4*>(queue)[2 * sub + 1];
    const int ids[8] = {ida.x, ida.y, ida.z, ida.w, idb.x, idb.y, idb.z, idb.w};
    uint4 v[8];
    #pragma unroll
    for (int j = 0; j < 8; ++j)
        v[j] = __ldg(reinterpret_cast<const uint4*>(r + static_cast<size_t>(max(ids[j], 0)) * 128) + part);
    int d[8];
    #pragma unroll
    for (int j = 0; j < 8; ++j) {
        uint32_t bb = __dp4a(v[j].x, v[j].x, 0u), qb = __dp4a(qv.x, v[j].x, 0u);
        bb = __dp4a(v[j].y, v[j].y, bb);
        qb = __dp4a(qv.y, v[j].y, qb);
        bb = __dp4a(v[j].z, v[j].z, bb);
        qb = __dp4a(qv.z, v[j].z, qb);
        bb = __dp4a(v[j].w, v[j].w, bb);
        qb = __dp4a(qv.w, v[j].w, qb);
        d[j] = static_cast<int>(bb) - 2 * static_cast<int>(qb);
    }
    // Sum over the 8 lanes of a row, halving the rows a lane holds each time.
    const bool h1 = part & 1, h2 = part & 2, h4 = part & 4;
    #pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int give = h1 ? d[j] : d[j + 4], keep = h1 ? d[j + 4] : d[j];
        d[j] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
    }
    #pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int give = h2 ? d[j] : d[j + 2], keep = h2 ? d[j + 2] : d[j];
        d[j] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
    const int give = h4 ? d[0] : d[1], keep = h4 ? d[1] : d[0];
    const int dist = qn + keep + __shfl_xor_sync(0xffffffffu, give, 4);
    const int id = queue[8 * sub + (h1 ? 4 : 0) + (h2 ? 2 : 0) + (h4 ? 1 : 0)];
    if (dist <= top.d2) top.push(dist, id);
}

template <int NW>
__global__ void __launch_bounds__(kScanThreads, 3) lsh_scan_kernel(
    const uint8_t* __restrict__ q, const uint8_t* __restrict__ r, int q_n, int r_n, int L, int probes, int shift,
    int nbins, const uint32_t* __restrict__ qcodes, const int* __restrict__ start, const int* __restrict__ order,
    const uint32_t* __restrict__ ocode, float thr, int ratio, float dscale, uint32_t* __restrict__ matches,
    uint32_t* __restrict__ counts, int32_t* __restrict__ nn_idx, float* __restrict__ nn_dist) {
    static_assert(NW == 1 || NW == kScanWarps, "a query is a warp's or a block's");
    extern __shared__ ScanEntry s_entries[];
    __shared__ __align__(16) int s_queue[kScanWarps][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = NW == 1 ? 0 : warp;  // warp of the query
    const int wq = NW == 1 ? blockIdx.x * kScanWarps + warp : blockIdx.x;
    if (NW == 1 && wq >= q_n) return;
    const int E = L * probes;
    ScanEntry* ent = s_entries + (NW == 1 ? warp * (E + 1) : 0);
    int* queue = s_queue[warp];
    auto sync = [] {
        if constexpr (NW == 1) __syncwarp();
        else __syncthreads();
    };
    const uint4 qv = __ldg(reinterpret_cast<const uint4*>(q + static_cast<size_t>(wq) * 128) + (lane & 7));
    int qn = static_cast<int>(__dp4a(qv.x, qv.x, __dp4a(qv.y, qv.y, __dp4a(qv.z, qv.z, __dp4a(qv.w, qv.w, 0u)))));
    qn += __shfl_xor_sync(0xffffffffu, qn, 1);
    qn += __shfl_xor_sync(0xffffffffu, qn, 2);
    qn += __shfl_xor_sync(0xffffffffu, qn, 4);
    const bool whole_bins = shift == 0;  // a group holds exactly one code

    // The entries: codes and bucket bounds, then their chunks' prefix sum.
    for (int i = w * 32 + lane; i < E; i += NW * 32) {
        const int t = i / probes;
        const uint32_t code = qcodes[static_cast<size_t>(i) * q_n + wq];
        const int* st = start + static_cast<size_t>(t) * (nbins + 1) + (code >> shift);
        ent[i].code = code;
        ent[i].pos = st[0];
        ent[i].end = st[1];
    }
    sync();
    for (int i = w * 32 + lane; i < E; i += NW * 32) {
        // A repeated probe code (fewer distinct probes than requested) is skipped.
        bool repeated = false;
        for (int j = i - i % probes; j < i; ++j) repeated |= ent[j].code == ent[i].code;
        ent[i].chunk0 = repeated ? 0 : (ent[i].end - ent[i].pos + 31) >> 5;
    }
    sync();
    if (w == 0) {
        const int per = (E + 31) / 32;
        const int e0 = min(lane * per, E), e1 = min(e0 + per, E);
        int mine = 0;
        for (int i = e0; i < e1; ++i) mine += ent[i].chunk0;
        int incl = mine;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        int run = incl - mine;
        for (int i = e0; i < e1; ++i) {
            const int n = ent[i].chunk0;
            ent[i].chunk0 = run;
            run += n;
        }
        if (lane == 31) ent[E].chunk0 = incl;
    }
    sync();

    ScanTop2 top;
    uint32_t seen = 0;  // candidates compared (bucket members)
    const long long chunks = ent[E].chunk0;
    const int c0 = static_cast<int>(chunks * w / NW), c1 = static_cast<int>(chunks * (w + 1) / NW);
    if (c0 < c1) {
        int e = 0;  // the entry of chunk c0: the last one that starts at or before it and is not empty
        for (int lo = 0, hi = E - 1; lo <= hi;) {
            const int mid = (lo + hi) >> 1;
            if (ent[mid].chunk0 <= c0) {
                e = mid;
                lo = mid + 1;
            } else {
                hi = mid - 1;
            }
        }
        int nid = -1;
        uint32_t ncode = 0, ecode = 0;
        auto fetch = [&](int c) {  // ids and codes of chunk c (chunks come in order)
            while (c >= ent[e + 1].chunk0) ++e;
            const ScanEntry& x = ent[e];
            const int p = x.pos + ((c - x.chunk0) << 5) + lane;
            const size_t at = static_cast<size_t>(e / probes) * r_n + p;
            ecode = x.code;
            nid = -1;
            if (p < x.end) {
                nid = order[at];
                ncode = whole_bins ? ecode : ocode[at];
            }
        };
        fetch(c0);
        int held = 0;  // ids in the queue
        for (int c = c0; c < c1; ++c) {
            const int id = nid;
            const bool hit = id >= 0 && ncode == ecode;
            if (c + 1 < c1) fetch(c + 1);
            const uint32_t mask = __ballot_sync(0xffffffffu, hit);
            if (hit) queue[held + __popc(mask & ((1u << lane) - 1u))] = id;
            held += __popc(mask);
            seen += __popc(mask);
            __syncwarp();
            if (held >= 32) {
                score32(r, queue, qv, qn, lane, top);
                held -= 32;
                const int rest = queue[32 + lane];
                __syncwarp();
                if (lane < held) queue[lane] = rest;
                __syncwarp();
            }
        }
        if (held > 0) {
            if (lane >= held) queue[lane] = -1;
            __syncwarp();
            score32(r, queue, qv, qn, lane, top);
        }
    }
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) top.merge_xor(o);
    if constexpr (NW > 1) {
        __syncwarp();
        if (lane == 0) {
            queue[0] = top.d1;
            queue[1] = top.i1;
            queue[2] = top.d2;
            queue[3] = top.i2;
            queue[4] = static_cast<int>(seen);
        }
        __syncthreads();
        if (warp > 0) return;
        top = ScanTop2{};
        seen = 0;
        if (lane < NW) {
            top = ScanTop2{s_queue[lane][0], s_queue[lane][1], s_queue[lane][2], s_queue[lane][3]};
            seen = static_cast<uint32_t>(s_queue[lane][4]);
        }
        #pragma unroll
        for (int o = 1; o < NW; o <<= 1) {
            top.merge_xor(o);
            seen += __shfl_xor_sync(0xffffffffu, seen, o);
        }
    }
    if (lane == 0) {
        if (counts) counts[wq] = seen;
        const bool v1 = top.i1 >= 0, v2 = top.i2 >= 0;
        const float f1 = v1 ? static_cast<float>(top.d1) * dscale : FLT_MAX;
        const float f2 = v2 ? static_cast<float>(top.d2) * dscale : FLT_MAX;
        if (matches) {
            bool pass = v1;
            if (v1 && ratio) pass = (sqrtf(f1) / (v2 ? sqrtf(f2) : INFINITY)) < thr;
            matches[wq] = pass ? static_cast<uint32_t>(top.i1) : UINT32_MAX;
        }
        if (nn_idx) {
            nn_idx[2 * wq] = top.i1;
            nn_idx[2 * wq + 1] = top.i2;
        }
        if (nn_dist) {
            nn_dist[2 * wq] = f1;
            nn_dist[2 * wq + 1] = f2;
        }
    }
}

// Warps per query from the average number of candidates that evenly spread
// codes would give (real codes crowd: 4-30 times that). Measured, scan kernel
// with 1 | 8 warps, 1M rows, 16 bits: 4,096 queries, 1 table and probe
// (15 expected) 44 | 52 us, 1 table x 4 probes (61) 116 | 89, 4 x 1 (61)
// 415 | 211, 4 x 4 (244) 1240 | 578; 20,000 rows, 8 x 4 (10) 69 | 80. With 500
// queries a warp each leaves the chip idle: 20,000 rows, 1 x 1 (0.3) 8.5 | 12.7,
// 4 x 4 (5) 29 | 19. More than 64 entries a query take the block as well (up to
// 2,688 of 16 bytes at 42 tables x 64 probes: 8 queries' would not fit in
// shared memory).
int scan_warps(int q_n, int r_n, int L, int probes, int nbins) {
    const double expected = static_cast<double>(L) * probes * r_n / nbins;
    const bool block = L * probes > 64 || expected >= 16.0 || (q_n <= 1024 && expected >= 2.0);
    return block ? kScanWarps : 1;
}

}  // namespace

int lsh_planes_padded(int L, int k) { return ((L * k + 31) / 32) * 32; }

size_t lsh_hash_smem(int P) { return hash_smem_bytes(P); }

cudaError_t launch_lsh_hash(const CUtensorMap& xmap, const CUtensorMap& pmap, int n, int P, int L, int k,
                            uint32_t* codes, float* z, int* err, int num_sms, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    const size_t smem = hash_smem_bytes(P);
    cudaError_t e = cudaFuncSetAttribute(lsh_hash_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    uint32_t slot = 32;
    while (slot < static_cast<uint32_t>(P)) slot <<= 1;
    const int nbuf = slot <= 128 ? 4 : 2;  // 512 TMEM columns
    const int tiles = (n + 127) / 128;
    const int grid = tiles < num_sms ? tiles : num_sms;
    lsh_hash_kernel<<<grid, kHThreads, smem, stream>>>(xmap, pmap, n, P, L, k, nbuf, slot, codes, z, err);
    return cudaGetLastError();
}

cudaError_t launch_lsh_buckets(const uint32_t* codes, int n, int L, int shift, int nbins, int* hist, int* start,
                               int* order, uint32_t* ocode, int num_sms, cudaStream_t stream) {
    cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(int) * static_cast<size_t>(L) * nbins, stream);
    if (e != cudaSuccess) return e;
    if (n <= 0) {
        e = cudaMemsetAsync(start, 0, sizeof(int) * static_cast<size_t>(L) * (nbins + 1), stream);
        return e;
    }
    const size_t smem_c = bucket_smem_bytes(nbins, false), smem_s = bucket_smem_bytes(nbins, true);
    e = cudaFuncSetAttribute(lsh_bucket_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem_c));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(lsh_bucket_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem_s));
    if (e != cudaSuccess) return e;
    const int chunks = bucket_chunks(n);
    const dim3 grid(std::min(chunks, num_sms), L);
    lsh_bucket_kernel<false><<<grid, kChunkThreads, smem_c, stream>>>(codes, n, shift, nbins, nullptr, hist, nullptr,
                                                                      nullptr);
    lsh_scan_bins_kernel<<<dim3((nbins + 4 * kScanBinsThreads - 1) / (4 * kScanBinsThreads), L), kScanBinsThreads, 0,
                           stream>>>(hist, nbins, n, start);
    lsh_bucket_kernel<true><<<grid, kChunkThreads, smem_s, stream>>>(codes, n, shift, nbins, start, hist, order, ocode);
    return cudaGetLastError();
}

cudaError_t launch_lsh_scan(const uint8_t* q, const uint8_t* r, int q_n, int r_n, int L, int probes, int shift,
                            int nbins, const uint32_t* qcodes, const int* start, const int* order,
                            const uint32_t* ocode, float thr, int ratio, float dist_scale, uint32_t* matches,
                            uint32_t* counts, int32_t* nn_idx, float* nn_dist, cudaStream_t stream) {
    if (q_n <= 0) return cudaSuccess;
    const int entries = L * probes;
    const int nw = scan_warps(q_n, r_n, L, probes, nbins);
    const size_t smem = scan_smem_bytes(entries, nw);
    if (nw == 1)
        lsh_scan_kernel<1><<<(q_n + kScanWarps - 1) / kScanWarps, kScanThreads, smem, stream>>>(
            q, r, q_n, r_n, L, probes, shift, nbins, qcodes, start, order, ocode, thr, ratio, dist_scale, matches,
            counts, nn_idx, nn_dist);
    else
        lsh_scan_kernel<kScanWarps><<<q_n, kScanThreads, smem, stream>>>(
            q, r, q_n, r_n, L, probes, shift, nbins, qcodes, start, order, ocode, thr, ratio, dist_scale, matches,
            counts, nn_idx, nn_dist);
    return cudaGetLastError();
}

}  // namespace sift
