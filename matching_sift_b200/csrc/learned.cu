// Learned-hash inference on sm_100a: both MLP layers on the tensor cores
// (tcgen05 kind::f16, BF16 operands, FP32 accumulators in TMEM), fused with
// the conversion of the u8 descriptors to BF16 and the packing of the output
// signs into bucket codes; plus query-directed probe generation.
//
// Per CTA (persistent over 128-row tiles), shared memory holds W1 (256 x 128)
// and W2 (32 x 256, rows >= k zero) for the whole launch, one BF16 input tile
// (128 x 128) and one BF16 hidden tile (128 x 256), all K-major with the
// 128-byte swizzle (the layout TMA writes for the weights; the epilogue warps
// write the activations in the same layout themselves).
//
// Warps: 0 = weight and input-tile TMA, TMEM allocation, MMA issue (one
//            thread); the u8 input tiles stream through a 2-stage ring,
//            loaded two tiles ahead;
//        1..16 = conversion and epilogue, four warps per TMEM lane quarter:
//            thread = tile row (TMEM lane), warp group g converts 32 columns of
//            the input row and applies layer 1's epilogue to hidden columns
//            [64 g, 64 g + 64); group i % 4 forms the codes of tile i.
// Two tiles are in flight, so that the epilogue warps never wait for the tensor
// cores; TMEM holds layer 1's accumulators of both, buffer i % 2 of 256 columns,
// and layer 2's 32 columns reuse the first ones of their tile's buffer once they
// are read. Per tile i (epilogue threads), while MMA1(i) has just completed:
//   convert x(i+1) -> x_s (free: MMA1(i) is done)
//   take layer 2's accumulators of tile i - 1
//   [x_ready]  MMA1(i+1): TMEM[256 ((i+1) % 2)] = x W1^T
//   epi1(i): h = bf16(relu(acc / 64 + b1)) -> h_s (free: MMA2(i-1) is done)
//   [h_ready]  MMA2(i): TMEM[256 (i % 2)], 32 columns = h W2^T
//   epi2(i-1): z = acc + b2 -> code bits (and z)
// Bound by shared memory (about 340 KB of operand reads and activation writes a
// tile, 2,650 cycles of 128 bytes, against 2,000 of MMAs) and by the chain MMA1 ->
// convert -> MMA1 over the one x_s buffer. 1M rows, 16 bits: 154 us with 8
// epilogue warps, MMA1 in line with them and a branch per output bit, 105 us now.
// Every wait is bounded (2 s) and reports through `err`.
#include <climits>
#include <cuda_bf16.h>
#include "exact2nn.cuh"
#include "learned.cuh"
#include "ptx.cuh"

namespace sift {
namespace {

constexpr int kLEpiWarps = 16;  // four per TMEM lane quarter
constexpr int kLThreads = 32 * (1 + kLEpiWarps);
constexpr int kXKBlock = 128 * 128;                     // bytes of one K block of a 128-row BF16 tile
constexpr int kW1Bytes = kMlpHidden * kMlpIn * 2;       // 64 KB
constexpr int kW2Bytes = kMlpOutRows * kMlpHidden * 2;  // 16 KB
constexpr int kXBytes = 128 * kMlpIn * 2;               // 32 KB
constexpr int kHBytes = 128 * kMlpHidden * 2;           // 64 KB
constexpr uint32_t kLTmemCols = 512;
constexpr int kXStages = 2;                             // u8 input tile ring
constexpr int kXTileBytes = 128 * kMlpIn;               // 16 KB

struct __align__(16) MlpCtl {
    uint64_t w_full, x_ready, h_ready, m1, m2, drain;
    uint64_t xfull[kXStages];
    uint32_t tmem_base;
    int abort_flag, no_abort;
    alignas(16) float b1[kMlpHidden];
    alignas(16) float b2[kMlpOutRows];
};

constexpr size_t kLSmemBytes = 1024 + kW1Bytes + kW2Bytes + kXBytes + kHBytes + kXStages * kXTileBytes + sizeof(MlpCtl);
static_assert(kLSmemBytes <= 227 * 1024, "MLP hash shared memory");

// Byte offset of the 16-byte chunk `ch` (0..7) of row r in a K block of a
// SW128 K-major tile (rows of 128 bytes, 8-row atoms).
__device__ __forceinline__ uint32_t sw128_off(int r, int ch) {
    return static_cast<uint32_t>(r * 128 + ((ch ^ (r & 7)) << 4));
}

__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Byte b of w as a float: 2^23 + byte built in the mantissa, minus 2^23 (exact).
template <int B>
__device__ __forceinline__ float byte_float(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u + B)) - 8388608.0f;
}

// 16-byte chunks 2 g and 2 g + 1 of row r of a u8 tile in shared memory (TMA,
// 128-byte swizzle; rows past the end of the input are zeros) -> BF16 in x_s.
__device__ __forceinline__ void convert_row(const uint8_t* u8_tile, int r, uint8_t* x_s, int g) {
    #pragma unroll
    for (int c = 2 * g; c < 2 * g + 2; ++c) {
        const uint4 v = *reinterpret_cast<const uint4*>(u8_tile + sw128_off(r, c));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        uint32_t o[8];
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
            o[2 * q] = bf16x2(byte_float<0>(w[q]), byte_float<1>(w[q]));
            o[2 * q + 1] = bf16x2(byte_float<2>(w[q]), byte_float<3>(w[q]));
        }
        // elements 16c .. 16c + 15: K block c / 4, chunks 2 (c % 4) and 2 (c % 4) + 1
        uint8_t* blk = x_s + (c >> 2) * kXKBlock;
        const int ch = 2 * (c & 3);
        *reinterpret_cast<uint4*>(blk + sw128_off(r, ch)) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(blk + sw128_off(r, ch + 1)) = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

__global__ void __launch_bounds__(kLThreads, 1)
    mlp_hash_kernel(const __grid_constant__ CUtensorMap xmap, int n, const __grid_constant__ CUtensorMap w1map,
                    const __grid_constant__ CUtensorMap w2map, const float* __restrict__ b1,
                    const float* __restrict__ b2, int k, uint32_t* __restrict__ codes, float* __restrict__ zout,
                    int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = ptx::smem_u32(smem_raw);
    uint8_t* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
    uint8_t* w1_s = smem;
    uint8_t* w2_s = w1_s + kW1Bytes;
    uint8_t* x_s = w2_s + kW2Bytes;
    uint8_t* h_s = x_s + kXBytes;
    uint8_t* xr_s = h_s + kHBytes;  // u8 tile ring
    MlpCtl* ctl = reinterpret_cast<MlpCtl*>(xr_s + kXStages * kXTileBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = (n + 127) / 128;
    const int bx = static_cast<int>(blockIdx.x), gx = static_cast<int>(gridDim.x);
    const int my_tiles = bx < tiles ? (tiles - 1 - bx) / gx + 1 : 0;

    const uint32_t bar_w = ptx::smem_u32(&ctl->w_full), bar_x = ptx::smem_u32(&ctl->x_ready);
    const uint32_t bar_h = ptx::smem_u32(&ctl->h_ready), bar_m1 = ptx::smem_u32(&ctl->m1);
    const uint32_t bar_m2 = ptx::smem_u32(&ctl->m2), bar_drain = ptx::smem_u32(&ctl->drain);
    if (threadIdx.x == 0) {
        ptx::mbar_init(bar_w, 1);
        ptx::mbar_init(bar_x, 32 * kLEpiWarps);
        ptx::mbar_init(bar_h, 32 * kLEpiWarps);
        ptx::mbar_init(bar_m1, 1);
        ptx::mbar_init(bar_m2, 1);
        ptx::mbar_init(bar_drain, 1);
        for (int s = 0; s < kXStages; ++s) ptx::mbar_init(ptx::smem_u32(&ctl->xfull[s]), 1);
        ctl->abort_flag = 0;
        ctl->no_abort = 0;
        ptx::fence_mbar_init();
    }
    for (int j = threadIdx.x; j < kMlpHidden; j += kLThreads) ctl->b1[j] = b1[j];
    for (int j = threadIdx.x; j < kMlpOutRows; j += kLThreads) ctl->b2[j] = j < k ? b2[j] : 0.0f;
    if (warp == 0) {
        ptx::tmem_alloc(ptx::smem_u32(&ctl->tmem_base), kLTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    volatile int* abort_flag = &ctl->abort_flag;
    volatile int* never = &ctl->no_abort;
    const uint32_t w1_a = ptx::smem_u32(w1_s), w2_a = ptx::smem_u32(w2_s);
    const uint32_t x_a = ptx::smem_u32(x_s), h_a = ptx::smem_u32(h_s);
    const uint32_t xr_a = ptx::smem_u32(xr_s), bar_xf = ptx::smem_u32(&ctl->xfull[0]);

    if (warp == 0) {
        if (lane == 0 && my_tiles > 0) {
            ptx::tma_prefetch_desc(&w1map);
            ptx::tma_prefetch_desc(&w2map);
            ptx::tma_prefetch_desc(&xmap);
            int issued = 0;  // input tiles whose TMA load has been issued
            for (; issued < kXStages && issued < my_tiles; ++issued) {
                ptx::mbar_arrive_expect_tx(bar_xf + 8 * issued, kXTileBytes);
                ptx::tma_load_2d(xr_a + issued * kXTileBytes, &xmap, 0, (bx + issued * gx) * 128, bar_xf + 8 * issued);
            }
            ptx::mbar_arrive_expect_tx(bar_w, kW1Bytes + kW2Bytes);
            for (int kb = 0; kb < 2; ++kb) ptx::tma_load_2d(w1_a + kb * (kMlpHidden * 128), &w1map, kb * 64, 0, bar_w);
            for (int kb = 0; kb < 4; ++kb) ptx::tma_load_2d(w2_a + kb * (kMlpOutRows * 128), &w2map, kb * 64, 0, bar_w);
            // layer 1: M = 128, N = 256, K = 16 per MMA; layer 2: M = 128, N = 32
            constexpr uint32_t idesc1 = ptx::idesc_make(1 /*F32*/, 1 /*BF16*/, 1 /*BF16*/, 128, kMlpHidden);
            constexpr uint32_t idesc2 = ptx::idesc_make(1 /*F32*/, 1 /*BF16*/, 1 /*BF16*/, 128, kMlpOutRows);
            const bool ok = ptx::mbar_wait(bar_w, 0, abort_flag, err, kErrWaitMmaFull);
            auto layer2 = [&](int i) -> bool {
                if (!ptx::mbar_wait(bar_h, i & 1, abort_flag, err, kErrWaitMmaTmem)) return false;
                ptx::tc_fence_after();
                #pragma unroll
                for (int kb = 0; kb < 4; ++kb) {
                    #pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        ptx::mma_f16(tmem + (i & 1) * kMlpHidden, ptx::sdesc_sw128(h_a + kb * kXKBlock + kk * 32),
                                     ptx::sdesc_sw128(w2_a + kb * (kMlpOutRows * 128) + kk * 32), idesc2,
                                     (kb | kk) ? 1u : 0u);
                }
                ptx::tc_commit(bar_m2);
                return true;
            };
            bool run = ok;
            for (int i = 0; i < my_tiles && run; ++i) {
                if (!ptx::mbar_wait(bar_x, i & 1, abort_flag, err, kErrWaitMmaFull)) {
                    run = false;
                    break;
                }
                ptx::tc_fence_after();
                #pragma unroll
                for (int kb = 0; kb < 2; ++kb) {
                    #pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        ptx::mma_f16(tmem + (i & 1) * kMlpHidden, ptx::sdesc_sw128(x_a + kb * kXKBlock + kk * 32),
                                     ptx::sdesc_sw128(w1_a + kb * (kMlpHidden * 128) + kk * 32), idesc1,
                                     (kb | kk) ? 1u : 0u);
                }
                ptx::tc_commit(bar_m1);
                // Tile i's u8 stage was converted (x_ready): reuse it for tile i + 2.
                if (issued < my_tiles) {
                    const int st = issued % kXStages;
                    ptx::mbar_arrive_expect_tx(bar_xf + 8 * st, kXTileBytes);
                    ptx::tma_load_2d(xr_a + st * kXTileBytes, &xmap, 0, (bx + issued * gx) * 128, bar_xf + 8 * st);
                    ++issued;
                }
                if (i > 0) run = layer2(i - 1);
            }
            if (run) layer2(my_tiles - 1);
            if (!ok) ptx::mbar_wait(bar_w, 0, never, err, kErrWaitDrain);  // weights landed before exit
            // Input tiles in flight land before exit (the last kXStages issued).
            for (int t = (issued > kXStages ? issued - kXStages : 0); t < issued; ++t)
                ptx::mbar_wait(bar_xf + 8 * (t % kXStages), (t / kXStages) & 1, never, err, kErrWaitDrain);
            ptx::tc_commit(bar_drain);
            ptx::mbar_wait(bar_drain, 0, never, err, kErrWaitDrain);
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3;
        const int grp = (warp - 1) >> 2;    // input columns [32 grp, + 32), hidden columns [64 grp, + 64)
        const int r = quarter * 32 + lane;  // tile row = TMEM lane
        const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
        auto wait_all = [&](uint32_t bar, uint32_t parity) -> bool {
            const bool w = __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag, err, kErrWaitEpilogue));
            ptx::tc_fence_after();
            return w;
        };
        auto convert = [&](int i) -> bool {
            const int st = i % kXStages;
            const bool w = __all_sync(0xffffffffu, ptx::mbar_wait(bar_xf + 8 * st, (i / kXStages) & 1, abort_flag, err,
                                                                  kErrWaitEpilogue));
            if (w) convert_row(xr_s + st * kXTileBytes, r, x_s, grp);
            return w;
        };
        // Layer 2 of tile i: every warp waits for it (h_s and the TMEM buffer are
        // reused next); group i % 4 takes the accumulators, and forms the codes
        // once the next MMAs have been started.
        uint32_t v2[32];
        auto take2 = [&](int i) -> bool {
            if (!wait_all(bar_m2, i & 1)) return false;
            if ((i & 3) == grp) {
                ptx::tmem_ld32(tmem + lane_base + (i & 1) * kMlpHidden, v2);
                ptx::tmem_ld_wait(v2);
            }
            return true;
        };
        auto codes2 = [&](int i) {
            if ((i & 3) != grp) return;
            const int g = (bx + i * gx) * 128 + r;
            uint32_t code = 0;
            float z[32];
            #pragma unroll
            for (int j = 0; j < kMlpMaxBits; j += 4) {  // outputs past k are 0 + 0
                const float4 b = *reinterpret_cast<const float4*>(&ctl->b2[j]);
                z[j] = __uint_as_float(v2[j]) + b.x;
                z[j + 1] = __uint_as_float(v2[j + 1]) + b.y;
                z[j + 2] = __uint_as_float(v2[j + 2]) + b.z;
                z[j + 3] = __uint_as_float(v2[j + 3]) + b.w;
            }
            #pragma unroll
            for (int j = 0; j < kMlpMaxBits; ++j) code |= z[j] > 0.0f ? 1u << j : 0u;
            if (g < n) {
                codes[g] = code & (0xffffffffu >> (32 - k));
                if (zout) {
                    #pragma unroll
                    for (int j = 0; j < kMlpMaxBits; ++j)
                        if (j < k) zout[static_cast<size_t>(g) * k + j] = z[j];
                }
            }
        };
        bool ok = my_tiles > 0 && convert(0);
        if (ok) {
            ptx::fence_proxy_async();
            ptx::mbar_arrive(bar_x);
        }
        for (int i = 0; i < my_tiles && ok; ++i) {
            ok = wait_all(bar_m1, i & 1);
            if (ok && i + 1 < my_tiles) ok = convert(i + 1);
            if (ok && i > 0) ok = take2(i - 1);
            if (!ok) break;
            ptx::tc_fence_before();
            ptx::fence_proxy_async();
            if (i + 1 < my_tiles) ptx::mbar_arrive(bar_x);
            const uint32_t acc = tmem + lane_base + (i & 1) * kMlpHidden + 64 * grp;
            uint8_t* blk = h_s + grp * kXKBlock;
            #pragma unroll
            for (int m = 0; m < 2; ++m) {
                uint32_t v[32];
                ptx::tmem_ld32(acc + 32 * m, v);
                ptx::tmem_ld_wait(v);
                #pragma unroll
                for (int c8 = 0; c8 < 4; ++c8) {
                    uint32_t o[4];
                    #pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float4 bj = *reinterpret_cast<const float4*>(&ctl->b1[64 * grp + 32 * m + 8 * c8 + 4 * e]);
                        const uint32_t* a = v + 8 * c8 + 4 * e;
                        o[2 * e] = bf16x2(fmaxf(fmaf(__uint_as_float(a[0]), kMlpInScale, bj.x), 0.0f),
                                          fmaxf(fmaf(__uint_as_float(a[1]), kMlpInScale, bj.y), 0.0f));
                        o[2 * e + 1] = bf16x2(fmaxf(fmaf(__uint_as_float(a[2]), kMlpInScale, bj.z), 0.0f),
                                              fmaxf(fmaf(__uint_as_float(a[3]), kMlpInScale, bj.w), 0.0f));
                    }
                    *reinterpret_cast<uint4*>(blk + sw128_off(r, 4 * m + c8)) = make_uint4(o[0], o[1], o[2], o[3]);
                }
            }
            ptx::tc_fence_before();
            ptx::fence_proxy_async();
            ptx::mbar_arrive(bar_h);
            if (i > 0) codes2(i - 1);
        }
        if (ok && my_tiles > 0 && take2(my_tiles - 1)) {
            ptx::tc_fence_before();
            codes2(my_tiles - 1);
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, kLTmemCols);
    }
}

// Probe codes of every (table, query): the `flip` smallest-|z| bits, all
// their subsets ordered by summed |z| (ties by subset mask), the first
// n_probes applied. One warp per (table, query): lane j ranks |z_j| against
// the k magnitudes, lane s ranks subsets s and s + 32 against all 64 by
// shuffles, so there is no serial selection and no indexed local memory; a
// block holds 32 consecutive queries of one table and stages the codes in
// shared memory so that each probe's codes leave as one 128-byte store.
// Latency and issue bound (a few hundred instructions per query, 4 k bytes
// read). 4,096 queries, 8 tables of 16 bits, 16 probes: 8 launches of 225 us
// with one thread per query selecting probe after probe; now one launch, the
// whole index search 15.14 -> 13.39 ms.
constexpr int kProbeRows = 32;
constexpr int kProbeThreads = 256;

// The probes of a query with a NaN margin (weights or sums that are not finite):
// comparisons with it are all false, so counting gives several bits or subsets the
// same rank. One thread selects instead, bits by insertion in bit order and then, for
// each probe, the first subset left that none is lighter than, with the empty one
// (sum 0) first. Rare and slow (a few thousand steps); out: one code per kProbeRows + 1.
__device__ __noinline__ void probe_codes_unordered(const float* __restrict__ z, uint32_t code, int k, int flip,
                                                   int n_probes, uint32_t* out) {
    int bit[6];
    float mag[6];
    int m = 0;
    for (int j = 0; j < k; ++j) {
        const float a = fabsf(z[j]);
        int p;
        if (m < flip) p = m++;
        else if (flip > 0 && a < mag[flip - 1]) p = flip - 1;
        else continue;
        for (; p > 0 && mag[p - 1] > a; --p) {
            mag[p] = mag[p - 1];
            bit[p] = bit[p - 1];
        }
        mag[p] = a;
        bit[p] = j;
    }
    uint64_t taken = 0;
    for (int p = 0; p < n_probes; ++p) {
        int best = -1;
        float lightest = 0.0f;
        for (int s = 0; s < (1 << m); ++s) {
            if ((taken >> s) & 1u) continue;
            float sum = 0.0f;
            for (int b = 0; b < m; ++b)
                if ((s >> b) & 1) sum += mag[b];
            if (best < 0 || sum < lightest) {
                best = s;
                lightest = sum;
            }
        }
        uint32_t c = code;
        if (best >= 0) {
            taken |= 1ull << best;
            for (int b = 0; b < m; ++b)
                if ((best >> b) & 1) c ^= 1u << bit[b];
        }
        out[p * (kProbeRows + 1)] = c;
    }
}

__global__ void __launch_bounds__(kProbeThreads)
    probe_codes_kernel(const uint32_t* __restrict__ codes, const float* __restrict__ z, int n, int k, int flip,
                       int n_probes, uint32_t* __restrict__ out) {
    __shared__ uint32_t s_out[64][kProbeRows + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t t = blockIdx.y;
    const int row0 = blockIdx.x * kProbeRows;
    codes += t * n;
    z += t * n * k;
    out += t * n_probes * n;
    constexpr int kRows = kProbeRows / (kProbeThreads / 32);  // queries per warp
    float mags[kRows];
    #pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const int i = row0 + warp * kRows + r;
        mags[r] = i < n && lane < k ? fabsf(z[static_cast<size_t>(i) * k + lane]) : INFINITY;
    }
    #pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const int col = warp * kRows + r;
        if (row0 + col >= n) break;
        const uint32_t code = codes[row0 + col];
        const float a = mags[r];
        if (__any_sync(0xffffffffu, isnan(a))) {
            if (lane == 0)
                probe_codes_unordered(z + static_cast<size_t>(row0 + col) * k, code, k, flip, n_probes, &s_out[0][col]);
            continue;
        }
        int rank = 0;
        for (int j = 0; j < k; ++j) {
            const float b = __shfl_sync(0xffffffffu, a, j);
            rank += (b < a || (b == a && j < lane)) ? 1 : 0;
        }
        // Sums of the kept magnitudes in ascending rank, and the bits they flip.
        float s0 = 0.0f, s1 = 0.0f;
        uint32_t f0 = 0, f1 = 0;
        #pragma unroll
        for (int b = 0; b < 6; ++b) {
            if (b < flip) {
                const uint32_t who = __ballot_sync(0xffffffffu, lane < k && rank == b);
                const int src = who ? __ffs(who) - 1 : 0;
                const float m = __shfl_sync(0xffffffffu, a, src);
                const uint32_t bit = who ? 1u << src : 0u;
                if (b < 5) {
                    if ((lane >> b) & 1) {
                        s0 += m;
                        f0 |= bit;
                        s1 += m;
                        f1 |= bit;
                    }
                } else {  // subsets lane + 32
                    s1 += m;
                    f1 |= bit;
                }
            }
        }
        const int subsets = 1 << flip;
        if (lane >= subsets) s0 = INFINITY;
        if (lane + 32 >= subsets) s1 = INFINITY;
        int r0 = 0, r1 = 0;  // ranks by (sum, subset)
        #pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            const float u = __shfl_sync(0xffffffffu, s0, j), v = __shfl_sync(0xffffffffu, s1, j);
            r0 += (u < s0 || (u == s0 && j < lane)) ? 1 : 0;
            r0 += v < s0 ? 1 : 0;
            r1 += u <= s1 ? 1 : 0;
            r1 += (v < s1 || (v == s1 && j < lane)) ? 1 : 0;
        }
        // Past the subsets: the code again (skipped by the scan).
        for (int p = lane; p < n_probes; p += 32) s_out[p][col] = code;
        __syncwarp();
        if (lane < subsets && r0 < n_probes) s_out[r0][col] = code ^ f0;
        if (lane + 32 < subsets && r1 < n_probes) s_out[r1][col] = code ^ f1;
    }
    __syncthreads();
    if (row0 + lane < n)
        for (int p = warp; p < n_probes; p += kProbeThreads / 32)
            out[static_cast<size_t>(p) * n + row0 + lane] = s_out[p][lane];
}

}  // namespace

size_t mlp_hash_smem_bytes() { return kLSmemBytes; }

cudaError_t launch_mlp_hash(const CUtensorMap& xmap, int n, const CUtensorMap& w1map, const CUtensorMap& w2map,
                            const float* b1, const float* b2, int k, uint32_t* codes, float* z, int* err,
                            int num_sms, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(mlp_hash_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kLSmemBytes));
    if (e != cudaSuccess) return e;
    const int tiles = (n + 127) / 128;
    const int grid = tiles < num_sms ? tiles : num_sms;
    mlp_hash_kernel<<<grid, kLThreads, kLSmemBytes, stream>>>(xmap, n, w1map, w2map, b1, b2, k, codes, z, err);
    return cudaGetLastError();
}

cudaError_t launch_probe_codes(const uint32_t* codes, const float* z, int n, int tables, int k, int flip, int n_probes,
                               uint32_t* probe_codes, cudaStream_t stream) {
    if (n <= 0 || tables <= 0) return cudaSuccess;
    if (flip < 0 || flip > 6 || n_probes < 1 || n_probes > 64 || flip > k || k > kMlpMaxBits || tables > 65535)
        return cudaErrorInvalidValue;
    probe_codes_kernel<<<dim3((n + kProbeRows - 1) / kProbeRows, tables), kProbeThreads, 0, stream>>>(
        codes, z, n, k, flip, n_probes, probe_codes);
    return cudaGetLastError();
}

}  // namespace sift
