// Epilogue building blocks shared by the exact-search kernels: per-thread
// running top-2 of one query row and the pruned scan of 32 accumulator
// columns (see exact2nn.cu for the pruning argument).
#pragma once
#include <climits>
#include <cstdint>

namespace sift {
namespace {

__device__ __forceinline__ int max8(const uint32_t* v) {
    int m = __vimax3_s32(static_cast<int>(v[0]), static_cast<int>(v[1]), static_cast<int>(v[2]));
    m = __vimax3_s32(m, static_cast<int>(v[3]), static_cast<int>(v[4]));
    m = __vimax3_s32(m, static_cast<int>(v[5]), static_cast<int>(v[6]));
    return max(m, static_cast<int>(v[7]));
}

// Per-thread running top-2 of one query row over base rows visited in
// increasing index order (strict '<' keeps the lower index on ties).
struct Top2 {
    int k1, i1, k2, i2;
    int thr;  // prune bound: rows with key > thr cannot enter the final top-2
};

__device__ __forceinline__ void top2_update(Top2& s, int key, int idx) {
    if (key < s.k2) {
        if (key < s.k1) {
            s.k2 = s.k1; s.i2 = s.i1;
            s.k1 = key; s.i1 = idx;
        } else {
            s.k2 = key; s.i2 = idx;
        }
        s.thr = min(s.thr, s.k2 - 1);
    }
}

// One group of 32 consecutive base rows [row0, row0 + 32) for this thread's
// query row; v[c] = q.b(row0 + c). nrm points at the group's 32 norms in the
// shared-memory record, gm8 at its four 8-row minima. Each 8-row subgroup is
// bounded from below by gm8[k] - 2 max(v[8k..8k+8)) (no key of its rows is
// smaller), so a subgroup whose bound exceeds the thread's threshold holds no
// candidate; the four bounds are tested with one vote. A passing subgroup
// forms its 8 exact keys and updates the top-2 only when their minimum is
// within the threshold (a key above it cannot reach the final top-2: the
// threshold never exceeds the final second-best key).
__device__ __forceinline__ void scan_group(const uint32_t (&v)[32], int row0, const int32_t* nrm, const int32_t* gm8,
                                           Top2& s) {
    int mx[4];
    #pragma unroll
    for (int k = 0; k < 4; ++k) mx[k] = max8(v + 8 * k);
    const int4 g8 = *reinterpret_cast<const int4*>(gm8);
    const int bnd[4] = {g8.x - 2 * mx[0], g8.y - 2 * mx[1], g8.z - 2 * mx[2], g8.w - 2 * mx[3]};
    const int bmin = min(__vimin3_s32(bnd[0], bnd[1], bnd[2]), bnd[3]);
    if (__any_sync(0xffffffffu, bmin <= s.thr)) {
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool ps = bnd[k] <= s.thr;
            if (__any_sync(0xffffffffu, ps)) {
                if (ps) {
                    const int4 na = *reinterpret_cast<const int4*>(nrm + 8 * k);
                    const int4 nb = *reinterpret_cast<const int4*>(nrm + 8 * k + 4);
                    const int nr[8] = {na.x, na.y, na.z, na.w, nb.x, nb.y, nb.z, nb.w};
                    int key[8];
                    #pragma unroll
                    for (int e = 0; e < 8; ++e)
                        key[e] = nr[e] - 2 * static_cast<int>(v[8 * k + e]);
                    // Exact keys first; the (rare) updates only when one can enter.
                    int mk = __vimin3_s32(key[0], key[1], key[2]);
                    mk = __vimin3_s32(mk, key[3], key[4]);
                    mk = __vimin3_s32(mk, key[5], key[6]);
                    mk = min(mk, key[7]);
                    if (mk <= s.thr) {
                        const int base = row0 + 8 * k;
                        #pragma unroll
                        for (int e = 0; e < 8; ++e) top2_update(s, key[e], base + e);
                    }
                }
            }
        }
    }
}

// Accumulator kinds of bound16 / exact8.
enum AccKind : int {
    kAccS32 = 0,    // s32 dot products (u8 kernel)
    kAccF32Int = 1, // f32 accumulators holding integer dot products / dscale (FP16 kernel), float norms
    kAccFloat = 2,  // f32 dot products of general floats (float keys, float norms)
};

// ---- packed top-2 (batches and small searches, whose thresholds stay loose)
// For squared distances of u8 rows the key |b|^2 - 2 q.b lies in
// [-|q|^2, |b|^2], i.e. within +/- 8,323,200 < 2^23, so y = -key and the column
// of the base row within its tile fit one int32:
//     w = 128 y + (127 - col) = 256 q.b + K[col],   K[col] = 127 - col - 128 |b|^2,
// whose order is the (key, index) order of the tile, and which one shift-add per
// element forms from the accumulator (modulo 2^32; the result fits). The top-2
// of a tile is then a max / min network without votes, branches or index
// registers: 2.5 operations per element, and every value is exact, so the test
// that skips a chunk (its largest w against the running second) has no slack
// from the spread of the norms. At 500-8,000 base rows per problem a warp of 32
// queries finds something new in more than half of its 16-row chunks, and the
// scan with 8-row bounds and serial updates took ~4,800 cycles per unit there.
// Measured: 512 image pairs (plan replay) 2,276 -> 1,118 us, mutual matching of
// 128 pairs 1,175 -> 566 us.
// The first kPackedDenseTiles tiles of a base set (2,048 rows, where 60-100% of
// the chunks hold something new for some of the 32 queries) run the network with
// no test at all, so that the chunks overlap freely; later tiles skip a chunk by
// a vote on its largest w. 512 pairs of 500-8,000 rows: always testing 1,251 us,
// never 1,168, from tile 8 / 16 / 28 on 1,139 / 1,117 / 1,117; 64 pairs of
// 7,000-8,000 rows: 863, 962, 848 / 843 / 855.
// The FP16 kernel runs it for the first kPackedFirstUnits units of a worker, whose
// bounds are loose (they took 2-5 times a later unit's 1,250 cycles): 2,000 x 100,000
// 94 -> 89 us per call, 2,561 x 500,003 304.6 -> 299.6, 5,000 x 300,000 311 -> 301,
// 10,000 x 1,000,000 equal within 0.3%; 4, 6, 16 and 32 units: 301.5, 300, 304.5, 322
// at 2,561 x 500,003. The u8 kernel's steady state lost more to the added code
// (10,000 x 1,000,000 1,167 -> 1,187-1,214) than its first units gave.
constexpr int kPackedFirstUnits = 8;
constexpr int kPackedMaxKey = 1 << 23;
constexpr int kPackedNone = INT_MIN;  // w of a padding row: below every floor

// A value below every w of rows with key <= thr, and not below any other row's.
__device__ __forceinline__ int packed_floor(int thr) { return -(min(thr, kPackedMaxKey) * 128) - 1; }

// Two largest of a[0..4) (no order among the rest).
__device__ __forceinline__ void top2_of4(const int* a, int& hi, int& lo) {
    const int h0 = max(a[0], a[1]), l0 = min(a[0], a[1]);
    const int h1 = max(a[2], a[3]), l1 = min(a[2], a[3]);
    hi = max(h0, h1);
    lo = __vimax3_s32(min(h0, h1), l0, l1);
}
// {hi, lo} = two largest of {hi, lo, h, l} (hi >= lo, h >= l).
__device__ __forceinline__ void top2_join(int& hi, int& lo, int h, int l) {
    lo = __vimax3_s32(min(hi, h), lo, l);
    hi = max(hi, h);
}

// w of one accumulator. FLOAT (FP16 rows of u8 values): acc and the record's norm k
// are floats, integers below 2^23 once multiplied by dscale: adding 2^23 leaves the
// integer in the low bits of the sum, and the exponents' share of w, (256 - 128) x
// 0x4B000000, is 2^31 (modulo 2^32). With the norms 0 of plain dot products w is
// 256 q.b + 127 - col < 2^31.
template <bool FLOAT>
__device__ __forceinline__ int packed_w(uint32_t acc, int32_t k, int col, float dscale) {
    if constexpr (FLOAT) {
        const uint32_t a = __float_as_uint(fmaf(__uint_as_float(acc), dscale, 8388608.0f));
        const uint32_t n = __float_as_uint(fmaf(__int_as_float(k), dscale, 8388608.0f));
        return static_cast<int>((a << 8) - (n << 7) + (0x80000000u + static_cast<uint32_t>(127 - col)));
    } else {
        return static_cast<int>((acc << 8) + static_cast<uint32_t>(k));
    }
}

// Rows [0, 16) of the chunk that starts at tile column c0: accumulators v, K (FLOAT:
// norms) at k (16-byte aligned), nv valid rows in the tile; m1 >= m2: the running two
// largest w. DENSE: the network at once; else only where some lane's largest w
// passes its second.
template <bool DENSE, bool FLOAT = false>
__device__ __forceinline__ void packed16(const uint32_t (&v)[16], int c0, int nv, const int32_t* k, int& m1,
                                         int& m2, float dscale = 0.0f) {
    int w[16];
    #pragma unroll
    for (int g = 0; g < 4; ++g) {
        const int4 kv = *reinterpret_cast<const int4*>(k + 4 * g);
        w[4 * g] = packed_w<FLOAT>(v[4 * g], kv.x, c0 + 4 * g, dscale);
        w[4 * g + 1] = packed_w<FLOAT>(v[4 * g + 1], kv.y, c0 + 4 * g + 1, dscale);
        w[4 * g + 2] = packed_w<FLOAT>(v[4 * g + 2], kv.z, c0 + 4 * g + 2, dscale);
        w[4 * g + 3] = packed_w<FLOAT>(v[4 * g + 3], kv.w, c0 + 4 * g + 3, dscale);
    }
    if (c0 + 16 > nv) {  // the last tile of a base set: rows past it (any values) never count
        #pragma unroll
        for (int e = 0; e < 16; ++e)
            if (c0 + e >= nv) w[e] = kPackedNone;
    }
    auto network = [&] {
        int hi, lo, h, l;
        top2_of4(w, hi, lo);
        #pragma unroll
        for (int g = 1; g < 4; ++g) {
            top2_of4(w + 4 * g, h, l);
            top2_join(hi, lo, h, l);
        }
        top2_join(m1, m2, hi, lo);
    };
    if constexpr (DENSE) {
        network();
    } else {
        const int mx = max(max8(reinterpret_cast<const uint32_t*>(w)), max8(reinterpret_cast<const uint32_t*>(w) + 8));
        if (__any_sync(0xffffffffu, mx > m2)) network();
    }
}

// Adds the two largest w of a tile whose rows start at row0 to the running
// top-2 (only those above the tile's floor are new).
__device__ __forceinline__ void packed_merge(int m1, int m2, int floor, int row0, Top2& s) {
    if (m1 > floor) {
        top2_update(s, -(m1 >> 7), row0 + 127 - (m1 & 127));
        if (m2 > floor) top2_update(s, -(m2 >> 7), row0 + 127 - (m2 & 127));
    }
}

// The pruned scan of a TMEM slot in two passes, so that an epilogue can bound
// every 8-row subgroup with no vote and no branch and form exact keys only
// where a bound passes.
//
// bound16: the pass bits of the chunk's two 8-row subgroups (bit k set when
// subgroup k's lower bound, the 8-row minimum gm8[k] minus twice the largest
// q.b of its rows, is within thr; the same bound as scan_group). gm8: the two
// 8-row minima (8-byte aligned). kAccF32Int: minima and bounds are floats in
// the units of the accumulators, exact, and thrf is thr in those units.
template <int KIND>
__device__ __forceinline__ uint32_t bound16(const uint32_t (&v)[16], const int32_t* gm8, int thr, float thrf) {
    const int2 g8 = *reinterpret_cast<const int2*>(gm8);
    uint32_t bits = 0;
    #pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int g = k ? g8.y : g8.x;
        bool pass;
        if constexpr (KIND == kAccFloat) {
            float m = __uint_as_float(v[8 * k]);
            #pragma unroll
            for (int e = 1; e < 8; ++e) m = fmaxf(m, __uint_as_float(v[8 * k + e]));
            pass = float_key(fmaf(-2.0f, m, __int_as_float(g))) <= thr;
        } else if constexpr (KIND == kAccF32Int) {
            const float m = __uint_as_float(static_cast<uint32_t>(max8(v + 8 * k)));
            pass = fmaf(-2.0f, m, __int_as_float(g)) <= thrf;
        } else {
            pass = g - 2 * max8(v + 8 * k) <= thr;
        }
        bits |= (pass ? 1u : 0u) << k;
    }
    return bits;
}

// fold_bits16: the pass bits of a chunk's two 8-row subgroups in the fold
// variant, whose accumulators hold q.b - c and whose keys are r - 2 acc with
// residuals r >= -1: subgroup k may hold a key within thr only when its
// largest accumulator reaches vt = -floor((thr + 1) / 2).
__device__ __forceinline__ uint32_t fold_bits16(const uint32_t (&v)[16], int vt) {
    return (max8(v) >= vt ? 1u : 0u) | (max8(v + 8) >= vt ? 2u : 0u);
}

// exact8: the exact keys of one 8-row subgroup [row0, row0 + 8) (v: its
// accumulators, nrm: its 8 norms, 16-byte aligned); they update the running
// top-2 only when their minimum is within the thread's current threshold (a
// key above it cannot reach the final top-2).
template <int KIND>
__device__ __forceinline__ void exact8(const uint32_t (&v)[8], int row0, const int32_t* nrm, Top2& s,
                                       float dscale) {
    const int4 na = *reinterpret_cast<const int4*>(nrm);
    const int4 nb = *reinterpret_cast<const int4*>(nrm + 4);
    const int nr[8] = {na.x, na.y, na.z, na.w, nb.x, nb.y, nb.z, nb.w};
    int key[8];
    #pragma unroll
    for (int e = 0; e < 8; ++e) {
        if constexpr (KIND == kAccFloat)
            key[e] = float_key(fmaf(-2.0f, __uint_as_float(v[e]), __int_as_float(nr[e])));
        else if constexpr (KIND == kAccF32Int)
            key[e] = __float2int_rn(fmaf(-2.0f, __uint_as_float(v[e]), __int_as_float(nr[e])) * dscale);
        else
            key[e] = nr[e] - 2 * static_cast<int>(v[e]);
    }
    int mk = __vimin3_s32(key[0], key[1], key[2]);
    mk = __vimin3_s32(mk, key[3], key[4]);
    mk = __vimin3_s32(mk, key[5], key[6]);
    mk = min(mk, key[7]);
    if (mk <= s.thr) {
        #pragma unroll
        for (int e = 0; e < 8; ++e) top2_update(s, key[e], row0 + e);
    }
}

}  // namespace
}  // namespace sift
