// Input conversion kernels: float / half descriptors -> u8 (with an exactness
// flag). Replaces the reference's float2half (src/knn_brute.cu:315-338), which
// converted every batch to FP16; here descriptors whose values are integers in
// [0, 255], or such integers times one common power of two (the reference's
// own benchmark divides SIFT1M's integer components by 512, src/test.cu:99-103),
// are packed once to u8, the format the tensor-core kernel consumes.
#include <algorithm>
#include <climits>
#include <cuda_fp16.h>
#include "exact2nn.cuh"
#include "launch.cuh"
#include "pack.cuh"

namespace sift {
namespace {

// v * mul (mul a power of two; the product is an integer in [0, 255]) as u8.
__device__ __forceinline__ uint32_t to_u8(float v, float mul) { return __float2uint_rz(v * mul) & 0xffu; }
__device__ __forceinline__ uint32_t pack4(float4 v, float mul) {
    return to_u8(v.x, mul) | (to_u8(v.y, mul) << 8) | (to_u8(v.z, mul) << 16) | (to_u8(v.w, mul) << 24);
}

// ---- survey of one value (launch_survey in pack.cuh)
// Returns v * 2^24 as an unsigned integer (exact unless kValueNotFixed), whose
// top byte is v itself when v is an integer in [0, 255].
__device__ __forceinline__ uint32_t survey_one(float v, uint32_t& flags, uint32_t& bits, float& mx) {
    const float a = fabsf(v), t = v * 16777216.0f;
    if (!(a <= 3.0e38f)) flags |= kValueNotFinite;
    mx = fmaxf(mx, a);
    // v in [0, 256): t < 2^32, exact; an integer t fits a uint32.
    const uint32_t u = __float2uint_rz(t);
    if (!(v >= 0.0f && v < 256.0f && __uint2float_rn(u) == t)) flags |= kValueNotFixed;
    bits |= u;
    return u;
}
// Two halves at once (w, as floats f): every finite half is a multiple of 2^-24,
// so f * 2^24 is an integer, below 2^32 for values in [0, 256); range, sign and
// finiteness follow from the largest magnitude and the OR of all words (a set
// sign bit is looked at again: it may be a negative zero).
__device__ __forceinline__ void survey_half2(uint32_t w, float2 f, uint32_t& bits, uint32_t& mx2, uint32_t& words) {
    mx2 = __vmaxu2(mx2, w & 0x7fff7fffu);
    words |= w;
    bits |= __float2uint_rz(f.x * 16777216.0f) | __float2uint_rz(f.y * 16777216.0f);
}
__device__ __forceinline__ bool negative_half2(uint32_t w) {
    return ((w & 0x8000u) && (w & 0x7fffu)) || ((w >> 31) && (w & 0x7fff0000u));
}
__device__ __forceinline__ float2 half2_floats(uint32_t w) {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
// The largest magnitude as a float, and the flags it decides.
__device__ __forceinline__ float half_max(uint32_t mx2, uint32_t& flags) {
    const uint32_t m = max(mx2 & 0xffffu, mx2 >> 16);
    if (m >= 0x5c00u) flags |= kValueNotFixed;  // 256 and above
    if (m >= 0x7c00u) flags |= kValueNotFinite;
    return m >= 0x7c00u ? 0.0f : __half2float(__ushort_as_half(static_cast<unsigned short>(m)));
}
// A block's findings (256 threads). They all meet at three addresses: reduced
// within the block first, and added only where they change what is there (the
// words only grow, so a stale read costs one atomic).
__device__ __forceinline__ void survey_flush(uint32_t flags, uint32_t bits, float mx, int* stats) {
    __shared__ uint32_t s_part[3][8];
    flags = __reduce_or_sync(0xffffffffu, flags);
    bits = __reduce_or_sync(0xffffffffu, bits);
    uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));  // mx >= 0: bits order like values
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        s_part[0][warp] = flags;
        s_part[1][warp] = bits;
        s_part[2][warp] = m;
    }
    __syncthreads();
    if (warp > 0) return;
    flags = __reduce_or_sync(0xffffffffu, lane < 8 ? s_part[0][lane] : 0u);
    bits = __reduce_or_sync(0xffffffffu, lane < 8 ? s_part[1][lane] : 0u);
    m = __reduce_max_sync(0xffffffffu, lane < 8 ? s_part[2][lane] : 0u);
    if (lane == 0) {
        if (flags & ~static_cast<uint32_t>(__ldcg(stats))) atomicOr(stats, static_cast<int>(flags));
        if (bits & ~static_cast<uint32_t>(__ldcg(stats + 1))) atomicOr(stats + 1, static_cast<int>(bits));
        if (m > static_cast<uint32_t>(__ldcg(stats + 2))) atomicMax(stats + 2, static_cast<int>(m));
    }
}

// One pass over the query and the base rows (n_q and n_r groups of 16 bytes):
// the survey of all values and, with out pointers, their u8 form (mul = 1),
// final when every value is an integer in [0, 255]. Four loads in flight per
// thread; HBM-bound (512 or 256 bytes read per row, 128 written).
// One launch for both sets instead of separate pack, scale and range passes, and
// one synchronisation for the caller instead of up to three: cublas_2nn_sift
// on 1,000 x 10,000 rows of integers / 512 132 -> 82 us,
// general float match() of 2,053 x 131,077 rows 339 -> 257 us (with the fused split).
template <bool HALF, bool SURVEY>
__global__ void __launch_bounds__(256)
    convert_kernel(const uint4* __restrict__ q, size_t n_q, const uint4* __restrict__ r, size_t n_r, float mul,
                   uint8_t* __restrict__ q_out, uint8_t* __restrict__ r_out, int* __restrict__ stats) {
    uint32_t flags = 0, bits = 0, mx2 = 0, words = 0;
    float mx = 0.0f;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x, n = n_q + n_r;
    for (size_t i0 = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i0 < n; i0 += 4 * stride) {
        uint4 v[4];
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            const size_t i = i0 + k * stride;
            v[k] = i < n ? (i < n_q ? q[i] : r[i - n_q]) : make_uint4(0u, 0u, 0u, 0u);
        }
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            const size_t i = i0 + k * stride;
            if (i >= n) break;
            const bool in_q = i < n_q;
            const size_t at = in_q ? i : i - n_q;
            uint8_t* out = in_q ? q_out : r_out;
            if constexpr (HALF) {
                if constexpr (SURVEY) {
                    const uint32_t w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
                    words = 0;
                    #pragma unroll
                    for (int e = 0; e < 4; ++e) survey_half2(w[e], half2_floats(w[e]), bits, mx2, words);
                    if ((words & 0x80008000u) &&
                        (negative_half2(w[0]) || negative_half2(w[1]) || negative_half2(w[2]) || negative_half2(w[3])))
                        flags |= kValueNotFixed;
                }
                if (out) {
                    const float2 a = half2_floats(v[k].x), b = half2_floats(v[k].y), c = half2_floats(v[k].z),
                                 d = half2_floats(v[k].w);
                    reinterpret_cast<uint2*>(out)[at] = make_uint2(pack4(make_float4(a.x, a.y, b.x, b.y), mul),
                                                                   pack4(make_float4(c.x, c.y, d.x, d.y), mul));
                }
            } else {
                const float4 f = *reinterpret_cast<const float4*>(&v[k]);
                uint32_t packed;
                if constexpr (SURVEY) {
                    packed = survey_one(f.x, flags, bits, mx) >> 24;
                    packed |= (survey_one(f.y, flags, bits, mx) >> 24) << 8;
                    packed |= (survey_one(f.z, flags, bits, mx) >> 24) << 16;
                    packed |= (survey_one(f.w, flags, bits, mx) >> 24) << 24;
                } else {
                    packed = pack4(f, mul);
                }
                if (out) reinterpret_cast<uint32_t*>(out)[at] = packed;
            }
        }
    }
    if constexpr (SURVEY) {
        if constexpr (HALF) mx = half_max(mx2, flags);
        // Integers in [0, 255]: in range and no bit below 2^24.
        if ((bits & 0xffffffu) || (flags & kValueNotFixed)) flags |= kValueNotU8;
        survey_flush(flags, bits, mx, stats);
    }
}

template <bool SURVEY>
cudaError_t launch_convert(const void* q, size_t q_rows, const void* r, size_t r_rows, bool half, float mul,
                           uint8_t* q_out, uint8_t* r_out, int* stats, int num_sms, cudaStream_t stream) {
    const size_t per_row = half ? 16 : 32, n_q = q_rows * per_row, n_r = r_rows * per_row;
    if (n_q + n_r == 0) return cudaSuccess;
    const size_t blocks = std::min<size_t>((n_q + n_r + 1023) / 1024, static_cast<size_t>(num_sms) * 8);
    const auto* qp = static_cast<const uint4*>(q);
    const auto* rp = static_cast<const uint4*>(r);
    if (half)
        convert_kernel<true, SURVEY><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(qp, n_q, rp, n_r, mul, q_out,
                                                                                       r_out, stats);
    else
        convert_kernel<false, SURVEY><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(qp, n_q, rp, n_r, mul, q_out,
                                                                                        r_out, stats);
    return cudaGetLastError();
}

// ---- FP16 rows: survey, norms and records in one pass
// One block per 128 rows (8 threads per row, four 32-byte loads in flight per
// thread): the survey of its values and the rows' squared norms, FP32 sums of
// the squares as they are. For integers times 2^-s every partial sum is an
// integer below 2^23 times 2^-2s, exact at any scale, so the norms need not
// wait for s. Blocks [0, base_tiles) write records (norms, 8-row minima), the
// others query norms and clear the shared bounds. HBM-bound: 256 bytes per row.
// FP16 2,561 x 500,003: survey 77 + norms 25 us in two passes before, 30 us now
// (65 with per-element integer shifts and three atomics per warp).
__global__ void __launch_bounds__(256)
    survey_norms_f16_kernel(const __half* __restrict__ r, int r_n, int base_tiles, int metric, int32_t* __restrict__ rec,
                            const __half* __restrict__ q, int q_n, int q_pad, int32_t* __restrict__ qnorm,
                            int32_t* __restrict__ thresh, int* __restrict__ stats) {
    const int sub = threadIdx.x & 7, lrow = threadIdx.x >> 3;
    const bool is_base = static_cast<int>(blockIdx.x) < base_tiles;
    const __half* x = is_base ? r : q;
    const int n = is_base ? r_n : q_n;
    const int row0 = (static_cast<int>(blockIdx.x) - (is_base ? 0 : base_tiles)) * kBN;
    uint4 v[4][2];
    #pragma unroll
    for (int part = 0; part < 4; ++part) {
        const int row = row0 + part * 32 + lrow;
        const uint4* p = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * kDim) + 2 * sub;
        v[part][0] = row < n ? p[0] : make_uint4(0u, 0u, 0u, 0u);
        v[part][1] = row < n ? p[1] : make_uint4(0u, 0u, 0u, 0u);
    }
    __shared__ float nrm[kBN];
    uint32_t flags = 0, bits = 0, mx2 = 0, words = 0;
    #pragma unroll
    for (int part = 0; part < 4; ++part) {
        float s = 0.0f;
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t w[4] = {v[part][h].x, v[part][h].y, v[part][h].z, v[part][h].w};
            #pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = half2_floats(w[k]);
                survey_half2(w[k], f, bits, mx2, words);
                s = fmaf(f.x, f.x, s);
                s = fmaf(f.y, f.y, s);
            }
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        const int col = part * 32 + lrow, row = row0 + col;
        if (sub != 0) continue;
        if (is_base) {
            nrm[col] = row < n ? (metric == kMetricL2 ? s : 0.0f) : kFloatKeyPad;
        } else if (row < q_pad) {
            qnorm[row] = __float_as_int(s);
            thresh[row] = thresh[static_cast<size_t>(q_pad) + row] = INT_MAX;
        }
    }
    __syncthreads();
    if (is_base) {
        int32_t* o = rec + static_cast<size_t>(blockIdx.x) * kRecInts;
        if (threadIdx.x < kBN) o[threadIdx.x] = __float_as_int(nrm[threadIdx.x]);
        if (threadIdx.x < 16) {
            float m = nrm[8 * threadIdx.x];
            #pragma unroll
            for (int i = 1; i < 8; ++i) m = fminf(m, nrm[8 * threadIdx.x + i]);
            o[kBN + threadIdx.x] = __float_as_int(m);
        }
    }
    if (words & 0x80008000u) {
        #pragma unroll
        for (int part = 0; part < 4; ++part)
            #pragma unroll
            for (int h = 0; h < 2; ++h)
                if (negative_half2(v[part][h].x) || negative_half2(v[part][h].y) || negative_half2(v[part][h].z) ||
                    negative_half2(v[part][h].w))
                    flags |= kValueNotFixed;
    }
    const float mx = half_max(mx2, flags);
    survey_flush(flags, bits, mx, stats);
}

// ---- general float rows: split and norms in one pass
// Float rows times mul -> split FP16 rows [n][256], halves [0, 128) holding
// hi = fp16(x * mul) and [128, 256) lo = fp16(x * mul - hi), so hi + lo carries
// 22 significant bits of x * mul (mul a power of two: exact); and the squared
// norms of x * mul (FP32, 16 elements in order per thread, then the 8 threads of
// a row), as row_norms_float_kernel lays them out: base records, then query
// norms and cleared bounds. One block per 32 rows; HBM-bound, 512 bytes read and
// 512 written per row instead of 512 read twice.
__global__ void __launch_bounds__(256)
    split_norms_f32_kernel(const float* __restrict__ r, int r_n, int r_pad, int metric, __half* __restrict__ r_out,
                           int32_t* __restrict__ rec, const float* __restrict__ q, int q_n, int q_pad,
                           __half* __restrict__ q_out, int32_t* __restrict__ qnorm, int32_t* __restrict__ thresh,
                           float mul) {
    launch_next();
    const int base_blocks = r_pad / 32;
    const bool is_base = static_cast<int>(blockIdx.x) < base_blocks;
    const int b = static_cast<int>(blockIdx.x) - (is_base ? 0 : base_blocks);
    const int lrow = threadIdx.x >> 3, sub = threadIdx.x & 7, row = b * 32 + lrow;
    const int n = is_base ? r_n : q_n;
    float s = 0.0f;
    if (row < n) {
        const float4* p = reinterpret_cast<const float4*>((is_base ? r : q) + static_cast<size_t>(row) * kDim) + 4 * sub;
        float f[16];
        #pragma unroll
        for (int h = 0; h < 4; ++h) {
            const float4 v = p[h];
            f[4 * h] = v.x * mul;
            f[4 * h + 1] = v.y * mul;
            f[4 * h + 2] = v.z * mul;
            f[4 * h + 3] = v.w * mul;
        }
        __half hi[16], lo[16];
        #pragma unroll
        for (int i = 0; i < 16; ++i) {
            s = fmaf(f[i], f[i], s);
            hi[i] = __float2half_rn(f[i]);
            lo[i] = __float2half_rn(f[i] - __half2float(hi[i]));
        }
        uint4* o = reinterpret_cast<uint4*>((is_base ? r_out : q_out) + static_cast<size_t>(row) * 256 + 16 * sub);
        o[0] = reinterpret_cast<const uint4*>(hi)[0];
        o[1] = reinterpret_cast<const uint4*>(hi)[1];
        o[16] = reinterpret_cast<const uint4*>(lo)[0];
        o[17] = reinterpret_cast<const uint4*>(lo)[1];
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    __shared__ float nrm[32];
    if (is_base) {
        const float v = row < n ? (metric == kMetricL2 ? s : 0.0f) : kFloatKeyPad;
        int32_t* o = rec + static_cast<size_t>(b / 4) * kRecInts;
        const int part = b & 3;
        if (sub == 0) {
            nrm[lrow] = v;
            o[part * 32 + lrow] = __float_as_int(v);
        }
        __syncthreads();
        if (threadIdx.x < 4) {
            float m = nrm[8 * threadIdx.x];
            #pragma unroll
            for (int i = 1; i < 8; ++i) m = fminf(m, nrm[8 * threadIdx.x + i]);
            o[kBN + part * 4 + threadIdx.x] = __float_as_int(m);
        }
    } else if (sub == 0 && row < q_pad) {
        qnorm[row] = __float_as_int(row < n ? s : kFloatKeyPad);
        thresh[row] = thresh[static_cast<size_t>(q_pad) + row] = INT_MAX;
    }
}

}  // namespace

int value_shift(uint32_t bits) {
    int low = 0;
    while (low < 24 && !((bits >> low) & 1u)) ++low;
    return bits ? 24 - low : 0;
}

cudaError_t launch_survey(const void* q, size_t q_rows, const void* r, size_t r_rows, bool half, uint8_t* q_out,
                          uint8_t* r_out, int* stats, int num_sms, cudaStream_t stream) {
    return launch_convert<true>(q, q_rows, r, r_rows, half, 1.0f, q_out, r_out, stats, num_sms, stream);
}

cudaError_t launch_pack_u8(const void* q, size_t q_rows, const void* r, size_t r_rows, bool half, float mul,
                           uint8_t* q_out, uint8_t* r_out, int num_sms, cudaStream_t stream) {
    return launch_convert<false>(q, q_rows, r, r_rows, half, mul, q_out, r_out, nullptr, num_sms, stream);
}

cudaError_t launch_survey_norms_f16(const void* r, int r_n, int base_tiles, int metric, int32_t* rec, const void* q,
                                    int q_n, int q_pad, int32_t* qnorm, int32_t* thresh, int* stats,
                                    cudaStream_t stream) {
    const int blocks = base_tiles + q_pad / kBN;
    if (blocks <= 0) return cudaSuccess;
    survey_norms_f16_kernel<<<blocks, 256, 0, stream>>>(static_cast<const __half*>(r), r_n, base_tiles, metric, rec,
                                                        static_cast<const __half*>(q), q_n, q_pad, qnorm, thresh, stats);
    return cudaGetLastError();
}

cudaError_t launch_split_norms_f32(const float* r, int r_n, int r_pad, int metric, void* r_out, int32_t* rec,
                                   const float* q, int q_n, int q_pad, void* q_out, int32_t* qnorm, int32_t* thresh,
                                   float mul, cudaStream_t stream) {
    const int blocks = r_pad / 32 + q_pad / 32;
    if (blocks <= 0) return cudaSuccess;
    split_norms_f32_kernel<<<blocks, 256, 0, stream>>>(r, r_n, r_pad, metric, static_cast<__half*>(r_out), rec, q, q_n,
                                                       q_pad, static_cast<__half*>(q_out), qnorm, thresh, mul);
    return cudaGetLastError();
}

}  // namespace sift
