// Training kernels of the learned hash (forward, loss, backward, Adam).
//
// Model (learned.cuh): a1 = W1 (x / 64) + b1, h = bf16(relu(a1)),
// z = W2 h + b2, t = tanh(z) (the sign surrogate; codes use sign(z)).
// One step sees R = 3B rows: B training queries, their exact nearest
// neighbours (labelled by the exact search kernel) and B random base rows.
// With s(a, b) = (1/k) sum_j t_aj t_bj and m_j = mean over the R rows of t_j:
//   loss = mean_i (1 - s(q_i, p_i)) + neg * mean_i s(q_i, n_i)^2 + balance * sum_j m_j^2
// (neighbours agree bit by bit, random pairs decorrelate, every bit splits
// the data evenly). Gradients pass straight through the BF16 roundings of the
// weights and of h. Every reduction runs in a fixed order, so a step is
// deterministic.
//
// Three launches per step, FP32 throughout (CUDA cores):
//   mlp_fwd_kernel   h and t of kFwdRows rows per block, column sums of t
//   mlp_bwd_kernel   per (64 hidden units, chunk of pairs): dz, the hidden
//                    gradient and the chunk's share of every weight gradient;
//                    four more blocks form the pairs' loss terms
//   mlp_reduce_kernel  the shares of all chunks, the loss, and in training the
//                    Adam update with the BF16 copies of the next step
// The step is bound by FP32 issue (0.43 GFMA at a batch of 2,048 pairs, 14 us on
// 148 SMs at the 1.2 cycles that a warp's FMA takes; paired FMAs (f32x2) take
// 2.4), by the bandwidth from shared memory to registers and by the latency of
// three short launches, each of which starts while the one before still runs
// (launch.cuh). One step at 2,048 pairs, 16 bits (whole mlp_loss_grad call): 76 us,
// of which the forward 16 and the backward 22, against 865 with eight launches whose
// weight gradients walked all rows in 8 and 32 blocks. The gradients' error against
// FP64 is 1.7e-7 of the norm at 2,048 pairs (1.0e-6 with the longer sums).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_bf16.h>
#include <type_traits>
#include "launch.cuh"
#include "learned.cuh"

namespace sift {
namespace {

// ---------------------------------------------------------------- forward
// 48 rows per block (128 blocks for 3 x 2,048 rows: one wave). W1 arrives
// transposed ([in][hidden], 64 KB) so that it is copied as it is; warp w owns
// rows 6 w .. 6 w + 5 and lane l hidden units 8 l .. 8 l + 7, so one 16-byte
// load of weights and three broadcast loads of inputs feed 48 FMAs (19,000 cycles
// of the block's 31,000; a warp's FMAs alone would take 14,700). 16 warps of 6 rows
// and 4 units each took 20,900: as many FMAs for more loaded bytes. The weights
// arrive by asynchronous copies under the conversion of the inputs. Sums run over
// the inputs (hidden units) in order.
constexpr int kFwdRows = 48;
constexpr int kFwdThreads = 256;
constexpr int kFwdWarpRows = kFwdRows / (kFwdThreads / 32);
constexpr int kFwdHPitch = kMlpHidden + 4;
constexpr int kFwdW2Pitch = kMlpOutRows + 1;
constexpr size_t kFwdSmem = kMlpIn * kMlpHidden * 2 + kMlpHidden * kFwdW2Pitch * 4 + kFwdRows * kMlpIn * 4 +
                            kFwdRows * kFwdHPitch * 4;

// Layer 2 of NR rows of a warp (h: the first of them), one output per lane.
template <int NR>
__device__ __forceinline__ void fwd_layer2(const float* __restrict__ h, const float* __restrict__ w2m, float (&acc)[NR]) {
    #pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = 0.0f;
    #pragma unroll 4
    for (int j = 0; j < kMlpHidden; j += 4) {
        float w[4];
        #pragma unroll
        for (int u = 0; u < 4; ++u) w[u] = w2m[(j + u) * kFwdW2Pitch];
        #pragma unroll
        for (int r = 0; r < NR; ++r) {
            const float4 hv = *reinterpret_cast<const float4*>(h + r * kFwdHPitch + j);
            acc[r] = fmaf(hv.x, w[0], acc[r]);
            acc[r] = fmaf(hv.y, w[1], acc[r]);
            acc[r] = fmaf(hv.z, w[2], acc[r]);
            acc[r] = fmaf(hv.w, w[3], acc[r]);
        }
    }
}

__global__ void __launch_bounds__(kFwdThreads, 1)
    mlp_fwd_kernel(const uint8_t* x, int R, const __nv_bfloat16* w1t,
                   const float* b1, const __nv_bfloat16* w2b, const float* b2,
                   int k, float* __restrict__ h_out, float* __restrict__ t_out, float* __restrict__ colpart) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t* w1s = smem;                                                            // [128][256] bf16
    float* xs = reinterpret_cast<float*>(smem + kMlpIn * kMlpHidden * 2);           // [128][48]
    float* hs = xs + kFwdRows * kMlpIn;                                             // [48][260]
    float* w2s = hs + kFwdRows * kFwdHPitch;                                        // [256][33]
    __shared__ float s_col[kFwdThreads / 32][32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = blockIdx.x * kFwdRows;
    wait_previous();
    uint4 xv[(kFwdRows * 8 + kFwdThreads - 1) / kFwdThreads], wv[kMlpOutRows * kMlpHidden / 8 / kFwdThreads];
    #pragma unroll
    for (int u = 0; u < static_cast<int>(sizeof(xv) / 16); ++u) {
        const int e = tid + u * kFwdThreads, r = e % kFwdRows, c = e / kFwdRows;
        xv[u] = make_uint4(0u, 0u, 0u, 0u);
        if (c < 8 && row0 + r < R) xv[u] = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row0 + r) * kMlpIn)[c];
    }
    const float4 bj[2] = {reinterpret_cast<const float4*>(b1)[2 * lane], reinterpret_cast<const float4*>(b1)[2 * lane + 1]};
    #pragma unroll
    for (int u = 0; u < static_cast<int>(sizeof(xv) / 16); ++u) {
        const int e = tid + u * kFwdThreads, r = e % kFwdRows, c = e / kFwdRows;
        if (c >= 8) break;
        const uint32_t w[4] = {xv[u].x, xv[u].y, xv[u].z, xv[u].w};
        #pragma unroll
        for (int i = 0; i < 16; ++i)
            xs[(16 * c + i) * kFwdRows + r] = static_cast<float>((w[i >> 2] >> (8 * (i & 3))) & 0xffu) * kMlpInScale;
    }
    for (int e = tid; e < kMlpIn * kMlpHidden / 8; e += kFwdThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(w1s + 16 * e))),
                     "l"(w1t + 8 * e)
                     : "memory");
    #pragma unroll
    for (int u = 0; u < static_cast<int>(sizeof(wv) / 16); ++u) {
        const int e = tid + u * kFwdThreads, m = e % kMlpOutRows, c = e / kMlpOutRows;
        wv[u] = make_uint4(0u, 0u, 0u, 0u);
        if (m < k) wv[u] = reinterpret_cast<const uint4*>(w2b + m * kMlpHidden)[c];
    }
    #pragma unroll
    for (int u = 0; u < static_cast<int>(sizeof(wv) / 16); ++u) {
        const int e = tid + u * kFwdThreads, m = e % kMlpOutRows, c = e / kMlpOutRows;
        const uint32_t w[4] = {wv[u].x, wv[u].y, wv[u].z, wv[u].w};
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            w2s[(8 * c + 2 * i) * kFwdW2Pitch + m] = __uint_as_float(w[i] << 16);
            w2s[(8 * c + 2 * i + 1) * kFwdW2Pitch + m] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    {
        float acc[kFwdWarpRows][8];
        #pragma unroll
        for (int r = 0; r < kFwdWarpRows; ++r)
            #pragma unroll
            for (int c = 0; c < 8; ++c) acc[r][c] = 0.0f;
        const uint4* wp = reinterpret_cast<const uint4*>(w1s) + lane;
        const float* xp = xs + warp * kFwdWarpRows;
        #pragma unroll 8
        for (int i = 0; i < kMlpIn; ++i) {
            const uint4 v = wp[i * (kMlpHidden / 8)];
            const uint32_t w2[4] = {v.x, v.y, v.z, v.w};
            float w[8];
            #pragma unroll
            for (int c = 0; c < 4; ++c) {
                w[2 * c] = __uint_as_float(w2[c] << 16);
                w[2 * c + 1] = __uint_as_float(w2[c] & 0xffff0000u);
            }
            #pragma unroll
            for (int r = 0; r < kFwdWarpRows; r += 2) {
                const float2 xv2 = *reinterpret_cast<const float2*>(xp + i * kFwdRows + r);
                #pragma unroll
                for (int c = 0; c < 8; ++c) {
                    acc[r][c] = fmaf(xv2.x, w[c], acc[r][c]);
                    acc[r + 1][c] = fmaf(xv2.y, w[c], acc[r + 1][c]);
                }
            }
        }
        #pragma unroll
        for (int r = 0; r < kFwdWarpRows; ++r) {
            const int lr = warp * kFwdWarpRows + r;
            #pragma unroll
            for (int g = 0; g < 2; ++g) {
                const float* z = acc[r] + 4 * g;
                const float4 o = make_float4(__bfloat162float(__float2bfloat16_rn(fmaxf(z[0] + bj[g].x, 0.0f))),
                                             __bfloat162float(__float2bfloat16_rn(fmaxf(z[1] + bj[g].y, 0.0f))),
                                             __bfloat162float(__float2bfloat16_rn(fmaxf(z[2] + bj[g].z, 0.0f))),
                                             __bfloat162float(__float2bfloat16_rn(fmaxf(z[3] + bj[g].w, 0.0f))));
                *reinterpret_cast<float4*>(hs + lr * kFwdHPitch + 8 * lane + 4 * g) = o;
                if (row0 + lr < R)
                    *reinterpret_cast<float4*>(h_out + static_cast<size_t>(row0 + lr) * kMlpHidden + 8 * lane + 4 * g) =
                        o;
            }
        }
    }
    __syncwarp();  // layer 2 reads the warp's own rows
    float col = 0.0f;
    auto finish = [&](int lr, int m, float z) {  // t of row lr, output m
        if (row0 + lr < R) {
            const float t = m < k ? tanhf(z + (m < k ? b2[m] : 0.0f)) : 0.0f;
            t_out[static_cast<size_t>(row0 + lr) * kMlpOutRows + m] = t;
            col += t;
        }
    };
    if (k <= kMlpOutRows / 2) {
        // Half the lanes would have no output: each half of a warp takes half its rows.
        constexpr int NR = kFwdWarpRows / 2;
        const int m = lane & 15, lr = warp * kFwdWarpRows + (lane >> 4) * NR;
        float acc[NR];
        fwd_layer2<NR>(hs + lr * kFwdHPitch, w2s + m, acc);
        #pragma unroll
        for (int r = 0; r < NR; ++r) {
            finish(lr + r, m, acc[r]);
            if (row0 + lr + r < R) t_out[static_cast<size_t>(row0 + lr + r) * kMlpOutRows + 16 + m] = 0.0f;
        }
        col += __shfl_xor_sync(0xffffffffu, col, 16);
        if (lane >= 16) col = 0.0f;
    } else {
        const int lr = warp * kFwdWarpRows;
        float acc[kFwdWarpRows];
        fwd_layer2<kFwdWarpRows>(hs + lr * kFwdHPitch, w2s + lane, acc);
        #pragma unroll
        for (int r = 0; r < kFwdWarpRows; ++r) finish(lr + r, lane, acc[r]);
    }
    s_col[warp][lane] = col;
    __syncthreads();
    if (warp == 0) {
        float c = 0.0f;
        #pragma unroll
        for (int w = 0; w < kFwdThreads / 32; ++w) c += s_col[w][lane];
        colpart[static_cast<size_t>(blockIdx.x) * 32 + lane] = c;
    }
}

// --------------------------------------------------------------- backward
// Block (a, c): hidden units [64 a, 64 a + 64) and pairs [B c / C, B (c + 1) / C),
// C = gridDim.y, 32 pairs (96 rows: queries, neighbours, random rows) at a time:
// dz of the 96 rows, then per 32 rows the hidden gradient
// da1[row][j] = (sum_m dz[row][m] W2[m][j]) (h[row][j] > 0) and the rank-32
// updates dW1 += da1^T (x / 64) (4 x 8 outputs per thread, 64 x 128 per half of the
// block) and dW2 += dz^T h in one loop: each half of the block's 16 warps takes
// every second row, and the halves' sums meet at the end. db1 and db2 are summed
// where da1 and dz are formed. The next 32 rows' x and h load meanwhile. 8 warps
// that took all rows and ran dW2 as a loop of its own needed 68,500 cycles, this
// 43,300 (38.5 -> 22 us); 8 x 8 outputs per thread over four row groups 53,200. The four
// blocks of a chunk recompute its dz (a few FMAs per row against the 8,192 of
// its share of dW1). The chunk's sums go to part[c][kMlpParamCount].
// Blocks (a, C) are the loss role, which only reads t and runs beside the
// others: the terms of every pair and 32 strided column sums of t, in one fixed
// order of additions (a thread per pair over the outputs in order; rows p,
// p + 32, ... per strided sum) that does not depend on the chunks.
constexpr int kBwdCols = 64;
constexpr int kBwdPairs = 32;
constexpr int kBwdThreads = 512;
constexpr int kBwdColBlocks = kMlpHidden / kBwdCols;
constexpr int kBwdMaxChunks = 36;  // + the loss role, x 4 column blocks = one block per SM
constexpr int kBwdPitch = kBwdCols + 4, kBwdXPitch = kMlpIn + 4, kBwdDzPitch = kMlpOutRows + 4;
constexpr size_t kBwdSmem = (3 * kBwdPairs * kBwdDzPitch + 32 * kBwdPitch * 2 + 32 * kBwdXPitch +
                             kMlpOutRows * kBwdCols + 32 + (kBwdThreads / 32) * 32) * 4;
// The sums at the end of a block reuse the buffers of its loop.
static_assert((kBwdCols * kMlpIn + kMlpOutRows * kBwdCols + 32 * kBwdCols + (kBwdThreads / 32) * 32) * 4 <= kBwdSmem,
              "buffers of the final sums");

__device__ __forceinline__ void loss_role(const float* t, int B, int k, int a, float* __restrict__ colp,
                                          float* __restrict__ terms) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int R = 3 * B;
    for (int p = a * (kBwdThreads / 32) + warp; p < 32; p += kBwdColBlocks * (kBwdThreads / 32)) {
        float s = 0.0f;
        #pragma unroll 16
        for (int r = p; r < R; r += 32) s += t[static_cast<size_t>(r) * kMlpOutRows + lane];
        colp[p * 32 + lane] = s;
    }
    for (int i = a * kBwdThreads + threadIdx.x; i < B; i += kBwdColBlocks * kBwdThreads) {
        const float* tq = t + static_cast<size_t>(i) * kMlpOutRows;
        const float* tp = t + (static_cast<size_t>(B) + i) * kMlpOutRows;
        const float* tn = t + (2 * static_cast<size_t>(B) + i) * kMlpOutRows;
        float sqp = 0.0f, sqn = 0.0f;
        for (int j0 = 0; j0 < k; j0 += 4) {
            const float4 q = *reinterpret_cast<const float4*>(tq + j0), p = *reinterpret_cast<const float4*>(tp + j0),
                         n = *reinterpret_cast<const float4*>(tn + j0);
            const float qv[4] = {q.x, q.y, q.z, q.w}, pv[4] = {p.x, p.y, p.z, p.w}, nv[4] = {n.x, n.y, n.z, n.w};
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j0 + j < k) {
                    sqp = fmaf(qv[j], pv[j], sqp);
                    sqn = fmaf(qv[j], nv[j], sqn);
                }
            }
        }
        sqp /= k;
        sqn /= k;
        terms[2 * static_cast<size_t>(i)] = 1.0f - sqp;
        terms[2 * static_cast<size_t>(i) + 1] = sqn * sqn;
    }
}

__global__ void __launch_bounds__(kBwdThreads, 1)
    mlp_bwd_kernel(const uint8_t* x, int B, int k, const float* h,
                   const float* t, const __nv_bfloat16* w2b, MlpLossWeights lw,
                   const float* colpart, int n_colpart, float* __restrict__ colp,
                   float* __restrict__ terms, float* __restrict__ part) {
    wait_previous();
    const int c = blockIdx.y, C = gridDim.y - 1;
    if (c == C) {
        loss_role(t, B, k, blockIdx.x, colp, terms);
        return;
    }
    extern __shared__ __align__(16) uint8_t smem[];
    float* hs = reinterpret_cast<float*>(smem);        // [32][68]
    float* as = hs + 32 * kBwdPitch;                   // [32][68]
    float* xs = as + 32 * kBwdPitch;                   // [32][132]
    float* w2s = xs + 32 * kBwdXPitch;                 // [32][64]
    float* dzs = w2s + kMlpOutRows * kBwdCols;         // [96][36]
    float* cs = dzs + 3 * kBwdPairs * kBwdDzPitch;     // [32]
    float* red = cs + 32;                              // [16][32]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int col0 = blockIdx.x * kBwdCols;
    const int i_begin = static_cast<int>(static_cast<long long>(B) * c / C);
    const int i_end = static_cast<int>(static_cast<long long>(B) * (c + 1) / C);
    const float rows = 3.0f * B;
    constexpr int kWarps = kBwdThreads / 32;

    // Row r4 of a part and its 4 hidden units (8 inputs) from 4 q4 (8 q4): what
    // this thread loads, and the hidden gradient that it forms.
    const int r4 = tid >> 4, q4 = tid & 15;
    uint2 nx;
    float4 nh;
    auto fetch = [&](int p, int i0, int np) {
        if (r4 < np) {
            const size_t row = static_cast<size_t>(p) * B + i0 + r4;
            nx = reinterpret_cast<const uint2*>(x + row * kMlpIn)[q4];
            nh = *reinterpret_cast<const float4*>(h + row * kMlpHidden + col0 + 4 * q4);
        } else {
            nx = make_uint2(0u, 0u);
            nh = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    if (i_begin < i_end) fetch(0, i_begin, min(kBwdPairs, i_end - i_begin));

    {
        float s = 0.0f;
        #pragma unroll 8
        for (int b = warp; b < n_colpart; b += kWarps) s += colpart[static_cast<size_t>(b) * 32 + lane];
        red[warp * 32 + lane] = s;
    }
    #pragma unroll
    for (int e = tid; e < kMlpOutRows * kBwdCols; e += kBwdThreads) {
        const int m = e / kBwdCols, j = e % kBwdCols;
        w2s[e] = m < k ? __bfloat162float(w2b[m * kMlpHidden + col0 + j]) : 0.0f;
    }
    __syncthreads();
    if (warp == 0) {
        float s = 0.0f;
        #pragma unroll
        for (int w = 0; w < kWarps; ++w) s += red[w * 32 + lane];
        cs[lane] = s;
    }
    __syncthreads();

    // Outputs of this thread, over the rows r with r % 2 == half: dW1 rows 4 ty .. + 3
    // (hidden units), columns 4 tx .. + 3 and 64 + 4 tx .. + 3; dW2 rows ty (and
    // 16 + ty), columns 4 tx .. + 3.
    const int half = tid >> 8, ty = (tid >> 4) & 15, tx = tid & 15;
    float acc[4][8], acc2[2][4], b1s[4] = {0.0f, 0.0f, 0.0f, 0.0f}, b2s = 0.0f;
    #pragma unroll
    for (int e = 0; e < 8; ++e) {
        acc2[e >> 2][e & 3] = 0.0f;
        #pragma unroll
        for (int q = 0; q < 4; ++q) acc[q][e] = 0.0f;
    }

    for (int i0 = i_begin; i0 < i_end; i0 += kBwdPairs) {
        const int np = min(kBwdPairs, i_end - i0);
        // dz of the 3 np rows: a warp per pair, a lane per output.
        constexpr int kPer = kBwdPairs / kWarps;
        float tv[kPer][3];
        #pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int pi = warp + u * kWarps;
            const size_t i = static_cast<size_t>(i0) + pi;
            #pragma unroll
            for (int p = 0; p < 3; ++p)
                tv[u][p] = pi < np ? t[(static_cast<size_t>(p) * B + i) * kMlpOutRows + lane] : 0.0f;
        }
        #pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int pi = warp + u * kWarps;
            const float tq = tv[u][0], tp = tv[u][1], tn = tv[u][2];
            float sqn = tq * tn;  // zero for lanes >= k
            #pragma unroll
            for (int o = 16; o > 0; o >>= 1) sqn += __shfl_xor_sync(0xffffffffu, sqn, o);
            sqn /= k;
            const float cp = -1.0f / (k * static_cast<float>(B));
            const float cn = lw.neg * 2.0f * sqn / (k * static_cast<float>(B));
            float dq = 0.0f, dp = 0.0f, dn = 0.0f;
            if (pi < np && lane < k) {
                const float bal = lw.balance * 2.0f * (cs[lane] / rows) / rows;
                dq = (cp * tp + cn * tn + bal) * (1.0f - tq * tq);
                dp = (cp * tq + bal) * (1.0f - tp * tp);
                dn = (cn * tq + bal) * (1.0f - tn * tn);
            }
            dzs[pi * kBwdDzPitch + lane] = dq;
            dzs[(kBwdPairs + pi) * kBwdDzPitch + lane] = dp;
            dzs[(2 * kBwdPairs + pi) * kBwdDzPitch + lane] = dn;
            b2s += dq + dp + dn;
        }
        for (int p = 0; p < 3; ++p) {
            {
                const uint32_t w[2] = {nx.x, nx.y};
                #pragma unroll
                for (int g = 0; g < 2; ++g)
                    *reinterpret_cast<float4*>(xs + r4 * kBwdXPitch + 8 * q4 + 4 * g) =
                        make_float4(static_cast<float>(w[g] & 0xffu) * kMlpInScale,
                                    static_cast<float>((w[g] >> 8) & 0xffu) * kMlpInScale,
                                    static_cast<float>((w[g] >> 16) & 0xffu) * kMlpInScale,
                                    static_cast<float>(w[g] >> 24) * kMlpInScale);
                *reinterpret_cast<float4*>(hs + r4 * kBwdPitch + 4 * q4) = nh;
            }
            const float4 hr = nh;
            if (p < 2)
                fetch(p + 1, i0, np);
            else if (i0 + kBwdPairs < i_end)
                fetch(0, i0 + kBwdPairs, min(kBwdPairs, i_end - i0 - kBwdPairs));
            __syncthreads();  // dzs, xs, hs
            const float* dz = dzs + p * kBwdPairs * kBwdDzPitch;
            {
                // dz and W2 are zero for outputs past k.
                float g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                #pragma unroll 4
                for (int m = 0; m < k; m += 4) {
                    const float4 d = *reinterpret_cast<const float4*>(dz + r4 * kBwdDzPitch + m);
                    const float dv[4] = {d.x, d.y, d.z, d.w};
                    #pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float4 w = *reinterpret_cast<const float4*>(w2s + (m + u) * kBwdCols + 4 * q4);
                        g[0] = fmaf(dv[u], w.x, g[0]);
                        g[1] = fmaf(dv[u], w.y, g[1]);
                        g[2] = fmaf(dv[u], w.z, g[2]);
                        g[3] = fmaf(dv[u], w.w, g[3]);
                    }
                }
                const float4 a = make_float4(hr.x > 0.0f ? g[0] : 0.0f, hr.y > 0.0f ? g[1] : 0.0f,
                                             hr.z > 0.0f ? g[2] : 0.0f, hr.w > 0.0f ? g[3] : 0.0f);
                *reinterpret_cast<float4*>(as + r4 * kBwdPitch + 4 * q4) = a;
                b1s[0] += a.x;
                b1s[1] += a.y;
                b1s[2] += a.z;
                b1s[3] += a.w;
            }
            __syncthreads();  // as
            auto updates = [&](auto two_tag) {
                constexpr bool TWO = decltype(two_tag)::value;  // more than 16 outputs
                #pragma unroll 4
                for (int r = half; r < np; r += 2) {
                    const float4 a = *reinterpret_cast<const float4*>(as + r * kBwdPitch + 4 * ty);
                    const float4 u = *reinterpret_cast<const float4*>(xs + r * kBwdXPitch + 4 * tx);
                    const float4 v = *reinterpret_cast<const float4*>(xs + r * kBwdXPitch + 64 + 4 * tx);
                    const float4 hv = *reinterpret_cast<const float4*>(hs + r * kBwdPitch + 4 * tx);
                    const float d = dz[r * kBwdDzPitch + ty];
                    const float av[4] = {a.x, a.y, a.z, a.w};
                    const float bv[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
                    const float cv[4] = {hv.x, hv.y, hv.z, hv.w};
                    #pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        #pragma unroll
                        for (int e = 0; e < 8; ++e) acc[q][e] = fmaf(av[q], bv[e], acc[q][e]);
                    }
                    #pragma unroll
                    for (int e = 0; e < 4; ++e) acc2[0][e] = fmaf(d, cv[e], acc2[0][e]);
                    if constexpr (TWO) {
                        const float d1 = dz[r * kBwdDzPitch + 16 + ty];
                        #pragma unroll
                        for (int e = 0; e < 4; ++e) acc2[1][e] = fmaf(d1, cv[e], acc2[1][e]);
                    }
                }
            };
            if (k > 16)
                updates(std::true_type{});
            else
                updates(std::false_type{});
            __syncthreads();  // xs, hs, as and (after the last part) dzs are rewritten
        }
    }

    // The two halves' sums, then the rows' shares of db1 and the warps' of db2, in order.
    float* f1 = reinterpret_cast<float*>(smem);  // [64][128]
    float* f2 = f1 + kBwdCols * kMlpIn;          // [32][64]
    float* fb1 = f2 + kMlpOutRows * kBwdCols;    // [32][64]
    float* fb2 = fb1 + 32 * kBwdCols;            // [16][32]
    if (half == 1) {
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
            float* row = f1 + (4 * ty + q) * kMlpIn + 4 * tx;
            *reinterpret_cast<float4*>(row) = make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
            *reinterpret_cast<float4*>(row + 64) = make_float4(acc[q][4], acc[q][5], acc[q][6], acc[q][7]);
        }
        #pragma unroll
        for (int g = 0; g < 2; ++g)
            *reinterpret_cast<float4*>(f2 + (16 * g + ty) * kBwdCols + 4 * tx) =
                make_float4(acc2[g][0], acc2[g][1], acc2[g][2], acc2[g][3]);
    }
    *reinterpret_cast<float4*>(fb1 + r4 * kBwdCols + 4 * q4) = make_float4(b1s[0], b1s[1], b1s[2], b1s[3]);
    fb2[warp * 32 + lane] = b2s;
    __syncthreads();
    float* o = part + static_cast<size_t>(c) * kMlpParamCount;
    float* o2 = o + kMlpHidden * kMlpIn + kMlpHidden;
    if (half == 0) {
        auto sum4 = [](const float* mine, const float* other) {
            const float4 b = *reinterpret_cast<const float4*>(other);
            return make_float4(mine[0] + b.x, mine[1] + b.y, mine[2] + b.z, mine[3] + b.w);
        };
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float* row = f1 + (4 * ty + q) * kMlpIn + 4 * tx;
            float* out = o + static_cast<size_t>(col0 + 4 * ty + q) * kMlpIn + 4 * tx;
            *reinterpret_cast<float4*>(out) = sum4(acc[q], row);
            *reinterpret_cast<float4*>(out + 64) = sum4(acc[q] + 4, row + 64);
        }
        #pragma unroll
        for (int g = 0; g < 2; ++g)
            *reinterpret_cast<float4*>(o2 + (16 * g + ty) * kMlpHidden + col0 + 4 * tx) =
                sum4(acc2[g], f2 + (16 * g + ty) * kBwdCols + 4 * tx);
    } else if (tid < 256 + kBwdCols) {
        const int j = tid - 256;
        float s = 0.0f;
        #pragma unroll
        for (int r = 0; r < 32; ++r) s += fb1[r * kBwdCols + j];
        o[kMlpHidden * kMlpIn + col0 + j] = s;
    } else if (blockIdx.x == 0 && warp == kWarps - 1) {
        float s = 0.0f;
        #pragma unroll
        for (int w = 0; w < kWarps; ++w) s += fb2[w * 32 + lane];
        o2[kMlpOutRows * kMlpHidden + lane] = s;
    }
}

// ------------------------------------------------- reduction and Adam step
// g[i] = sum over chunks of part[c][i] (in order), a thread per parameter; the
// last block forms loss[0..3] = total, positive, negative, balance from the
// loss role's sums. ADAM: the update of parameter i and, for weights, the BF16
// copies the next step reads (W1 transposed, W2 as it is). L2 bound: 4 C bytes
// per parameter.
struct AdamState {
    float* p;
    float* m;
    float* v;
    __nv_bfloat16* w1t;
    __nv_bfloat16* w2b;
    float lr, c1, c2;
};

// loss[0..3] = total, positive, negative, balance (one block of 256 threads, fixed order).
__device__ __forceinline__ void loss_of_terms(const float* colp, const float* terms, int B,
                                              int k, MlpLossWeights lw, float* __restrict__ loss) {
    __shared__ float sp[256], sn[256], colsum[32];
    float a = 0.0f, b = 0.0f;
    #pragma unroll 8
    for (int i = threadIdx.x; i < B; i += 256) {
        const float2 v = reinterpret_cast<const float2*>(terms)[i];
        a += v.x;
        b += v.y;
    }
    sp[threadIdx.x] = a;
    sn[threadIdx.x] = b;
    if (threadIdx.x < 32) {
        float t = 0.0f;
        #pragma unroll
        for (int q = 0; q < 32; ++q) t += colp[q * 32 + threadIdx.x];
        colsum[threadIdx.x] = t;
    }
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            sp[threadIdx.x] += sp[threadIdx.x + s];
            sn[threadIdx.x] += sn[threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        float bal = 0.0f;
        const float rows = 3.0f * B;
        for (int j = 0; j < k; ++j) bal += (colsum[j] / rows) * (colsum[j] / rows);
        const float pos = sp[0] / B, neg = sn[0] / B;
        loss[0] = pos + lw.neg * neg + lw.balance * bal;
        loss[1] = pos;
        loss[2] = neg;
        loss[3] = bal;
    }
}

template <bool ADAM>
__global__ void __launch_bounds__(256)
    mlp_reduce_kernel(const float* part, int C, const float* colp,
                      const float* terms, int B, int k, MlpLossWeights lw, float* __restrict__ g,
                      float* __restrict__ loss, const AdamState ad) {
    wait_previous();
    if (blockIdx.x == gridDim.x - 1) {
        loss_of_terms(colp, terms, B, k, lw, loss);
        return;
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < static_cast<int>(kMlpParamCount)) {
        float s = 0.0f;
        #pragma unroll 8
        for (int c = 0; c < C; ++c) s += part[static_cast<size_t>(c) * kMlpParamCount + i];
        if constexpr (ADAM) {
            const float mi = 0.9f * ad.m[i] + 0.1f * s;
            const float vi = 0.999f * ad.v[i] + 0.001f * s * s;
            ad.m[i] = mi;
            ad.v[i] = vi;
            const float p = ad.p[i] - ad.lr * (mi / ad.c1) / (sqrtf(vi / ad.c2) + 1e-8f);
            ad.p[i] = p;
            const int w2 = i - (kMlpHidden * kMlpIn + kMlpHidden);
            if (i < kMlpHidden * kMlpIn)
                ad.w1t[(i % kMlpIn) * kMlpHidden + i / kMlpIn] = __float2bfloat16_rn(p);
            else if (w2 >= 0 && w2 < k * kMlpHidden)
                ad.w2b[w2] = __float2bfloat16_rn(p);
        } else {
            g[i] = s;
        }
    }
}

// FP32 masters -> BF16 weights: W1 as it is (w1b) or transposed (w1t), W2, and biases.
__global__ void mlp_export_kernel(const float* w1, const float* b1,
                                  const float* w2, const float* b2, int k,
                                  __nv_bfloat16* __restrict__ w1b, __nv_bfloat16* __restrict__ w1t,
                                  __nv_bfloat16* __restrict__ w2b, float* __restrict__ b1o, float* __restrict__ b2o) {
    wait_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kMlpHidden * kMlpIn) {
        if (w1b) w1b[i] = __float2bfloat16_rn(w1[i]);
        if (w1t) w1t[i] = __float2bfloat16_rn(w1[(i % kMlpHidden) * kMlpIn + i / kMlpHidden]);
    }
    if (i < k * kMlpHidden) w2b[i] = __float2bfloat16_rn(w2[i]);
    if (b1o && i < kMlpHidden) b1o[i] = b1[i];
    if (b2o && i < k) b2o[i] = b2[i];
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Thread per 16-byte chunk of the 3B gathered rows.
__global__ void mlp_gather_kernel(const uint8_t* __restrict__ tq, int t_n, const int32_t* __restrict__ nn,
                                  const uint8_t* __restrict__ base, int r_n, int B, unsigned long long seed, int step,
                                  uint8_t* __restrict__ x) {
    const long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (e >= 3LL * B * 8) return;
    const int row = static_cast<int>(e >> 3), c = static_cast<int>(e & 7);
    const int i = row % B, part = row / B;
    const unsigned long long h = mix64(seed ^ (static_cast<unsigned long long>(step) << 32) ^
                                       (static_cast<unsigned long long>(i) * 0x632BE59BD9B4E019ull));
    const int qi = static_cast<int>(h % static_cast<unsigned long long>(t_n));
    const uint8_t* src;
    if (part == 0) {
        src = tq + static_cast<size_t>(qi) * kMlpIn;
    } else if (part == 1) {
        src = base + static_cast<size_t>(nn[2 * qi]) * kMlpIn;
    } else {
        const int ri = static_cast<int>(mix64(h) % static_cast<unsigned long long>(r_n));
        src = base + static_cast<size_t>(ri) * kMlpIn;
    }
    reinterpret_cast<uint4*>(x + static_cast<size_t>(row) * kMlpIn)[c] = reinterpret_cast<const uint4*>(src)[c];
}

}  // namespace

MlpParams mlp_params_at(float* base) {
    MlpParams p;
    p.w1 = base;
    p.b1 = p.w1 + kMlpHidden * kMlpIn;
    p.w2 = p.b1 + kMlpHidden;
    p.b2 = p.w2 + kMlpOutRows * kMlpHidden;
    return p;
}

int mlp_fwd_blocks(int R) { return (R + kFwdRows - 1) / kFwdRows; }

// One block per SM (4 column blocks x (36 chunks and the loss role)), at least 8 pairs per chunk.
int mlp_bwd_chunks(int B) { return std::max(1, std::min(kBwdMaxChunks, B / 8)); }

size_t mlp_train_bytes(int B) {
    const size_t R = 3 * static_cast<size_t>(B), C = static_cast<size_t>(mlp_bwd_chunks(B));
    return 4 * (R * (kMlpHidden + kMlpOutRows) + 32 * static_cast<size_t>(mlp_fwd_blocks(3 * B)) + 32 * 32 +
                C * kMlpParamCount + 2 * static_cast<size_t>(B));
}

MlpTrainBufs mlp_train_bufs_at(char* base, int B) {
    const size_t R = 3 * static_cast<size_t>(B), C = static_cast<size_t>(mlp_bwd_chunks(B));
    MlpTrainBufs tb;
    tb.h = reinterpret_cast<float*>(base);  // every array starts on a multiple of 32 floats
    tb.t = tb.h + R * kMlpHidden;
    tb.colpart = tb.t + R * kMlpOutRows;
    tb.colp = tb.colpart + 32 * static_cast<size_t>(mlp_fwd_blocks(3 * B));
    tb.part = tb.colp + 32 * 32;
    tb.terms = tb.part + C * kMlpParamCount;
    return tb;
}

namespace {

cudaError_t launch_fwd_bwd(const uint8_t* x, int B, int k, const MlpParams& p, const __nv_bfloat16* w1t,
                           const __nv_bfloat16* w2b, const MlpLossWeights& lw, const MlpTrainBufs& tb,
                           cudaStream_t stream) {
    if (B <= 0 || k < 1 || k > kMlpMaxBits) return cudaErrorInvalidValue;
    const int R = 3 * B, blocks = mlp_fwd_blocks(R);
    cudaError_t e = cudaFuncSetAttribute(mlp_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kFwdSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kBwdSmem));
    if (e != cudaSuccess) return e;
    e = launch_after(mlp_fwd_kernel, blocks, kFwdThreads, kFwdSmem, stream, x, R, w1t, p.b1, w2b, p.b2, k, tb.h, tb.t,
                     tb.colpart);
    if (e != cudaSuccess) return e;
    return launch_after(mlp_bwd_kernel, dim3(kBwdColBlocks, mlp_bwd_chunks(B) + 1), kBwdThreads, kBwdSmem, stream, x, B,
                        k, tb.h, tb.t, w2b, lw, tb.colpart, blocks, tb.colp, tb.terms, tb.part);
}

constexpr int kReduceBlocks = static_cast<int>((kMlpParamCount + 255) / 256) + 1;  // + the loss

}  // namespace

cudaError_t launch_mlp_loss_grad(const uint8_t* x, int B, int k, const MlpParams& p, const __nv_bfloat16* w1t,
                                 const __nv_bfloat16* w2b, const MlpLossWeights& lw, const MlpTrainBufs& tb,
                                 const MlpParams& g, float* loss, cudaStream_t stream) {
    const cudaError_t e = launch_fwd_bwd(x, B, k, p, w1t, w2b, lw, tb, stream);
    if (e != cudaSuccess) return e;
    return launch_after(mlp_reduce_kernel<false>, kReduceBlocks, 256, 0, stream, tb.part, mlp_bwd_chunks(B), tb.colp,
                        tb.terms, B, k, lw, g.w1, loss, AdamState{});
}

cudaError_t launch_mlp_train_step(const uint8_t* x, int B, int k, const MlpParams& p, const MlpParams& m,
                                  const MlpParams& v, __nv_bfloat16* w1t, __nv_bfloat16* w2b,
                                  const MlpLossWeights& lw, const MlpTrainBufs& tb, int step, float lr, float* loss,
                                  cudaStream_t stream) {
    const cudaError_t e = launch_fwd_bwd(x, B, k, p, w1t, w2b, lw, tb, stream);
    if (e != cudaSuccess) return e;
    const float c1 = 1.0f - powf(0.9f, static_cast<float>(step));
    const float c2 = 1.0f - powf(0.999f, static_cast<float>(step));
    return launch_after(mlp_reduce_kernel<true>, kReduceBlocks, 256, 0, stream, tb.part, mlp_bwd_chunks(B), tb.colp,
                        tb.terms, B, k, lw, nullptr, loss, AdamState{p.w1, m.w1, v.w1, w1t, w2b, lr, c1, c2});
}

cudaError_t launch_mlp_export(const MlpParams& p, int k, __nv_bfloat16* w1b, __nv_bfloat16* w1t, __nv_bfloat16* w2b,
                              float* b1_out, float* b2_out, cudaStream_t stream) {
    mlp_export_kernel<<<(kMlpHidden * kMlpIn + 255) / 256, 256, 0, stream>>>(p.w1, p.b1, p.w2, p.b2, k, w1b, w1t, w2b,
                                                                          b1_out, b2_out);
    return cudaGetLastError();
}

cudaError_t launch_mlp_gather(const uint8_t* tq, int t_n, const int32_t* nn, const uint8_t* base, int r_n, int B,
                              unsigned long long seed, int step, uint8_t* x, cudaStream_t stream) {
    const long long items = 3LL * B * 8;
    mlp_gather_kernel<<<static_cast<unsigned>((items + 255) / 256), 256, 0, stream>>>(tq, t_n, nn, base, r_n, B, seed,
                                                                                    step, x);
    return cudaGetLastError();
}

}  // namespace sift
