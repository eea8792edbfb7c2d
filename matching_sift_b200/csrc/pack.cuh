#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace sift {

// Survey of descriptor values, accumulated into stats[0..2] (caller zeroes
// them first):
//   stats[0]  flags below
//   stats[1]  OR of v * 2^24 as unsigned integers (meaningless with kValueNotFixed)
//   stats[2]  bit pattern of the largest |value| (as a float; meaningless with
//             kValueNotFinite)
// With shift s = value_shift(stats[1]) (the smallest s >= 0 that makes every
// v * 2^s an integer) the values suit the integer kernels when kValueNotFixed is
// not set and the largest value times 2^s is at most 255.
enum ValueFlags : uint32_t {
    kValueNotU8 = 1,      // some value is not an integer in [0, 255]
    kValueNotFixed = 2,   // some value is not in [0, 256) or not a multiple of 2^-24
    kValueNotFinite = 4,  // some value is infinite, NaN or above 3.0e38 in magnitude
};
int value_shift(uint32_t bits);

// The survey of q_rows + r_rows rows of 128 floats or halves (16-byte aligned)
// and, where out pointers are given, their u8 form (meaningful when kValueNotU8
// is not set).
cudaError_t launch_survey(const void* q, size_t q_rows, const void* r, size_t r_rows, bool half, uint8_t* q_out,
                          uint8_t* r_out, int* stats, int num_sms, cudaStream_t stream);
// Values times mul (a power of two; products known to be integers in [0, 255]) as u8.
cudaError_t launch_pack_u8(const void* q, size_t q_rows, const void* r, size_t r_rows, bool half, float mul,
                           uint8_t* q_out, uint8_t* r_out, int num_sms, cudaStream_t stream);

// FP16 rows in one pass: the survey, base-tile records of float norms (as
// launch_row_norms_float; padding rows kFloatKeyPad), query norms
// (float bit patterns) and cleared bounds thresh[2 q_pad].
cudaError_t launch_survey_norms_f16(const void* r, int r_n, int base_tiles, int metric, int32_t* rec, const void* q,
                                    int q_n, int q_pad, int32_t* qnorm, int32_t* thresh, int* stats,
                                    cudaStream_t stream);

// Float rows -> split FP16 rows (16-byte aligned, [rows][256]): halves [0, 128)
// = hi = fp16(x * mul), [128, 256) = lo = fp16(x * mul - hi), mul a power of two
// chosen so that the largest |x * mul| stays below the FP16 range; with the
// records, query norms and cleared bounds of launch_row_norms_float.
cudaError_t launch_split_norms_f32(const float* r, int r_n, int r_pad, int metric, void* r_out, int32_t* rec,
                                   const float* q, int q_n, int q_pad, void* q_out, int32_t* qnorm, int32_t* thresh,
                                   float mul, cudaStream_t stream);

}  // namespace sift
