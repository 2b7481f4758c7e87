// Arithmetic shared by the matrix attention kernels (attention.cu, attention_tc.cu).
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace tcb {
namespace attn {

// The product with V takes a probability p in (0, 1] as two fp16 numbers, hi + lo.
//
// As it stands fp16 ends at 2^-24, and probabilities below that would be lost to the output while the row sum still
// counts them; so exponentials are carried 2^15 times as large, the largest fp16 power of two, and the factor
// is taken out of the row's sum and output at the end (exactly: a power of two).  The two numbers then hold p to 21
// bits down to 2^-17 and to 2^-40 below: 8192 keys of any size leave out less than 2^-27 of the largest.
//
// Neither number is negative, and lo is not zero for a p above 2^-26: an infinite value under a visible key makes the
// result infinite, as one multiplication would, and not NaN (infinity minus infinity, zero times infinity).  hi is
// rounded towards zero, and lo holds the remainder of p (1 + 2^-14); that factor, too, comes out of the output.
// (Raising a lo of zero to the smallest fp16 number takes two instructions a pair: 2048 x 2048, 32 heads 162 us
// against 155 so.)
constexpr float kProbScale = 32768.0f, kProbUnscale = 1.0f / 32768.0f;
constexpr float kGrow = 1.0f + 1.0f / 16384.0f, kUngrow = 16384.0f / 16385.0f;

// a *= k and b *= k, one instruction.
__device__ __forceinline__ void scale2(float& a, float& b, float k) {
    asm("{\n\t.reg .b64 v, w;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 w, {%2, %2};\n\tmul.rn.f32x2 v, v, w;\n\tmov.b64 {%0, %1}, v;\n\t}"
        : "+f"(a), "+f"(b) : "f"(k));
}
// exp(x); exponentials below the normal range are zero.
__device__ __forceinline__ float exp_of(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
    return y;
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Two scaled probabilities as fp16 pairs hi + lo.
__device__ __forceinline__ void split_h2(float a, float b, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(b), "f"(a));
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
    lo = pack_h2(fmaf(a, kGrow, -f.x), fmaf(b, kGrow, -f.y));
}

}  // namespace attn
}  // namespace tcb
