// Arithmetic shared by the matrix attention kernels (attention.cu, attention_tc.cu).
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace tcb {
namespace attn {

// The product with V takes a probability p in (0, 1] as two fp16 numbers.  As it stands fp16 ends at 2^-24, and
// probabilities below that would be lost to the output while the row sum still counts them; so exponentials
// are carried 2^15 times as large, the largest fp16 power of two, and the factor is taken out of the row's sum and
// output at the end (exactly: a power of two).  The two numbers then hold p to 21 bits down to 2^-17 and
// to 2^-40 below: 8192 keys of any size leave out less than 2^-27 of the largest.
constexpr float kProbScale = 32768.0f, kProbUnscale = 1.0f / 32768.0f;

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
// Two scaled probabilities as fp16 pairs hi + lo.  hi is rounded towards zero and lo is at least the smallest
// fp16 number where hi is not zero: neither is negative and no lo of zero meets an infinity, so an infinite
// value under a visible key makes the result infinite, as one multiplication would, and not NaN.
__device__ __forceinline__ void split_h2(float a, float b, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(b), "f"(a));
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
    uint32_t least;                          // 1, the smallest fp16 number, where hi is not zero
    asm("min.u16x2 %0, %1, %2;" : "=r"(least) : "r"(hi), "r"(0x00010001u));
    asm("max.u16x2 %0, %1, %2;" : "=r"(lo) : "r"(pack_h2(a - f.x, b - f.y)), "r"(least));
}

}  // namespace attn
}  // namespace tcb
