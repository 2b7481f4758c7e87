// Handing partial results from one CTA of a launch to another through L2 without flags, tickets or fences: a word is
// kNothing until its value has been written, so a reader knows the value by its being there, in one trip.  The reader
// leaves kNothing behind for the next launch.  Store to use takes about 1.2 us; with a fence and a flag or a ticket 3 to 4.
//
// Who may wait: a CTA for those that started before it, or for what another's first piece of work is.  That CTAs of lower
// index start first is an assumption: GPUs deal them out so, CUDA does not promise it.  Were it otherwise, CTAs that wait
// could keep those they wait for from starting.  So waits are bounded, about a second and once a thread; then the error
// word is set, the kernel ends, and the words stay out of use until the host has emptied them (tcx_take_device_error).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace tcb {
namespace handover {

constexpr uint32_t kNothing = 0xFFFFFFFFu;      // a NaN; a value with these bits is stored as another NaN

__device__ __forceinline__ uint32_t word_of(float v) {
    const uint32_t w = __float_as_uint(v);
    return w == kNothing ? 0x7FFFFFFFu : w;
}
__device__ __forceinline__ void store(uint32_t* dst, uint32_t w) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(dst), "r"(w) : "memory");
}
__device__ __forceinline__ uint32_t load(const uint32_t* src) {
    uint32_t w;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(w) : "l"(src) : "memory");
    return w;
}
__device__ __forceinline__ void store4(uint32_t* dst, uint4 w) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w) : "memory");
}
__device__ __forceinline__ uint4 load4(const uint32_t* src) {
    uint4 w;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "l"(src) : "memory");
    return w;
}
__device__ __forceinline__ bool there(uint32_t w) { return w != kNothing; }
__device__ __forceinline__ bool there(const uint4& w) { return there(w.x) && there(w.y) && there(w.z) && there(w.w); }

}  // namespace handover
}  // namespace tcb
