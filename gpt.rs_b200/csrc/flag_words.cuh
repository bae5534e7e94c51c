// What the CTAs of a single-kernel decode step hand to each other: words {value, flag} of 64 bits in global memory, written and read with
// single accesses. The reader polls the data itself, so an exchange is one store and one load through L2. An arrival with its fence, a
// polled counter and the load behind it are three round trips (148 CTAs, a vector of 3072 bf16 read by all: 1.3 us against 2.0; 21504: 2.4
// against 3.4). A flag is the number of the step and layer; every buffer has one writer per word and is written again only after every
// reader's own output of that layer has been consumed.
#pragma once

#include "common.cuh"

namespace gptrs {

struct FlagWords { uint64_t a, b; };

__device__ __forceinline__ void put_word(void* p, uint32_t v, uint32_t flag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;\n" ::"l"(p), "l"(((uint64_t)flag << 32) | v) : "memory");
}
__device__ __forceinline__ void put_words(void* p, uint32_t v0, uint32_t v1, uint32_t flag) {   // two neighbours, 16-byte aligned
    const uint64_t f = (uint64_t)flag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};\n" ::"l"(p), "l"(f | v0), "l"(f | v1) : "memory");
}
__device__ __forceinline__ uint64_t peek_word(const void* p) {
    uint64_t w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];\n" : "=l"(w) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ FlagWords peek_words(const void* p) {
    FlagWords w;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];\n" : "=l"(w.a), "=l"(w.b) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ bool has_flag(uint64_t w, uint32_t flag) { return (uint32_t)(w >> 32) == flag; }
__device__ __forceinline__ bool has_flag(const FlagWords& w, uint32_t flag) { return has_flag(w.a, flag) && has_flag(w.b, flag); }
__device__ __forceinline__ float word_f32(uint64_t w) { return __uint_as_float((uint32_t)w); }

// A thread's waits, `while (!found && wait.again())`: bounded over the whole step, after the first one that gave up (status 5) none waits any
// more. Where many threads wait for neighbouring words, one lane of a warp asks first (wait_word): with every lane asking for its own, the
// requests for a few hot lines delay everything else.
struct FlagWaiter {
    uint32_t left;
    int* status;
    __device__ __forceinline__ bool again() {
        if (left == 0) return false;
        if (--left == 0) { atomicExch(status, 5); return false; }
        __nanosleep(20);
        return true;
    }
    __device__ __forceinline__ uint32_t wait_word(const void* p, uint32_t flag) {
        uint64_t w;
#pragma unroll 1
        do w = peek_word(p); while (!has_flag(w, flag) && again());
        return (uint32_t)w;
    }
    __device__ __forceinline__ FlagWords wait_words(const void* p, uint32_t flag) {
        FlagWords w;
#pragma unroll 1
        do w = peek_words(p); while (!has_flag(w, flag) && again());
        return w;
    }
};
constexpr uint32_t kFlagPolls = 1u << 23;   // of a thread, over the whole step
// Polls of a wait on a barrier, of a thread's waits for words, and the test switch of gptrs_cuda_debug_matmul_fault (quant_step.cu).
void step_wait_limits(uint32_t* spin_limit, uint32_t* flag_polls, int* starve);

}  // namespace gptrs
