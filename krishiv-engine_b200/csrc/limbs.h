// limbs.h -- sums kept in 32-bit words, each updated by an atomic of its own.
// Plain C++: a host program adds with plain words, a kernel with atomics.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define KRV_HD __host__ __device__ __forceinline__
#else
#define KRV_HD inline
#endif

namespace krv {

// Adds x to a signed sum of 96 bits in words 0 (lowest) to 2. add(w, v) adds v
// to word w, modulo 2^32, and returns what the word held. Every addition's
// carry goes up with it, so the sum is exact once all have finished, in any
// order, modulo 2^96. Returned: 1 or -1 when this addition took the top word
// past its end, that is when 2^96 or -2^96 belongs to the sum beside its words;
// 0 otherwise.
template <class Add> KRV_HD int sum96_add(const Add &add, int64_t x) {
    const uint32_t x0 = (uint32_t)x;
    const uint32_t o0 = add(0, x0);
    const uint64_t a1 = (uint64_t)(uint32_t)((uint64_t)x >> 32) + (o0 + x0 < o0 ? 1u : 0u);
    uint32_t a2 = (x < 0 ? 0xFFFFFFFFu : 0u) + (uint32_t)(a1 >> 32);
    const uint32_t x1 = (uint32_t)a1;
    if (x1) {
        const uint32_t o1 = add(1, x1);
        a2 += o1 + x1 < o1 ? 1u : 0u;
    }
    if (!a2) return 0;
    const uint32_t o2 = add(2, a2), n2 = o2 + a2;
    if (!((~(o2 ^ a2) & (o2 ^ n2)) >> 31)) return 0;
    return (a2 >> 31) ? -1 : 1;
}

}  // namespace krv
