// grid_words.cuh -- exchange between the blocks of a cooperative launch through 64-bit words that
// carry 32 bits of payload and a tag: a word is valid when it carries the sweep's tag, so there
// is no flag, no fence and one L2 round trip.  Two sets of words alternate (tag & 1): a block
// publishes set s + 2 only after it has seen every block's set s + 1, which those published after
// reading set s.  Waits are bounded.
#pragma once

#include "common.cuh"

namespace pasc {

constexpr unsigned int WORD_WAIT_LIMIT = 1u << 22;  // polls of a word before giving up

__device__ __forceinline__ void word_store2(unsigned long long *p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void word_load2(const unsigned long long *p, unsigned long long &a, unsigned long long &b)
{
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void word_store(unsigned long long *p, unsigned long long a)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(a) : "memory");
}
__device__ __forceinline__ unsigned long long word_load(const unsigned long long *p)
{
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    return a;
}
__device__ __forceinline__ unsigned long long word_of(unsigned int v, unsigned int tag)
{
    return (unsigned long long)v | ((unsigned long long)tag << 32);
}
__device__ __forceinline__ unsigned long long word_of(float v, unsigned int tag)
{
    return word_of(__float_as_uint(v), tag);
}
__device__ __forceinline__ bool word_valid(unsigned long long w, unsigned int tag) { return (unsigned int)(w >> 32) == tag; }
__device__ __forceinline__ float word_float(unsigned long long w) { return __uint_as_float((unsigned int)w); }

// a double as two words at an even index
__device__ __forceinline__ void word_store_double(unsigned long long *p, double v, unsigned int tag)
{
    word_store2(p, word_of((unsigned int)__double2hiint(v), tag), word_of((unsigned int)__double2loint(v), tag));
}
__device__ __forceinline__ bool word_wait_double(const unsigned long long *p, unsigned int tag, double &v)
{
    for (unsigned int it = 0; it < WORD_WAIT_LIMIT; it++) {
        unsigned long long hi, lo;
        word_load2(p, hi, lo);
        if (word_valid(hi, tag) && word_valid(lo, tag)) {
            v = __hiloint2double((int)(unsigned int)hi, (int)(unsigned int)lo);
            return true;
        }
    }
    v = 0.0;
    return false;
}

// largest key over a warp (every lane gets it)
__device__ __forceinline__ long long warp_max_key(long long key)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long k = __shfl_xor_sync(0xffffffffu, key, o);
        key = k > key ? k : key;
    }
    return key;
}

}  // namespace pasc
