// f3.cuh -- sums in three FP32 terms, for places whose sums were FP64 and whose number of terms makes
// the FP64 pipe (about 2 lanes per clock and SM) the bound.  A value is the unevaluated a + b + c; two
// levels of Knuth's TwoSum (exact for any operands short of overflow) collect the rounding errors, so
// only the additions to c round, at about 2^-72 of the largest partial sum: closer than FP64's 2^-53,
// at 13 FP32 additions per term and 19 per pair.  A sum that may leave the FP32 range, and infinities,
// need FP64: a is then not finite (or is checked before).
#pragma once

#ifdef __CUDACC__
#define PASC_HD __host__ __device__ __forceinline__
#else
#define PASC_HD inline
#endif

namespace pasc {

struct F3 {
    float a, b, c;
};

PASC_HD float f3_two_sum(float x, float y, float &e)
{
    const float s = x + y, yv = s - x, xv = s - yv;
    e = (x - xv) + (y - yv);
    return s;
}

PASC_HD F3 f3_add(F3 x, float v)
{
    float e1, e2;
    const float a = f3_two_sum(x.a, v, e1), b = f3_two_sum(x.b, e1, e2);
    return F3{a, b, x.c + e2};
}

PASC_HD F3 f3_add(F3 x, F3 y)
{
    float e1, e2, e3;
    const float a = f3_two_sum(x.a, y.a, e1), s = f3_two_sum(x.b, y.b, e2), b = f3_two_sum(s, e1, e3);
    return F3{a, b, (x.c + y.c) + (e2 + e3)};
}

PASC_HD double f3_value(F3 x) { return (double)x.a + ((double)x.b + (double)x.c); }

#ifdef __CUDACC__
__device__ __forceinline__ F3 f3_shfl_xor(F3 x, int m)
{
    return F3{__shfl_xor_sync(0xffffffffu, x.a, m), __shfl_xor_sync(0xffffffffu, x.b, m),
              __shfl_xor_sync(0xffffffffu, x.c, m)};
}

// Sums of N values over a warp: while a lane carries more than one value, a step halves their
// number instead of adding all of them.  The sum of value f3_lane_value<N0>(lane) is in v[0].
template <int N, int OFF = 16, int N0>
__device__ __forceinline__ void f3_warp_sum(F3 (&v)[N0], int lane)
{
    if constexpr (OFF >= 1) {
        constexpr int H = (N + 1) / 2;
        const bool up = N > 1 && (lane & OFF);
#pragma unroll
        for (int j = 0; j < H; j++) {
            const F3 w = N > 1 && H + j < N ? v[H + j < N0 ? H + j : 0] : F3{0.f, 0.f, 0.f};
            const F3 keep = up ? w : v[j], give = N > 1 ? (up ? v[j] : w) : v[j];
            v[j] = f3_add(keep, f3_shfl_xor(give, OFF));
        }
        f3_warp_sum<H, OFF / 2>(v, lane);
    }
}

// which of N0 values a lane's v[0] is the sum of; -1: none, or one that another lane has too
template <int N0>
__device__ __forceinline__ int f3_lane_value(int lane)
{
    static_assert(N0 <= 32, "one value per lane at most");
    int n = N0, q = 0, have = N0;  // have: of the lane's n values those that are not padding
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const int h = (n + 1) / 2;
        if (lane & off) {
            if (n == 1) return -1;
            q += h;
            have -= h;
        } else if (have > h) {
            have = h;
        }
        n = h;
    }
    return have >= 1 ? q : -1;
}
#endif

}  // namespace pasc
