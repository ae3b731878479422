// project64.cuh -- the FP64 projection in the reference's order (project_ref_f64), K at compile time
// and sparing the part's slow FP64 pipe: values are sorted and compared as integer keys, the
// division by K - i is its reciprocal with one correction, and the scan ends with the threshold.
// Bit for bit project_ref_f64.
#pragma once

#include "common.cuh"
#include "project.cuh"
#include "sweep_common.cuh"

namespace pasc {

static __device__ __noinline__ void project_f64_any(double *x, int K)
{
    double y[KMAX_FUSED];
    project_ref_f64(x, K, y);
}

// v / N rounded to nearest: the quotient by the rounded reciprocal, corrected once (Markstein)
template <int N>
__device__ __forceinline__ double div_const(double v)
{
    if constexpr ((N & (N - 1)) == 0) {
        return __dmul_rn(v, 1.0 / N);  // exact
    } else {
        constexpr double rec = 1.0 / N;
        const double q = __dmul_rn(v, rec);
        return fma(fma(-(double)N, q, v), rec, q);
    }
}

// t_hat candidates i = I .. 1 of the scan; y sorted ascending
template <int K, int I>
__device__ __forceinline__ void scan_f64(const double (&y)[K], double &t, bool &found)
{
    if constexpr (I >= 1) {
        if (!found) {
            double s = y[I];  // (0.0 + y_i is y_i)
#pragma unroll
            for (int j = I + 1; j < K; j++) s = __dadd_rn(s, y[j]);
            const double ti = div_const<K - I>(__dadd_rn(s, -1.0));
            if (fs_key(ti) >= fs_key(y[I - 1])) {
                t = ti;
                found = true;
            }
        }
        scan_f64<K, I - 1>(y, t, found);
    }
}

template <int K>
__device__ __forceinline__ void project_f64(double (&x)[K])
{
    bool inside = true;
    double sum = x[0];
#pragma unroll
    for (int k = 1; k < K; k++) sum = __dadd_rn(sum, x[k]);
    if (((__double2hiint(sum) >> 20) & 0x7ff) == 0x7ff) {  // infinities or NaN: the reference's own comparisons
        project_f64_any(x, K);
        return;
    }
#pragma unroll
    for (int k = 0; k < K; k++) inside &= fs_key(x[k]) >= -1;  // -0.0 (key -1) is not below 0
    if (inside && __double_as_longlong(sum) == __double_as_longlong(1.0)) return;
    double y[K];
#pragma unroll
    for (int k = 0; k < K; k++) y[k] = x[k];
#pragma unroll
    for (int r = 0; r < K; r++) {
#pragma unroll
        for (int a = (r & 1); a + 1 < K; a += 2) {
            const bool sw = fs_key(y[a + 1]) < fs_key(y[a]);
            const double lo = sw ? y[a + 1] : y[a], hi = sw ? y[a] : y[a + 1];
            y[a] = lo;
            y[a + 1] = hi;
        }
    }
    double t = 0.0;
    bool found = false;
    scan_f64<K, K - 1>(y, t, found);
    if (!found) t = div_const<K>(__dadd_rn(sum, -1.0));
#pragma unroll
    for (int k = 0; k < K; k++) {
        const double v = __dadd_rn(x[k], -t);
        x[k] = __double2hiint(v) < 0 ? 0.0 : v;
    }
}

}  // namespace pasc
