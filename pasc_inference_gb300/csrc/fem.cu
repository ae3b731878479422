// fem.cu -- FEM temporal coarsening (GraphH1FEMModel with fem_reduce < 1): the gamma QP is
// solved on T2 = ceil(T*fem_reduce) timesteps; gamma and the residual are reduced onto the
// coarse grid before the solve and the solution is prolongated back after it.
//
//   type 0, FEM-SUM (src/petscvector/common/fem.cpp:32-115, 124-210): diff = T1/T2; coarse t2
//     sums the fine t in [round(t2*diff), round((t2+1)*diff)); prolongation copies it back.
//   type 1, FEM-HAT (src/petscvector/common/femhat.cpp:27-215, include/general/common/
//     femhat.h:154-195): diff = (T1-1)/(T2-1); reduction weights the fine values by the hat
//     function centred at t2*diff (the reference's loop bounds, which start at floor of the
//     hat's left end, kept as they are); prolongation interpolates linearly between the two
//     coarse neighbours (a neighbour past the last coarse point counts as 0).
// One thread per (coarse or fine timestep, cluster); the index arithmetic is FP64 with the
// reference's expressions and no contraction, so the block bounds are the reference's.  (The
// reference's own CUDA FEM kernels are declared under other names than the ones it calls and
// do not link; its sequential code defines the behaviour restated here.)
#include <math.h>

#include "common.cuh"
#include "f3.cuh"
#include "internal.h"
#include "launch_rules.h"

namespace pasc {

__device__ __forceinline__ double fem_mul(long a, double b) { return __dmul_rn((double)a, b); }

// value of the fine field at (t, k): a stored field, or the residual (x_t - theta_k)^2
template <typename TIn>
struct FineField {
    const TIn *g;          // T1*K, or null
    const double *data;    // T1 (residual form)
    const double *theta;   // K
    int K;
    __device__ __forceinline__ double operator()(long t, int k) const
    {
        if (g) return (double)g[t * K + k];
        const double r = data[t] - theta[k];
        return r * r;
    }
};

template <typename TIn, typename TOut>
__global__ void fem_reduce_kernel(FineField<TIn> f, TOut *g2, long T1, long T2, int K, int type, double diff,
                                  long right_t1_idx, double scale)
{
    const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (idx >= T2 * K) return;
    const long t2 = idx / K;
    const int k = (int)(idx - t2 * K);
    double mysum = 0.0;
    if (type == 0) {
        const long lo = (long)round(fem_mul(t2, diff)), hi = (long)round(fem_mul(t2 + 1, diff));
        for (long i = lo; i < hi; i++) mysum = __dadd_rn(mysum, f(i, k));
    } else {
        const double center = fem_mul(t2, diff), left = fem_mul(t2 - 1, diff), right = fem_mul(t2 + 1, diff);
        long t1 = (long)floor(left), id = t1;
        while ((double)t1 <= center) {
            const double phi = __ddiv_rn(__dsub_rn((double)t1, left), __dsub_rn(center, left));
            if (id >= 0) mysum = __dadd_rn(mysum, __dmul_rn(phi, f(id, k)));
            t1 += 1;
            id += 1;
        }
        while ((double)t1 < right) {
            const double phi = __ddiv_rn(__dsub_rn((double)t1, right), __dsub_rn(center, right));
            if (id < right_t1_idx) mysum = __dadd_rn(mysum, __dmul_rn(phi, f(id, k)));
            t1 += 1;
            id += 1;
        }
    }
    g2[idx] = (TOut)__dmul_rn(mysum, scale);
}

template <typename TIn, typename TOut>
__global__ void fem_prolongate_kernel(const TIn *g2, TOut *g1, long T1, long T2, int K, int type, double diff)
{
    if (type == 0) {
        // one thread per coarse (t2, k), writing its block
        const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
        if (idx >= T2 * K) return;
        const long t2 = idx / K;
        const int k = (int)(idx - t2 * K);
        const long lo = (long)round(fem_mul(t2, diff)), hi = (long)round(fem_mul(t2 + 1, diff));
        const TIn v = g2[idx];
        for (long i = lo; i < hi; i++) g1[i * K + k] = (TOut)v;
        return;
    }
    const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (idx >= T1 * K) return;
    const long t1 = idx / K;
    const int k = (int)(idx - t1 * K);
    const long l = (long)floor(__ddiv_rn((double)t1, diff)), r = l + 1;
    const double t1_left = fem_mul(l, diff), t1_right = fem_mul(r, diff);
    const double phi_l = __ddiv_rn(__dsub_rn((double)t1, t1_left), __dsub_rn(t1_right, t1_left));
    const double phi_r = __ddiv_rn(__dsub_rn((double)t1, t1_right), __dsub_rn(t1_left, t1_right));
    const double gr = r < T2 ? (double)g2[r * K + k] : 0.0;
    const double gl = l < T2 ? (double)g2[l * K + k] : 0.0;
    double v = 0.0;
    v = __dadd_rn(v, __dmul_rn(phi_l, gr));
    v = __dadd_rn(v, __dmul_rn(phi_r, gl));
    g1[idx] = (TOut)v;
}

// ---- FEM-SUM of the mixed path ----
// (Signals that fem_sum_indexable accepts.)
// lo[j]: the first fine timestep of coarse timestep j (lo[T2] = T1), computed once when the
// reduction is set up: the FP64 rounding of the reference's expressions costs as much as the sums.
// The fine field is read, and the prolongated one written, in consecutive order.  Sums: an FP32
// field in three FP32 terms (f3.cuh), which hold more than FP64 does, with FP64 where they leave the
// FP32 range; the residual in FP64 with three instead of 3K operations per fine timestep,
//     sum (x_t - theta_k)^2 = S2 - 2 e S1 + n e^2,   S1 = sum (x_t - c), S2 = sum (x_t - c)^2, e = theta_k - c
// with c the block's first value.  c is one of the summands, so S2 is at most 2 + 2n times the sum:
// where the first value lies far from all others that is n digits' worth of cancellation, and
// infinities give inf - inf.  Where the sum is below 2^-8 of S2 (c some 16 standard deviations off) or not a
// number it is therefore taken term by term; elsewhere at most 11 of FP64's 53 bits are lost of a sum that
// is stored in 24.
// Both reductions at T = 2e6, K = 3, one thread per coarse entry summing in FP64 with a stride of K / float-float
// sums / here: T2 = T/10 95 / 42 / 41 us, T2 = T/2 180 / 89 / 75.  The copy back: 15.
constexpr int FEM_NT = (int)FEM_SUM_THREADS;

__global__ void __launch_bounds__(FEM_NT) fem_bounds_kernel(int *lo, long T2, double diff)
{
    const long j = (long)blockIdx.x * FEM_NT + threadIdx.x;
    if (j <= T2) lo[j] = (int)(long)round(fem_mul(j, diff));
}

__global__ void __launch_bounds__(FEM_NT) fem_sum_field_kernel(const float *__restrict__ g1, float *__restrict__ g2,
                                                               const int *__restrict__ lo, unsigned int n, int K, double scale)
{
    const unsigned int e = blockIdx.x * FEM_NT + threadIdx.x;
    if (e >= n) return;
    const unsigned int j = e / (unsigned int)K;
    const int k = (int)(e - j * K);
    const int hi = lo[j + 1];
    F3 s{0.f, 0.f, 0.f};
#pragma unroll 8
    for (int i = lo[j]; i < hi; i++) s = f3_add(s, __ldg(g1 + (long)i * K + k));
    if (scale == 1.0 && isfinite(s.a)) {  // gamma: the nearest FP32 number, off the FP64 pipe
        float r;
        const float h = f3_two_sum(s.a, s.b, r);
        g2[e] = h + (r + s.c);
        return;
    }
    double sum = f3_value(s);
    if (!isfinite(s.a)) {  // beyond the FP32 range, or a value that is not finite
        sum = 0.0;
        for (int i = lo[j]; i < hi; i++) sum = __dadd_rn(sum, (double)__ldg(g1 + (long)i * K + k));
    }
    g2[e] = (float)__dmul_rn(sum, scale);
}

template <int K>
__global__ void __launch_bounds__(FEM_NT) fem_sum_residual_kernel(const double *__restrict__ data,
                                                                  const double *__restrict__ theta, float *__restrict__ g2,
                                                                  const int *__restrict__ lo, int T2, double scale)
{
    const int j = blockIdx.x * FEM_NT + threadIdx.x;
    if (j >= T2) return;
    const int a = lo[j], b = lo[j + 1];
    const double c = a < b ? data[a] : 0.0;
    double u = 0.0, v = 0.0;
#pragma unroll 4
    for (int i = a; i < b; i++) {
        const double d = data[i] - c;
        u += d;
        v = fma(d, d, v);
    }
    const double n = (double)(b - a), u2 = -2.0 * u;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const double d = theta[k] - c;
        double sum = fma(d, fma(n, d, u2), v);
        if (!(sum >= 0x1p-8 * v)) {  // (also where it is NaN)
            sum = 0.0;
            for (int i = a; i < b; i++) {
                const double r = data[i] - theta[k];
                sum = __dadd_rn(sum, __dmul_rn(r, r));
            }
        }
        g2[(long)j * K + k] = (float)__dmul_rn(sum, scale);
    }
}

__global__ void __launch_bounds__(FEM_NT) fem_copy_kernel(const float *__restrict__ g2, float *__restrict__ g1,
                                                          const int *__restrict__ lo, int T1, int T2, int K, double inv)
{
    const int t = blockIdx.x * FEM_NT + threadIdx.x;
    if (t >= T1) return;
    int j = (int)((double)t * inv);  // a guess, corrected by the bounds
    j = j < T2 ? j : T2 - 1;
    while (j > 0 && t < __ldg(lo + j)) j--;
    while (j < T2 - 1 && t >= __ldg(lo + j + 1)) j++;
    for (int k = 0; k < K; k++) g1[(long)t * K + k] = __ldg(g2 + (long)j * K + k);
}

cudaError_t launch_fem_bounds(int *lo, long T1, long T2, cudaStream_t s)
{
    fem_bounds_kernel<<<(unsigned int)(T2 / FEM_NT + 1), FEM_NT, 0, s>>>(lo, T2, (double)T1 / (double)T2);
    return cudaGetLastError();
}

cudaError_t launch_fem_sum_field(const float *g1, float *g2, const int *lo, long T2, int K, double scale, cudaStream_t s)
{
    const long n = T2 * K;
    fem_sum_field_kernel<<<(unsigned int)((n + FEM_NT - 1) / FEM_NT), FEM_NT, 0, s>>>(g1, g2, lo, (unsigned int)n, K, scale);
    return cudaGetLastError();
}

cudaError_t launch_fem_sum_residual(const double *data, const double *theta, float *g2, const int *lo, long T2, int K,
                                    double scale, cudaStream_t s)
{
    const unsigned int grid = (unsigned int)((T2 + FEM_NT - 1) / FEM_NT);
    switch (K) {
#define PASC_CASE(KK) \
    case KK: fem_sum_residual_kernel<KK><<<grid, FEM_NT, 0, s>>>(data, theta, g2, lo, (int)T2, scale); break;
        PASC_CASE(1) PASC_CASE(2) PASC_CASE(3) PASC_CASE(4)
        PASC_CASE(5) PASC_CASE(6) PASC_CASE(7) PASC_CASE(8)
#undef PASC_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_fem_copy(const float *g2, float *g1, const int *lo, long T1, long T2, int K, cudaStream_t s)
{
    fem_copy_kernel<<<(unsigned int)((T1 + FEM_NT - 1) / FEM_NT), FEM_NT, 0, s>>>(g2, g1, lo, (int)T1, (int)T2, K,
                                                                                 (double)T2 / (double)T1);
    return cudaGetLastError();
}

static double fem_diff(long T1, long T2, int type)
{
    return type == 0 ? (double)T1 / (double)T2 : (double)(T1 - 1) / (double)(T2 - 1);
}

static long fem_right_t1_idx(long T2, double diff) { return (long)floor(diff * (double)(T2 - 1)); }

static unsigned int fem_grid(long n) { return (unsigned int)((n + 255) / 256); }

template <typename TIn, typename TOut>
cudaError_t launch_fem_reduce(const TIn *g1, const double *data, const double *theta, TOut *g2, long T1, long T2,
                              int K, int type, double scale, cudaStream_t s)
{
    if (T2 * K == 0) return cudaSuccess;
    const double diff = fem_diff(T1, T2, type);
    FineField<TIn> f{g1, data, theta, K};
    fem_reduce_kernel<TIn, TOut><<<fem_grid(T2 * K), 256, 0, s>>>(f, g2, T1, T2, K, type, diff,
                                                                  fem_right_t1_idx(T2, diff), scale);
    return cudaGetLastError();
}

template <typename TIn, typename TOut>
cudaError_t launch_fem_prolongate(const TIn *g2, TOut *g1, long T1, long T2, int K, int type, cudaStream_t s)
{
    const double diff = fem_diff(T1, T2, type);
    const long n = type == 0 ? T2 * K : T1 * K;
    if (n == 0) return cudaSuccess;
    fem_prolongate_kernel<TIn, TOut><<<fem_grid(n), 256, 0, s>>>(g2, g1, T1, T2, K, type, diff);
    return cudaGetLastError();
}

template cudaError_t launch_fem_reduce<double, double>(const double *, const double *, const double *, double *, long,
                                                       long, int, int, double, cudaStream_t);
template cudaError_t launch_fem_reduce<float, float>(const float *, const double *, const double *, float *, long,
                                                     long, int, int, double, cudaStream_t);
template cudaError_t launch_fem_prolongate<double, double>(const double *, double *, long, long, int, int,
                                                           cudaStream_t);
template cudaError_t launch_fem_prolongate<float, float>(const float *, float *, long, long, int, int, cudaStream_t);

long fem_T_reduced(long T, double fem_reduce) { return fem_reduce < 1.0 ? (long)ceil((double)T * fem_reduce) : T; }

}  // namespace pasc

using namespace pasc;

extern "C" {

int pasc_gb300_fem_reduce_f64(const double *g1_dev, double *g2_dev, long T1, long T2, int K, int fem_type,
                              void *stream)
{
    if ((!g1_dev || !g2_dev) && T1 > 0) { record_error("fem_reduce: NULL argument"); return PASC_ERR_ARG; }
    if (T1 < 1 || T2 < 1 || T2 > T1 || K < 1 || (fem_type != 0 && fem_type != 1) || (fem_type == 1 && T2 < 2)) {
        record_error("fem_reduce: need 1 <= T2 <= T1, K >= 1, fem_type 0 or 1 (FEM-HAT: T2 >= 2)");
        return PASC_ERR_ARG;
    }
    if (launch_fem_reduce<double, double>(g1_dev, nullptr, nullptr, g2_dev, T1, T2, K, fem_type, 1.0,
                                          (cudaStream_t)stream) != cudaSuccess) {
        record_error("fem_reduce: kernel launch failed");
        return PASC_ERR_CUDA;
    }
    return PASC_OK;
}

int pasc_gb300_fem_prolongate_f64(const double *g2_dev, double *g1_dev, long T1, long T2, int K, int fem_type,
                                  void *stream)
{
    if ((!g1_dev || !g2_dev) && T1 > 0) { record_error("fem_prolongate: NULL argument"); return PASC_ERR_ARG; }
    if (T1 < 1 || T2 < 1 || T2 > T1 || K < 1 || (fem_type != 0 && fem_type != 1) || (fem_type == 1 && T2 < 2)) {
        record_error("fem_prolongate: need 1 <= T2 <= T1, K >= 1, fem_type 0 or 1 (FEM-HAT: T2 >= 2)");
        return PASC_ERR_ARG;
    }
    if (launch_fem_prolongate<double, double>(g2_dev, g1_dev, T1, T2, K, fem_type, (cudaStream_t)stream) !=
        cudaSuccess) {
        record_error("fem_prolongate: kernel launch failed");
        return PASC_ERR_CUDA;
    }
    return PASC_OK;
}

}  // extern "C"
