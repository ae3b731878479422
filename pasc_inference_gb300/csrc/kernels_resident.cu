// kernels_resident.cu -- a whole SPG solve of one signal in ONE cooperative launch, for signals
// whose state fits in the shared memory of the GPU (152 SMs x 227 KB = 34 MB: T up to about
// 1.2e6 at K = 3).
//
// The per-iteration sweeps (kernels_sweep_tma.cu) read x and the data from L2 or HBM, form
// d_{c+1} a second time to apply it, and pay a launch, a ramp of the pipeline and a grid
// reduction through one last block per iteration; below about 1e6 timesteps these fixed costs
// are most of the iteration.  Measured, us per iteration, sweeps / resident: T = 1000, K = 2 8.8 /
// 2.4; T = 1e4, K = 2 8.3 / 3.9; T = 123 457, K = 5 10.2 / 4.6; T = 1e6, K = 3 13.8 / 7.4; T =
// 4e5, K = 8 17.7 / 9.6.  What bounds it now: about 2.4 us of a block's own chain (walk of one
// group, three barriers, the sums and the step lengths), 1.4 us of exchange, and from 1e5
// timesteps on the walk's issue rate.  Here block b keeps its C timesteps for the whole solve: x, d and
// the data (MODE 1: b) stay in shared memory, so an iteration reads no HBM, needs ONE projection
// (the stored d is applied, x^{c+1} = x^c + beta d), and ends in one all-to-all exchange of the
// blocks' four partial sums.
//
//   walk      thread i owns M consecutive timesteps and walks them in groups of four (two for K >=
//             6): x^{c+1}, g^{c+1}, f, d_{c+2}, d'd, g'd and the neighbour differences of d (the
//             arithmetic, entry by entry, of the bulk-copy sweep).  Its neighbours'
//             edge values come from their shared rows, read before anyone writes.  Rows are
//             padded to an odd stride: a warp's loads at one step meet 32 banks.
//   edges     a block needs x at one timestep to its left and two to its right (the second one
//             to form the d of its right neighbour's first timestep, for the d'Ad pair that
//             crosses the blocks).  It keeps x and d of these three and advances them itself;
//             per iteration it receives their new d with the neighbours' sums.
//   exchange  every block publishes its sums (four float-float pairs) and edge values as tagged
//             words (grid_words.cuh) and polls the words of the others.  All blocks add the sums
//             in the same order and apply the reference's step rules (sweep_common.cuh) to
//             their own copy of the state.
//
// The launch is cooperative, so all blocks are resident while they wait for one another; every
// wait is bounded and one that gives up sets the state's error word (PASC_ERR_TIMEOUT).
#include <limits.h>
#include <stddef.h>
#include <algorithm>

#include "common.cuh"
#include "project.cuh"
#include "sweep_common.cuh"
#include "grid_words.cuh"
#include "internal.h"

namespace pasc {

constexpr int RES_WORDS = 8 + 3 * KMAX_FUSED;      // words of a block's slot: sums, three edge rows

// Threads of a block: up to NT that walk timesteps, and RES_MGR (the last four warps) that
// exchange the sums and keep the solver state.  Walkers per block, us per iteration: T = 1e6, K =
// 3: 512 (96 registers) 7.4, 640 (80) 7.3, but T = 1000, K = 2 2.4 to 2.5 against 2.5 and T =
// 1e4 3.9 against 4.0; T = 6e5, K = 5: 384 (128 registers) 7.5, 320 7.9; T = 4e5, K = 8: 384 9.6,
// 320 10.7.
constexpr int RES_MGR = 128;
template <int K>
struct ResShape {
    static constexpr int NT = K <= 3 ? 512 : 384;
    static constexpr int R = K <= 5 ? 4 : 2;  // timesteps of a group (as the bulk-copy sweep's threads)
};

template <int K>
struct ResSmem {
    SpgDevState st;
    float hlx[K], hld[K];        // x, d of the timestep before the block
    float hrx[2][K], hrd[2][K];  // x, d of the two after it
    float hb[K];                 // b of the first one after it
    float2 red[28][4];           // sums of the walking warps (float-float)
    float2 red2[RES_MGR / 32][4];  // sums over the blocks, per manager warp
    float beta, alpha;           // of the next sweep
    int status;
};

// Lanes hold partial sums of value lane & 3: sums over the lanes of each value.
__device__ __forceinline__ FF lane_sum4_ff(FF r)
{
#pragma unroll
    for (int m = 4; m <= 16; m <<= 1) r = ff_acc(r, ff_shfl_xor(r, m));
    return r;
}

// Sums of the four values over a warp: the first two steps halve the number of values a lane
// carries instead of adding all four (6 additions instead of 20).  Lane l returns the sum of
// value l & 3.
__device__ __forceinline__ FF warp_sum4_ff(const FF (&v)[4], int lane)
{
    const bool h1 = lane & 1, h2 = lane & 2;
    // step 1: even lanes keep values 0 and 2, odd lanes 1 and 3; step 2: lanes with bit 1 keep
    // values 2 and 3
    const FF a = ff_acc(h1 ? v[1] : v[0], ff_shfl_xor(h1 ? v[0] : v[1], 1));
    const FF b = ff_acc(h1 ? v[3] : v[2], ff_shfl_xor(h1 ? v[2] : v[3], 1));
    return lane_sum4_ff(ff_acc(h2 ? b : a, ff_shfl_xor(h2 ? a : b, 2)));
}

// What the next finish step needs besides the sums, prepared while the sweep runs: the largest
// objective of the GLL ring without the slot it replaces, and whether the step is a plain one
// (no stop test holds, the regular rules) that res_finish may take.
struct ResAhead {
    double fmax_other;
    bool plain;
};

__device__ __forceinline__ ResAhead res_look_ahead(const SpgDevState &h, int lane)
{
    ResAhead r;
    int li = h.fs_last + 1;
    if (li >= h.m) li = 0;
    long long key = LLONG_MIN;
    for (int q = lane; q < h.m; q += 32) {
        const long long k = fs_key(h.fs[q]);
        if (q != li && k > key) key = k;
    }
    key = warp_max_key(key);
    r.fmax_other = h.m > 1 ? fs_unkey(key) : -DBL_MAX;
    // the stop tests concern the direction about to be applied (spg_finish_sweep)
    const double dfx = h.beta * h.gd + 0.5 * h.beta * h.beta * h.dAd;
    const bool stop = (h.stop_difff && fabs(dfx) < h.eps) || (h.stop_normgp && h.dd < h.eps) ||
                      (h.stop_normgp_normb && h.dd < h.eps * h.normb) || (h.stop_Anormgp && h.dAd < h.eps) ||
                      (h.stop_Anormgp_normb && h.dAd < h.eps * h.normb);
    r.plain = !stop && !h.coeffmode && h.it + 1 < h.maxit;
    return r;
}

// The finish step of a warp.  Lane l holds the sum of value l & 3 (objective, d'd, neighbour
// differences of d, g'd).  A plain step (see ResAhead; finite sums, d'd and d'Ad positive and in
// range) takes the step lengths of spg_finish_sweep with the four values side by side in the
// lanes; everything else goes through spg_finish_sweep itself.  Returns true after a plain step:
// beta and alpha are then in sm, and the state still has to be brought forward (res_record).
template <int K>
__device__ __forceinline__ bool res_finish(ResSmem<K> &sm, FF tot, const ResAhead &ah, bool init, int cur, int lane,
                                           double &value, float &nbeta, float &nalpha)
{
    const int role = lane & 3;
    const double eps = sm.st.coeff;
    double v = ff_value(tot);
    const double w = v;
    v *= role == 0 ? 0.5 : (role == 2 ? 2.0 * eps : (role == 3 ? -1.0 : 1.0));
    value = v;
    const int hi = __double2hiint(v);
    if (role == 0) {
        v = ah.fmax_other - v;  // fx_max - fnew with fx_max = max(other, fnew)
        if (__double2hiint(v) < 0) v = 0.0;
    }
    const bool odd = ((hi >> 20) & 0x7ff) == 0x7ff || ((role == 1 || role == 2) && hi <= 0);
    const int ha = __shfl_sync(0xffffffffu, hi, 2);
    const int e = ((ha >> 20) & 0x7ff) - 1023;
    const bool fast = !__any_sync(0xffffffffu, odd) && ah.plain && !init && e > -120 && e < 120;
    if (fast) {
        const float fv = (float)(v * __hiloint2double((1023 - e) << 20, 0));
        const float q = fv / __shfl_sync(0xffffffffu, fv, 2);
        const float xi = __shfl_sync(0xffffffffu, q, 0), beta_bar = __shfl_sync(0xffffffffu, q, 3);
        const float g = (float)sm.st.gamma;
        nalpha = __shfl_sync(0xffffffffu, q, 1);
        nbeta = g * beta_bar + sqrtf(g * g * beta_bar * beta_bar + 2.f * xi);
        if (lane == 0) {
            // clamped as in spg_finish_sweep: a float is below a double sigma exactly when it is
            // below sigma rounded up to a float
            const float s1 = __double2float_ru(sm.st.sigma1), s2 = __double2float_ru(sm.st.sigma2);
            const double low = sm.st.sigma1 < sm.st.sigma2 ? sm.st.sigma1 : sm.st.sigma2;
            sm.beta = nbeta < s1 ? (float)low : (nbeta < s2 ? nbeta : (float)sm.st.sigma2);
            sm.alpha = nalpha;
        }
        return true;
    }
    double all[4];
#pragma unroll
    for (int q = 0; q < 4; q++) all[q] = __shfl_sync(0xffffffffu, w, q);
    if (lane == 0) {
        if (init) spg_finish_sweep<true>(&sm.st, cur, all);
        else spg_finish_sweep<false>(&sm.st, cur, all);
        sm.beta = (float)sm.st.beta;
        sm.alpha = (float)sm.st.alpha_cur;
        sm.status = sm.st.status;
    }
    return false;
}

// The state after a plain step, as spg_finish_sweep leaves it.
template <int K>
__device__ __forceinline__ void res_record(ResSmem<K> &sm, double value, float nbeta, float nalpha, int lane)
{
    const double fnew = __shfl_sync(0xffffffffu, value, 0), dd = __shfl_sync(0xffffffffu, value, 1);
    const double dAd = __shfl_sync(0xffffffffu, value, 2), gd = -__shfl_sync(0xffffffffu, value, 3);
    if (lane == 0) {
        SpgDevState &h = sm.st;
        h.sweeps += 1;
        h.it += 1;
        h.hessmult += 1;
        h.fx_old = h.fx;
        h.fx = fnew;
        int li = h.fs_last + 1;
        if (li >= h.m) li = 0;
        h.fs[li] = fnew;
        h.fs_last = li;
        double bh = (double)nbeta;
        if (bh < h.sigma1) bh = h.sigma1;
        h.alpha_prev = h.alpha_cur;
        h.alpha_cur = (double)nalpha;
        h.beta = bh < h.sigma2 ? bh : h.sigma2;
        h.dd = dd;
        h.dAd = dAd;
        h.gd = gd;
    }
    __syncwarp();
}

// b of one timestep, in the arithmetic of the sweeps
template <int K, int MODE>
__device__ __forceinline__ void res_b(const ResidentArgs &a, long t, const float (&theta)[K], float bscale, float (&b)[K])
{
    if (MODE == 1) {
#pragma unroll
        for (int k = 0; k < K; k++) b[k] = a.bmat[t * K + k];
    } else {
        const float v = a.data[t];
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float r = v - theta[k];
            b[k] = bscale * (r * r);
        }
    }
}

// The K values of a timestep, even K, in pieces of 8 or 16 bytes: by single values a warp's loads and
// stores are K * 4 bytes apart.  (T = 4e5, K = 8: a launch that continues a solve for one iteration, host call
// to host call, 51 -> 40 us, a solve of 30 iterations 335 -> 327; K = 4, T = 8e5 273 -> 266.  Odd K has no wider
// alignment.)
template <int K>
struct ResPiece {
    static constexpr int N = K % 4 == 0 ? 4 : 2;
    struct alignas(4 * N) type {
        float v[N];
    };
};
template <int K>
__device__ __forceinline__ void res_load(const float *p, float (&v)[K])
{
    using T = typename ResPiece<K>::type;
#pragma unroll
    for (int k = 0; k < K; k += ResPiece<K>::N) {
        const T t = *reinterpret_cast<const T *>(p + k);
#pragma unroll
        for (int j = 0; j < ResPiece<K>::N; j++) v[k + j] = t.v[j];
    }
}
template <int K>
__device__ __forceinline__ void res_store(float *p, const float *v)
{
    using T = typename ResPiece<K>::type;
#pragma unroll
    for (int k = 0; k < K; k += ResPiece<K>::N) {
        T t;
#pragma unroll
        for (int j = 0; j < ResPiece<K>::N; j++) t.v[j] = v[k + j];
        *reinterpret_cast<T *>(p + k) = t;
    }
}

// d = P(x - alpha g) - x at timestep t from x in global memory (launches that continue a solve)
template <int K, int MODE>
__device__ __forceinline__ void res_direction(const ResidentArgs &a, long t, const float (&theta)[K],
                                              const float (&c2)[K], float bscale, float alpha, float (&x)[K],
                                              float (&d)[K])
{
    float b[K];
    res_b<K, MODE>(a, t, theta, bscale, b);
    if constexpr (K % 2 == 0) {
        float xl[K], xr[K];
        res_load<K>(a.x + t * K, x);
        res_load<K>(a.x + (t > 0 ? t - 1 : t) * K, xl);
        res_load<K>(a.x + (t < a.T - 1 ? t + 1 : t) * K, xr);
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float Dl = t > 0 ? x[k] - xl[k] : 0.f;
            const float Dr = t < a.T - 1 ? xr[k] - x[k] : 0.f;
            d[k] = fmaf(-alpha, fmaf(c2[k], Dl - Dr, -b[k]), x[k]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; k++) {
            x[k] = a.x[t * K + k];
            const float Dl = t > 0 ? x[k] - a.x[(t - 1) * K + k] : 0.f;
            const float Dr = t < a.T - 1 ? a.x[(t + 1) * K + k] - x[k] : 0.f;
            d[k] = fmaf(-alpha, fmaf(c2[k], Dl - Dr, -b[k]), x[k]);
        }
    }
    project_reg<K>(d);
#pragma unroll
    for (int k = 0; k < K; k++) d[k] -= x[k];
}

// R consecutive timesteps of a thread (with PART `valid` of them, and range checks): from
// x^{c} and d to x^{c+1} and d_{c+2} in place, and their shares of the sums.  On entry xn holds the
// first one's x^{c+1} and El its difference to the timestep before; on return they belong to
// the timestep after the group (xe where the thread's range ends).  The terms of a group are added
// in plain FP32 in the order of the bulk-copy sweep (which takes the same groups of R, aligned to
// multiples of R timesteps), and the groups' sums in float-float: where that sweep has one tile
// per block, both arrive at the same sums.  (RND: where that sweep's tiles run with range checks,
// at the ends of the signal, the objective's products are rounded before they are added.)
template <int K, int MODE, bool PART, bool RND>
__device__ __forceinline__ void res_group(float *xr, float *dr, const float *br, int valid, bool end, bool atT,
                                          bool inner, float beta, float a1, float bscale, const float (&theta)[K],
                                          const float (&c2)[K], const float (&kw)[K], const float (&xe)[K],
                                          float (&xn)[K], float (&El)[K], float (&dprev)[K], KahanF &f, FF &dd, FF &dAd,
                                          FF &gd, float &pair)
{
    constexpr int R = ResShape<K>::R;
    float x1[R][K], g[R][K], d1[R][K];
    bool in[R];
#pragma unroll
    for (int r = 0; r < R; r++) in[r] = !PART || r < valid;
#pragma unroll
    for (int k = 0; k < K; k++) {
        x1[0][k] = xn[k];
#pragma unroll
        for (int r = 1; r < R; r++) x1[r][k] = in[r] ? fmaf(beta, dr[r * K + k], xr[r * K + k]) : 0.f;
        if (end) {
            if (in[R - 1]) xn[k] = atT ? x1[R - 1][k] : xe[k];
        } else {
            xn[k] = fmaf(beta, dr[R * K + k], xr[R * K + k]);
        }
    }
    float fpart = 0.f;
    {
        float v[R];
        if (MODE != 1) {
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = in[r] ? br[r] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
            float E[R + 1];
            E[0] = El[k];
#pragma unroll
            for (int r = 1; r < R; r++) E[r] = in[r] ? x1[r][k] - x1[r - 1][k] : 0.f;
            E[R] = in[R - 1] ? xn[k] - x1[R - 1][k] : 0.f;
            El[k] = E[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                float b;
                if (MODE == 1) {
                    b = in[r] ? br[r * K + k] : 0.f;
                } else {
                    const float w = v[r] - theta[k];
                    b = bscale * (w * w);
                }
                g[r][k] = fmaf(c2[k], E[r] - E[r + 1], -b);
                const float u = g[r][k] - b;
                fpart = RND ? __fadd_rn(fpart, in[r] ? __fmul_rn(u, x1[r][k]) : 0.f) : fmaf(u, x1[r][k], fpart);
                d1[r][k] = fmaf(-a1, g[r][k], x1[r][k]);
            }
        }
    }
    f.add(fpart);
#pragma unroll
    for (int r = 0; r < R; r++) {
        project_reg<K>(d1[r]);
#pragma unroll
        for (int k = 0; k < K; k++) d1[r][k] = in[r] ? d1[r][k] - x1[r][k] : 0.f;
    }
    if (inner) {  // the pair with the group before, which closes that group's d'Ad
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float df = d1[0][k] - dprev[k];
            pair = fmaf(MODE == 2 ? df * kw[k] : df, df, pair);
        }
        dAd = ff_acc(dAd, ff_make(pair));
    }
    pair = 0.f;
    float sdd = 0.f, sgd = 0.f;
#pragma unroll
    for (int k = 0; k < K; k++) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            sdd = fmaf(d1[r][k], d1[r][k], sdd);
            sgd = fmaf(g[r][k], d1[r][k], sgd);
            if (r < R - 1) {
                const float df = in[r + 1] ? d1[r + 1][k] - d1[r][k] : 0.f;
                pair = fmaf(MODE == 2 ? df * kw[k] : df, df, pair);
            }
            if (in[r]) {
                xr[r * K + k] = x1[r][k];
                dr[r * K + k] = d1[r][k];
            }
        }
        dprev[k] = d1[R - 1][k];
    }
    dd = ff_acc(dd, ff_make(sdd));
    gd = ff_acc(gd, ff_make(sgd));
}

__device__ __forceinline__ void res_mgr_sync() { asm volatile("bar.sync 1, %0;" ::"n"(RES_MGR) : "memory"); }

template <int K, int MODE>
__global__ void __launch_bounds__(ResShape<K>::NT + RES_MGR, 1) spg_resident_kernel(const __grid_constant__ ResidentArgs a)
{
    extern __shared__ __align__(16) float dyn[];
    __shared__ ResSmem<K> sm;
    const int nt = blockDim.x, walkers = nt - RES_MGR;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = walkers >> 5;
    constexpr int R = ResShape<K>::R;
    const int nb = gridDim.x, M = a.M;
    const int S = (M * K) | 1, Sd = MODE == 1 ? S : (M | 1);  // odd row strides
    const int rows = (a.C + M - 1) / M;
    float *xs = dyn, *ds = xs + (size_t)rows * S, *bs = ds + (size_t)rows * S;
    const long t0 = (long)blockIdx.x * a.C;
    const int Cb = (int)min((long)a.C, a.T - t0);

    // the state: every block works on its own copy (no block writes the global one before all
    // have read it: at least one exchange lies in between)
    {
        const unsigned int *src = reinterpret_cast<const unsigned int *>(a.st);
        unsigned int *dst = reinterpret_cast<unsigned int *>(&sm.st);
        for (int q = tid; q < (int)(sizeof(SpgDevState) / 4); q += nt) dst[q] = __ldcg(src + q);
    }
    __syncthreads();
    if (sm.st.status != PASC_SPG_RUNNING) return;  // uniform across the grid
    const float coeff = (float)sm.st.coeff, bscale = (float)sm.st.bscale;
    float theta[K], c2[K], kw[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        theta[k] = MODE == 1 ? 0.f : a.theta[k];
        kw[k] = MODE == 2 ? a.kw[k] : 1.f;
        c2[k] = MODE == 2 ? (2.f * coeff) * kw[k] : 2.f * coeff;
    }

    // x, d and the data (or b) of the block's timesteps and its edges
    const float alpha0 = (float)sm.st.alpha_prev;
    for (int tl = tid; tl < Cb; tl += nt) {
        const long t = t0 + tl;
        const int i = tl / M, j = tl - i * M;
        float x[K], d[K];
        if (a.init) {
            if constexpr (K % 2 == 0) res_load<K>(a.x + t * K, x);
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (K % 2) x[k] = a.x[t * K + k];
                d[k] = 0.f;
            }
            project_reg<K>(x);
        } else {
            res_direction<K, MODE>(a, t, theta, c2, bscale, alpha0, x, d);
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
            xs[i * S + j * K + k] = x[k];
            ds[i * S + j * K + k] = d[k];
            if (MODE == 1) bs[i * S + j * K + k] = a.bmat[t * K + k];
        }
        if (MODE != 1) bs[i * Sd + j] = a.data[t];
    }
    if (tid < 3) {
        const long t = tid == 0 ? t0 - 1 : t0 + Cb + (tid - 1);
        float x[K], d[K];
#pragma unroll
        for (int k = 0; k < K; k++) x[k] = d[k] = 0.f;
        if (t >= 0 && t < a.T) {
            if (a.init) {
#pragma unroll
                for (int k = 0; k < K; k++) x[k] = a.x[t * K + k];
                project_reg<K>(x);
            } else {
                res_direction<K, MODE>(a, t, theta, c2, bscale, alpha0, x, d);
            }
            if (tid == 1) {
                float b[K];
                res_b<K, MODE>(a, t, theta, bscale, b);
#pragma unroll
                for (int k = 0; k < K; k++) sm.hb[k] = b[k];
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (tid == 0) {
                sm.hlx[k] = x[k];
                sm.hld[k] = d[k];
            } else {
                sm.hrx[tid - 1][k] = x[k];
                sm.hrd[tid - 1][k] = d[k];
            }
        }
    }
    if (tid == 0) {
        sm.beta = (float)sm.st.beta;
        sm.alpha = (float)sm.st.alpha_cur;
        sm.status = PASC_SPG_RUNNING;
    }
    __syncthreads();

    if (tid < walkers) {
        const int m = min(M, Cb - tid * M);  // timesteps of this thread (<= 0: none)
        const bool last = m > 0 && tid * M + m == Cb;
        const bool at0 = t0 + (long)tid * M == 0, atT = last && t0 + Cb == a.T;
        float *xr = xs + tid * S, *dr = ds + tid * S, *br = bs + tid * Sd;
        const int groups = m > 0 ? (m + R - 1) / R : 0;
        // the groups without range checks: [q0, q1)
        const long tf = t0 + (long)tid * M;
        const int q0 = (int)max(0L, min((long)groups, (a.edge_lo - tf + R - 1) / R));
        const int q1 = (int)max(0L, min((long)(m / R), (a.edge_hi - tf + R - 1) / R));
        for (int s = 0; s < a.sweeps; s++) {
            const float beta = sm.beta, a1 = sm.alpha;
            float El[K], xn[K], xe[K], dprev[K];
            KahanF f;
            FF dd{0.f, 0.f}, dAd{0.f, 0.f}, gd{0.f, 0.f};
            float pair = 0.f;  // d'Ad terms of the current group, until its last pair is known
            if (m > 0) {
                const float *lx = tid ? xr - S + (M - 1) * K : sm.hlx, *ld = tid ? dr - S + (M - 1) * K : sm.hld;
                const float *rx = last ? sm.hrx[0] : xr + S, *rd = last ? sm.hrd[0] : dr + S;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    xn[k] = fmaf(beta, dr[k], xr[k]);
                    const float l = fmaf(beta, ld[k], lx[k]);
                    xe[k] = fmaf(beta, rd[k], rx[k]);
                    El[k] = at0 ? 0.f : xn[k] - l;
                }
            }
            __syncthreads();  // the neighbours' rows were read: rows may change from here on
            if (m > 0) {
                if (tid == 0) {
#pragma unroll
                    for (int k = 0; k < K; k++) sm.hlx[k] = fmaf(beta, sm.hld[k], sm.hlx[k]);
                }
#pragma unroll 1
                for (int q = 0; q < groups; q++) {
                    const int rest = min(R, m - q * R);
                    const bool end = q == groups - 1;
                    float *xg = xr + q * R * K, *dg = dr + q * R * K;
                    const float *bg = br + q * R * (MODE == 1 ? K : 1);
                    if (q >= q0 && q < q1)
                        res_group<K, MODE, false, false>(xg, dg, bg, R, end, atT, q > 0, beta, a1, bscale, theta, c2, kw,
                                                         xe, xn, El, dprev, f, dd, dAd, gd, pair);
                    else if (rest == R)
                        res_group<K, MODE, false, true>(xg, dg, bg, R, end, atT, q > 0, beta, a1, bscale, theta, c2, kw,
                                                        xe, xn, El, dprev, f, dd, dAd, gd, pair);
                    else
                        res_group<K, MODE, true, true>(xg, dg, bg, rest, end, atT, q > 0, beta, a1, bscale, theta, c2, kw,
                                                       xe, xn, El, dprev, f, dd, dAd, gd, pair);
                }
                if (last && !atT) {
                    // the right neighbour block's first timestep: its d, for the pair across the
                    // blocks
                    float d1[K];
                    const bool edge = t0 + Cb == a.T - 1;  // it is the signal's last one
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        const float x2 = fmaf(beta, sm.hrd[1][k], sm.hrx[1][k]);
                        const float Er = edge ? 0.f : x2 - xn[k];
                        d1[k] = fmaf(-a1, fmaf(c2[k], El[k] - Er, -sm.hb[k]), xn[k]);
                        sm.hrx[0][k] = xn[k];
                        sm.hrx[1][k] = x2;
                    }
                    project_reg<K>(d1);
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        const float df = (d1[k] - xn[k]) - dprev[k];
                        pair = fmaf(MODE == 2 ? df * kw[k] : df, df, pair);
                    }
                }
            }
            __syncthreads();
            if (m > 0) {
                if (!last) {
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        const float df = dr[S + k] - dprev[k];
                        pair = fmaf(MODE == 2 ? df * kw[k] : df, df, pair);
                    }
                }
                dAd = ff_acc(dAd, ff_make(pair));
            }
            const FF v[4] = {FF{f.s, f.c}, dd, dAd, gd};
            const FF r = warp_sum4_ff(v, lane);
            if (lane < 4) sm.red[warp][lane] = make_float2(r.hi, r.lo);
            __syncthreads();
            __syncthreads();  // the managers have set beta, alpha and the status
            if (sm.status != PASC_SPG_RUNNING) break;  // the same in every block
        }
    } else {
        const int mt = tid - walkers, mw = mt >> 5;
        const int cur = sm.st.cur ^ 1;  // the finish step flips it: x stays in its buffer
        ResAhead ah{0.0, false};
        bool plain = false;             // the last finish was a plain step, not yet recorded
        double value = 0.0;
        float nbeta = 0.f, nalpha = 0.f;
        for (int s = 0; s < a.sweeps; s++) {
            const unsigned int tag = a.tag + (unsigned int)s;
            unsigned long long *slots = a.slots + (size_t)(tag & 1u) * nb * RES_WORDS;
            __syncthreads();
            if (mw == 0) {
                if (plain) res_record<K>(sm, value, nbeta, nalpha, lane);
                ah = res_look_ahead(sm.st, lane);
            }
            __syncthreads();
            // the new d of the block's first two and last timesteps
            if (nb > 1 && mw == 1 && lane < 3 * K) {
                const int which = lane / K, k = lane - which * K;
                const int tl = which == 2 ? Cb - 1 : min(which, Cb - 1), i = tl / M;
                word_store(slots + (size_t)blockIdx.x * RES_WORDS + 8 + lane, word_of(ds[i * S + (tl - i * M) * K + k], tag));
            }
            __syncthreads();
            FF tot{0.f, 0.f};
            if (mw == 0) {
                for (int q = lane >> 2; q < nw; q += 8) {
                    const float2 p = sm.red[q][lane & 3];
                    tot = ff_acc(tot, FF{p.x, p.y});
                }
                tot = lane_sum4_ff(tot);
                if (nb > 1 && lane < 4)
                    word_store2(slots + (size_t)blockIdx.x * RES_WORDS + 2 * lane, word_of(tot.hi, tag),
                               word_of(tot.lo, tag));
            }
            if (nb > 1) {
                bool ok = true;
                // the neighbours' new d at this block's edges (warp 1)
                if (mw == 1 && lane < 3 * K) {
                    const int which = lane / K, k = lane - which * K;
                    const long t = which == 0 ? t0 - 1 : t0 + Cb + (which - 1);
                    if (t >= 0 && t < a.T) {
                        // left: the last row of the block before; right: rows 0 and 1 of the next one
                        const size_t ob = which == 0 ? blockIdx.x - 1 : blockIdx.x + 1;
                        const int ow = 8 + (which == 0 ? 2 * K : (which - 1) * K) + k;
                        unsigned long long w = 0;
                        for (unsigned int it = 0;; it++) {
                            w = word_load(slots + ob * RES_WORDS + ow);
                            if (word_valid(w, tag)) break;
                            if (it >= WORD_WAIT_LIMIT) {
                                ok = false;
                                break;
                            }
                        }
                        if (which == 0) sm.hld[k] = word_float(w);
                        else sm.hrd[which - 1][k] = word_float(w);
                    }
                }
                // all blocks' sums: 16 bytes (a float-float pair) per load, RES_POLL loads in flight
                constexpr int RES_POLL = 5;
                FF u{0.f, 0.f};
                for (int w0 = mt; w0 < 4 * nb; w0 += RES_POLL * RES_MGR) {
                    unsigned long long hi[RES_POLL], lo[RES_POLL];
                    for (unsigned int it = 0;; it++) {
                        bool all = true;
#pragma unroll
                        for (int q = 0; q < RES_POLL; q++) {
                            const int w = w0 + q * RES_MGR;
                            if (w < 4 * nb) {
                                word_load2(slots + (size_t)(w >> 2) * RES_WORDS + 2 * (w & 3), hi[q], lo[q]);
                            } else {
                                hi[q] = lo[q] = word_of(0.f, tag);
                            }
                        }
#pragma unroll
                        for (int q = 0; q < RES_POLL; q++)
                            all &= word_valid(hi[q], tag) && word_valid(lo[q], tag);
                        if (all) break;
                        if (it >= WORD_WAIT_LIMIT) {
                            ok = false;
                            break;
                        }
                    }
#pragma unroll
                    for (int q = 0; q < RES_POLL; q++) u = ff_acc(u, FF{word_float(hi[q]), word_float(lo[q])});
                }
                u = lane_sum4_ff(u);
                if (lane < 4) sm.red2[mw][lane] = make_float2(u.hi, u.lo);
                if (!ok) atomicExch(&a.st->error, 1);
                if (!__all_sync(0xffffffffu, ok) && lane == 0) sm.status = -1;
                res_mgr_sync();
                if (mw == 0) {
                    const float2 p = lane < 16 ? sm.red2[lane >> 2][lane & 3] : make_float2(0.f, 0.f);
                    tot = lane_sum4_ff(FF{p.x, p.y});
                }
            }
            if (mw == 0 && sm.status == PASC_SPG_RUNNING)
                plain = res_finish<K>(sm, tot, ah, a.init && s == 0, cur, lane, value, nbeta, nalpha);
            __syncthreads();
            if (sm.status != PASC_SPG_RUNNING) break;
        }
        if (mw == 0 && plain && sm.status == PASC_SPG_RUNNING) res_record<K>(sm, value, nbeta, nalpha, lane);
    }
    __syncthreads();
    // a wait gave up: the error word is set.  (gamma is undefined then: blocks that had all they waited for
    // in the last sweep write their rows.)
    if (sm.status < 0) return;
    for (int tl = tid; tl < Cb; tl += nt) {
        const int i = tl / M, j = tl - i * M;
        if constexpr (K % 2 == 0) {
            res_store<K>(a.x + (t0 + tl) * K, xs + i * S + j * K);
        } else {
#pragma unroll
            for (int k = 0; k < K; k++) a.x[(t0 + tl) * K + k] = xs[i * S + j * K + k];
        }
    }
    if (blockIdx.x == 0) {
        const unsigned int *src = reinterpret_cast<const unsigned int *>(&sm.st);
        unsigned int *dst = reinterpret_cast<unsigned int *>(a.st);
        for (int q = tid; q < (int)(sizeof(SpgDevState) / 4); q += nt)
            if (q != (int)(offsetof(SpgDevState, error) / 4)) dst[q] = src[q];
    }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
template <int K, int MODE>
static const void *res_kernel()
{
    return (const void *)spg_resident_kernel<K, MODE>;
}

static const void *res_kernel_of(int K, int mode)
{
    switch (K) {
#define PASC_CASE(KK) \
    case KK: return mode == 1 ? res_kernel<KK, 1>() : (mode == 2 ? res_kernel<KK, 2>() : res_kernel<KK, 0>());
        PASC_CASE(1) PASC_CASE(2) PASC_CASE(3) PASC_CASE(4)
        PASC_CASE(5) PASC_CASE(6) PASC_CASE(7) PASC_CASE(8)
#undef PASC_CASE
        default: return nullptr;
    }
}

static int res_threads(int K) { return K <= 3 ? ResShape<3>::NT : ResShape<8>::NT; }

static size_t res_dyn_bytes(int K, int mode, int C, int M)
{
    const size_t rows = (C + M - 1) / M, S = (M * K) | 1, Sd = mode == 1 ? S : (M | 1);
    return sizeof(float) * rows * (2 * S + Sd);
}

size_t resident_words(int sms) { return (size_t)2 * sms * RES_WORDS; }

// Blocks, and timesteps per block and thread.  A thread walks at least four timesteps (fewer
// warps to reduce; T = 1e4, K = 2 on 20 blocks: 3.95 us per iteration with one timestep per
// thread, 3.76 with four).  One block needs no exchange: it takes signals up to 4096 (K <= 2),
// 2048 (K <= 5) or 1024 timesteps (T = 2000: K = 2 2.6 us against 4.0 on four blocks, K = 5 3.5
// against 4.3, K = 8 4.8 against 4.6; T = 4000: K = 2 2.8 against 3.9, K = 5 4.8 against 4.0).
// Beyond, 512 timesteps per block up to one block per SM (T = 50 000, K = 4: 98 blocks 4.03 us,
// 49 blocks 4.07, 152 blocks 4.07), then as many as it takes.
bool resident_plan(int K, int mode, long T, int sms, int smem_optin, ResidentPlan *plan)
{
    if (K < 1 || K > KMAX_FUSED || sms < 1 || T < 1) return false;
    const size_t room = (size_t)smem_optin - sizeof(ResSmem<KMAX_FUSED>) - 1024;
    const long nt = res_threads(K), one = K <= 2 ? 4096 : (K <= 5 ? 2048 : 1024);
    long nb = T <= one ? 1 : (T + 511) / 512;
    if (nb > sms) nb = sms;
    // whole groups of timesteps per block and per thread
    const long C = ((T + nb - 1) / nb + 3) / 4 * 4;
    const long M = std::max(4L, ((C + nt - 1) / nt + 3) / 4 * 4);
    if (M > (1 << 16) || res_dyn_bytes(K, mode, (int)C, (int)M) > room) return false;
    nb = (T + C - 1) / C;
    plan->blocks = (int)nb;
    plan->C = (int)C;
    plan->M = (int)M;
    plan->threads = (int)(((C + M - 1) / M + 31) / 32 * 32) + RES_MGR;
    plan->smem = res_dyn_bytes(K, mode, (int)C, (int)M);
    return true;
}

cudaError_t resident_prepare(int K, int mode, const ResidentPlan &plan)
{
    const void *fn = res_kernel_of(K, mode);
    if (!fn) return cudaErrorInvalidValue;
    // the limit is raised to the same value (all a block can have) for every handle: the
    // attribute belongs to the process, and another handle may launch at any time
    cudaFuncAttributes fa;
    int dev = 0, optin = 0;
    cudaError_t e = cudaFuncGetAttributes(&fa, fn);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    if (e != cudaSuccess) return e;
    int nb = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, plan.threads, plan.smem);
    if (e != cudaSuccess) return e;
    return nb >= 1 ? cudaSuccess : cudaErrorCooperativeLaunchTooLarge;
}

cudaError_t launch_resident(int K, int mode, const ResidentPlan &plan, const ResidentArgs &a, cudaStream_t s)
{
    const void *fn = res_kernel_of(K, mode);
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {const_cast<ResidentArgs *>(&a)};
    return cudaLaunchCooperativeKernel(fn, dim3(plan.blocks), dim3(plan.threads), args, plan.smem, s);
}

}  // namespace pasc
