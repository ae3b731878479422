// kernels_fp64.cu -- the FP64 path's SPG iterations in one cooperative launch (K <= 8, 1-D
// signals; larger K and graphs keep one kernel per operation, kernels_plain.cu).
//
// One kernel per operation of the reference moves about 190 bytes per entry and iteration, stops
// twice per iteration for the host's scalars (74 us per iteration at T = 1e4), and spends the
// part's slow FP64 pipe (about 2 lanes per clock and SM) on comparisons and divisions.  Here
// an iteration is one pass, timed like the mixed sweeps: it applies the step of the direction at
// hand, x += beta d, g += beta Ad, f = 1/2 (g - b)'x, and forms the next one, d = P(x - alpha g) - x,
// Ad, d'd, d'Ad, g'd, with the gradient kept and updated recursively as in the reference
// (src/petscvector/solver/spgqpsolver.cpp:140-216).  x, g, d, Ad are updated in place; block b owns C
// timesteps and keeps x, g, d, Ad, b of the timestep before and after them, which it advances
// itself (only their new Ad comes from the neighbours).  The four sums and these edges travel as
// tagged words (grid_words.cuh), every block adds the sums in the same order and applies the step
// rules in FP64 to its own copy of the state.
//
// Bound: FP64 issue from about 1e5 timesteps on.  Per entry 15 FP64 instructions and a share
// of the projection (12 per timestep at K = 3), every value the reference's: the row of A_hat
// halved, (2 x_t - x_l) - x_r (the factor 2 goes into the coefficient, both exact), sort and sign
// tests on integer keys, and the projection's division by K - i by its reciprocal with one
// correction step (Markstein 1990: exactly rounded).  Below, the chain of one iteration.  Measured,
// us per iteration, one kernel per operation / here: T = 1e4, K = 2 74 / 8.3; T = 1e6, K = 3 340 /
// 182 (about 115 of FP64 issue; 152 with the sums taken where the terms arise, in another order).
#include <stddef.h>
#include <algorithm>

#include "common.cuh"
#include "project64.cuh"
#include "grid_words.cuh"
#include "sweep_common.cuh"
#include "internal.h"

namespace pasc {

// The sums are taken in the order of the one-kernel-per-operation path for every size: 256 * 4 * SMs
// threads each add the products of the entries a stride apart, trees over 256 threads, then over
// the trees.  The iterates are that path's bit for bit: where the reference's stopping rules stop,
// and where a solve at the limit of FP64 stalls, depends on the last bits of the sums (at T = 2e5,
// epssqr 100 another order stalled at a duality gap of 5e-12 f instead of 1e-12).  Two forms:
//   ORDERED  at most 256 * 4 * SMs entries, one entry per thread of that order: one tile of 64 to 256
//            timesteps per block (a multiple of 256 entries), the terms in shared memory;
//   STREAM   block b owns C timesteps, walked in tiles of W = 254 (one more thread each for the timestep
//            after the tile and the one before the block); after a grid barrier the blocks add the
//            terms from x, g, d, Ad, b in that order.
constexpr int F64_NT = 256;
constexpr int F64_W = F64_NT - 2;
constexpr int F64_NT_ORDERED = 288;            // 256 timesteps and a warp for the two edges

// ---------------------------------------------------------------------------------------
// sums and the finish step
// ---------------------------------------------------------------------------------------
// The warp sums of block_sum (common.cuh), lanes 16 apart first; lane l returns the sum of value
// ordered_value(l).
__device__ __forceinline__ int ordered_value(int lane) { return ((lane >> 4) & 1) + ((lane >> 2) & 2); }
__device__ __forceinline__ double warp_sum4_ordered(const double (&v)[4], int lane)
{
    const bool h1 = lane & 16, h2 = lane & 8;
    const double a = (h1 ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, h1 ? v[0] : v[1], 16);
    const double b = (h1 ? v[3] : v[2]) + __shfl_xor_sync(0xffffffffu, h1 ? v[2] : v[3], 16);
    double r = (h2 ? b : a) + __shfl_xor_sync(0xffffffffu, h2 ? a : b, 8);
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) r += __shfl_xor_sync(0xffffffffu, r, m);
    return r;
}
// over eight neighbouring lanes, lanes 4 apart first
__device__ __forceinline__ double sum8_ordered(double r)
{
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) r += __shfl_xor_sync(0xffffffffu, r, m);
    return r;
}

struct F64Step {
    double beta, beta_g, alpha;  // x += beta d, g += beta_g Ad, d = P(x - alpha g) - x
    int status;
};

// One warp: the reference's rules (spgqpsolver.cpp:176-274; SPGQPSolverC,
// spgqpsolver_coeff.h:611-835) on the sums (lane l: value l & 3 of x'(g - b), d'd, d'Ad, g'd).  first:
// the sums belong to the start point.  The three quotients by d'Ad are taken side by side.
__device__ __forceinline__ void f64_finish(Fp64DevState &h, F64Step &out, double sum, bool first, int lane)
{
    const double fnew = __dmul_rn(0.5, __shfl_sync(0xffffffffu, sum, 0));
    const double dd = __shfl_sync(0xffffffffu, sum, 1), dAd = __shfl_sync(0xffffffffu, sum, 2);
    const double gd = __shfl_sync(0xffffffffu, sum, 3);
    int li = h.fs_last + 1;
    if (li >= h.m) li = 0;
    long long key = fs_key(fnew);
    if (!first) {
        for (int q = lane; q < h.m; q += 32) {
            const long long k = fs_key(h.fs[q]);
            if (q != li && k > key) key = k;
        }
        key = warp_max_key(key);
    }
    const int role = lane & 3;
    const double num = role == 0 ? __dadd_rn(fs_unkey(key), -fnew) : (role == 1 ? dd : -gd);
    const double quot = __ddiv_rn(num, dAd);
    const double xi = __shfl_sync(0xffffffffu, quot, 0), beta_bar = __shfl_sync(0xffffffffu, quot, 3);
    const double bb = __shfl_sync(0xffffffffu, quot, 1);  // the BB step
    const bool cm = h.coeffmode != 0;
    const double eps = h.coeff, einv = eps == 0.0 ? 1.0 : 1.0 / eps;
    const double gb = __dmul_rn(h.gamma, beta_bar);
    const double rad = __dadd_rn(__dmul_rn(__dmul_rn(__dmul_rn(h.gamma, h.gamma), beta_bar), beta_bar),
                                 cm ? __dmul_rn(__dmul_rn(2.0, eps), xi) : __dmul_rn(2.0, xi));
    double beta_hat = __dadd_rn(gb, __dsqrt_rn(rad));
    __syncwarp();
    if (lane == 0) {
        int status = PASC_SPG_RUNNING;
        h.sweeps += 1;
        if (first) {
            h.fx = fnew;
            h.fx_old = DBL_MAX;
            for (int q = 0; q < h.m; q++) h.fs[q] = fnew;
            h.fs_last = 0;
            h.it = 0;
            h.hessmult = 1;
            if (h.maxit <= 0) status = PASC_SPG_MAXIT;
            else if (!isfinite(fnew)) status = PASC_SPG_NONFINITE;
        } else {
            const double ddo = h.dd, dAdo = h.dAd;
            h.it += 1;
            h.fx_old = h.fx;
            h.fx = fnew;
            h.fs_last = li;
            h.fs[li] = fnew;
            h.dd_done = ddo;
            h.dAd_done = dAdo;
            if (!isfinite(fnew)) status = PASC_SPG_NONFINITE;
            else if ((h.stop_difff && fabs(fnew - h.fx_old) < h.eps) || (h.stop_normgp && ddo < h.eps) ||
                     (h.stop_normgp_normb && ddo < h.eps * h.normb) || (h.stop_Anormgp && dAdo < h.eps) ||
                     (h.stop_Anormgp_normb && dAdo < h.eps * h.normb))
                status = PASC_SPG_CONVERGED;
            else if (h.it >= h.maxit) status = PASC_SPG_MAXIT;
        }
        if (status == PASC_SPG_RUNNING) {
            h.hessmult += 1;
            if (!(isfinite(dd) && isfinite(dAd) && isfinite(gd))) status = PASC_SPG_NONFINITE;
            else if (!(dd > 0.0)) status = PASC_SPG_DAD_ZERO;
            else if (dAd > 0.0) {
                double beta;
                if (cm) {
                    if (__dmul_rn(einv, beta_hat) < h.sigma1) beta_hat = h.sigma1;
                    beta = __dmul_rn(einv, beta_hat);
                } else {
                    if (beta_hat < h.sigma1) beta_hat = h.sigma1;
                    beta = beta_hat;
                }
                h.beta = beta < h.sigma2 ? beta : h.sigma2;
                h.alpha = bb;
            } else if (gd < 0.0) {
                h.beta = h.sigma2;  // linear along d: the reference's division by zero falls through to sigma2
            } else {
                status = PASC_SPG_DAD_ZERO;
            }
            h.dd = dd;
            h.dAd = dAd;
            h.gd = gd;
            h.ahead = status != PASC_SPG_RUNNING;
        }
        h.status = status;
        out.beta = h.beta;
        out.beta_g = cm ? __dmul_rn(eps, h.beta) : h.beta;
        out.alpha = cm ? __dmul_rn(einv, h.alpha) : h.alpha;
        out.status = status;
    }
}

// ---------------------------------------------------------------------------------------
// the iterations
// ---------------------------------------------------------------------------------------
template <int K>
struct F64Smem {
    Fp64DevState st;
    F64Step step;
    double d[(F64_NT + 2) * K];  // the tile's new d; row 0: the timestep before it
    double hx[2][K], hg[2][K], hd[2][K], hAd[2][K], hb[2][K];  // the block's edges: timestep before, after
    double red[KMAX_FUSED][F64_NT / 32][4];
};

// x, g of one timestep brought forward and its next direction.  Every product is rounded before it is
// added, as in the reference's VecAXPY: with fused products the rows of x drift off sum 1 with
// another bias, and at T = 1e7, epssqr 1000 the solve stalled at a duality gap of 4e-10 f, where
// the rounded ones reach 2e-11.
template <int K>
__device__ __forceinline__ void f64_advance(double (&x)[K], double (&g)[K], const double (&d)[K], const double (&Ad)[K],
                                            const F64Step &s, double (&dn)[K])
{
#pragma unroll
    for (int k = 0; k < K; k++) {
        x[k] = __dadd_rn(x[k], __dmul_rn(s.beta, d[k]));
        g[k] = __dadd_rn(g[k], __dmul_rn(s.beta_g, Ad[k]));
        dn[k] = __dadd_rn(x[k], __dmul_rn(-s.alpha, g[k]));
    }
    project_f64<K>(dn);
#pragma unroll
    for (int k = 0; k < K; k++) dn[k] = __dadd_rn(dn[k], -x[k]);
}

template <int K, bool ORDERED>
__global__ void __launch_bounds__(ORDERED ? F64_NT_ORDERED : F64_NT, K <= 5 ? 2 : 1)
    spg_fp64_kernel(const __grid_constant__ Fp64Args a)
{
    constexpr int NT = ORDERED ? F64_NT_ORDERED : F64_NT, W = ORDERED ? 256 : F64_W;
    // the terms of the four sums of 256 timesteps (ORDERED), then the sums of all trees
    extern __shared__ __align__(16) double terms[];
    __shared__ F64Smem<K> sm;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = gridDim.x;
    const long t0 = (long)blockIdx.x * a.C, T = a.T;
    const int Cb = (int)min((long)a.C, T - t0);
    const int trees = ORDERED ? (int)((T * K + 255) / 256) : a.trees;
    const int own_trees = ORDERED ? a.C * K / 256 : (trees + nb - 1) / nb;
    // a set of words: four sums per tree, the blocks' end timesteps, the barrier
    const size_t set_words = (size_t)trees * 8 + (size_t)nb * (4 * K + 2);
    {
        const unsigned int *src = reinterpret_cast<const unsigned int *>(a.st);
        unsigned int *dst = reinterpret_cast<unsigned int *>(&sm.st);
        for (int q = tid; q < (int)(sizeof(Fp64DevState) / 4); q += NT) dst[q] = __ldcg(src + q);
    }
    if (tid < 2 * K) {
        const int e = tid / K, k = tid - e * K;
        const long t = e ? t0 + Cb : t0 - 1;
        const bool in = t >= 0 && t < T;
        const long i = in ? t * K + k : 0;
        sm.hx[e][k] = in ? a.x[i] : 0.0;
        sm.hg[e][k] = in ? a.g[i] : 0.0;
        sm.hb[e][k] = in ? a.b[i] : 0.0;
        sm.hd[e][k] = in && !a.first ? a.d[i] : 0.0;
        sm.hAd[e][k] = in && !a.first ? a.Ad[i] : 0.0;
    }
    __syncthreads();
    if (sm.st.status != PASC_SPG_RUNNING) return;  // uniform across the grid
    if (tid == 0) {
        const Fp64DevState &h = sm.st;
        const bool cm = h.coeffmode != 0;
        const double einv = h.coeff == 0.0 ? 1.0 : 1.0 / h.coeff;
        sm.step.beta = h.beta;
        sm.step.beta_g = cm ? __dmul_rn(h.coeff, h.beta) : h.beta;
        sm.step.alpha = cm ? __dmul_rn(einv, h.alpha) : h.alpha;
        sm.step.status = PASC_SPG_RUNNING;
    }
    double c2[K];  // A = coefficient * A_hat, twice it for the halved rows
#pragma unroll
    for (int k = 0; k < K; k++) c2[k] = 2.0 * (a.kc ? a.kc[k] : (sm.st.coeffmode ? 1.0 : sm.st.coeff));
    bool ok = true;

    // sweep -1 only exchanges: no block may change x, g, d, Ad before its neighbours have read
    // their edges
    for (int s = nb > 1 ? -1 : 0; s < a.sweeps; s++) {
        const unsigned int tag = a.tag + (unsigned int)(s + 1);
        unsigned long long *slots = a.slots + (size_t)(tag & 1u) * set_words;
        // words of the blocks' end timesteps: Ad of the first, then of the last one
        unsigned long long *edges = slots + (size_t)trees * 8, *barrier = edges + (size_t)nb * 4 * K;
        __syncthreads();
        if (s >= 0) {
            const F64Step st = sm.step;
            const bool zero = a.first && s == 0;  // no direction yet
            for (int base = 0; base < Cb; base += W) {
                const int n = min(W, Cb - base);
                double x[K], g[K], d[K], Ad[K], b[K], dn[K];
                // thread i < n: timestep base + i; thread `after`: the one after the tile; the thread
                // behind it (first tile): the one before the block
                const int after = ORDERED ? W : n, before = after + 1;
                const int edge = tid == before ? 0 : 1;
                const bool mine = tid < n;
                const int row = tid == before ? 0 : (tid == after ? n + 1 : tid + 1);
                const long t = t0 + base + row - 1;
                const bool act = t >= 0 && t < T && (mine || tid == after || (tid == before && base == 0));
                const bool priv = act && !mine && (edge == 0 || base + n == Cb);  // the block's own copies
                if (act) {
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        const long i = t * K + k;
                        x[k] = priv ? sm.hx[edge][k] : a.x[i];
                        g[k] = priv ? sm.hg[edge][k] : a.g[i];
                        b[k] = priv ? sm.hb[edge][k] : a.b[i];
                        d[k] = zero ? 0.0 : (priv ? sm.hd[edge][k] : a.d[i]);
                        Ad[k] = zero ? 0.0 : (priv ? sm.hAd[edge][k] : a.Ad[i]);
                    }
                    f64_advance<K>(x, g, d, Ad, st, dn);
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        if (priv) {
                            sm.hx[edge][k] = x[k];
                            sm.hg[edge][k] = g[k];
                            sm.hd[edge][k] = dn[k];
                        }
                        sm.d[row * K + k] = dn[k];
                        if (ORDERED && mine) terms[tid * K + k] = __dmul_rn(x[k], __dadd_rn(g[k], -b[k]));
                    }
                }
                __syncthreads();
                double dlast[K];
                if (mine) {
                    const double *dl = sm.d + tid * K, *dr = sm.d + (tid + 2) * K;
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        double rw;
                        if (t > 0) rw = t < T - 1 ? __dadd_rn(fma(2.0, dn[k], -dl[k]), -dr[k]) : __dadd_rn(dn[k], -dl[k]);
                        else rw = t < T - 1 ? __dadd_rn(dn[k], -dr[k]) : 0.0;
                        Ad[k] = __dmul_rn(c2[k], rw);
                        if (ORDERED) {
                            double *q = terms + tid * K + k;
                            q[256 * K] = __dmul_rn(dn[k], dn[k]);
                            q[512 * K] = __dmul_rn(dn[k], Ad[k]);
                            q[768 * K] = __dmul_rn(dn[k], g[k]);
                        }
                        const long i = t * K + k;
                        a.x[i] = x[k];
                        a.g[i] = g[k];
                        a.d[i] = dn[k];
                        a.Ad[i] = Ad[k];
                        dlast[k] = dn[k];
                    }
                    if (nb > 1) {
                        // Ad at the block's ends, for the neighbours' copies of these timesteps
                        unsigned long long *e = edges + (size_t)blockIdx.x * 4 * K;
                        if (base + tid == 0) {
#pragma unroll
                            for (int k = 0; k < K; k++) word_store_double(e + 2 * k, Ad[k], tag);
                        }
                        if (base + tid == Cb - 1) {
#pragma unroll
                            for (int k = 0; k < K; k++) word_store_double(e + 2 * K + 2 * k, Ad[k], tag);
                        }
                    }
                }
                __syncthreads();
                if (!ORDERED && tid == n - 1) {  // the timestep before the next tile
#pragma unroll
                    for (int k = 0; k < K; k++) sm.d[k] = dlast[k];
                }
            }
        }
        if (!ORDERED && s >= 0 && nb > 1) {
            // every block's x, g, d, Ad are written (and visible) before the terms are read
            __threadfence();
            __syncthreads();
            if (tid == 0) word_store(barrier + 2 * blockIdx.x, word_of(1u, tag));
            for (int w = tid; w < nb; w += NT) {
                bool have = false;
                for (unsigned int it = 0; it < WORD_WAIT_LIMIT && !have; it++) have = word_valid(word_load(barrier + 2 * w), tag);
                ok &= have;
            }
            __threadfence();
            __syncthreads();
        }
        // the trees over 256 threads, published one by one
        const long n = T * K;
        if (tid < 256) {
#pragma unroll 1
            for (int c = 0; c < own_trees; c++) {
                double v[4] = {0.0, 0.0, 0.0, 0.0};
                if (ORDERED) {
                    const int e = c * 256 + tid;
                    if (s >= 0 && e < Cb * K) {
#pragma unroll
                        for (int q = 0; q < 4; q++) v[q] = terms[q * 256 * K + e];
                    }
                } else if (s >= 0 && blockIdx.x * own_trees + c < trees) {
#pragma unroll 4
                    for (long e = (long)(blockIdx.x * own_trees + c) * 256 + tid; e < n; e += (long)trees * 256) {
                        // (through L2: other blocks wrote them)
                        const double x = __ldcg(a.x + e), g = __ldcg(a.g + e), d = __ldcg(a.d + e), Ad = __ldcg(a.Ad + e);
                        v[0] = __dadd_rn(v[0], __dmul_rn(x, __dadd_rn(g, -a.b[e])));
                        v[1] = __dadd_rn(v[1], __dmul_rn(d, d));
                        v[2] = __dadd_rn(v[2], __dmul_rn(d, Ad));
                        v[3] = __dadd_rn(v[3], __dmul_rn(d, g));
                    }
                }
                const double r = warp_sum4_ordered(v, lane);
                if ((lane & 7) == 0) sm.red[c][warp][ordered_value(lane)] = r;
            }
        }
        __syncthreads();
        for (int w = tid; w < 32 * own_trees; w += NT) {  // (whole warps: 32 values per tree)
            const int c = w >> 5, q = (w >> 3) & 3, tree = blockIdx.x * own_trees + c;
            const double r = sum8_ordered(sm.red[c][w & 7][q]);
            if ((w & 7) == 0 && tree < trees) {
                if (nb > 1) word_store_double(slots + ((size_t)tree * 4 + q) * 2, r, tag);
                else terms[q * trees + tree] = r;
            }
        }
        if (nb > 1) {
            for (int w0 = tid; w0 < 4 * trees; w0 += 4 * NT) {
                double got[4];
                unsigned long long hi[4], lo[4];
                bool have = false;
                for (unsigned int it = 0; it < WORD_WAIT_LIMIT && !have; it++) {
                    have = true;
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int w = w0 + q * NT;
                        if (w < 4 * trees) word_load2(slots + (size_t)w * 2, hi[q], lo[q]);
                        else hi[q] = lo[q] = word_of(0u, tag);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        have &= word_valid(hi[q], tag) && word_valid(lo[q], tag);
                        got[q] = __hiloint2double((int)(unsigned int)hi[q], (int)(unsigned int)lo[q]);
                    }
                }
                ok &= have;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int w = w0 + q * NT;
                    if (w < 4 * trees) terms[(w & 3) * trees + (w >> 2)] = got[q];
                }
            }
        }
        if (nb > 1 && s >= 0 && tid >= 32 && tid < 32 + 2 * K) {
            const int e = (tid - 32) / K, k = tid - 32 - e * K;
            const long t = e ? t0 + Cb : t0 - 1;
            // left: the end of the block before; right: the start of the next one
            if (t >= 0 && t < T)
                ok &= word_wait_double(edges + (size_t)(e ? blockIdx.x + 1 : blockIdx.x - 1) * 4 * K + (e ? 0 : 2 * K) + 2 * k,
                                       tag, sm.hAd[e][k]);
        }
        if (!__syncthreads_and(ok)) {
            if (tid == 0) atomicExch(&a.st->error, 1);
            return;
        }
        if (s < 0) continue;
        // over the trees: thread b takes trees b, b + 256, ..., then the tree over the threads
        if (tid < 256) {
            double v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                v[q] = 0.0;
                for (int c = tid; c < trees; c += 256) v[q] = __dadd_rn(v[q], terms[q * trees + c]);
            }
            const double r = warp_sum4_ordered(v, lane);
            if ((lane & 7) == 0) sm.red[0][warp][ordered_value(lane)] = r;
        }
        __syncthreads();
        double tot = 0.0;  // warp 0: lane l's sum of value l & 3
        if (warp == 0) tot = __shfl_sync(0xffffffffu, sum8_ordered(sm.red[0][lane & 7][lane >> 3]), 8 * (lane & 3));
        if (warp == 0) f64_finish(sm.st, sm.step, tot, a.first && s == 0, lane);
        __syncthreads();
        if (sm.step.status != PASC_SPG_RUNNING) break;  // the same in every block
    }
    if (blockIdx.x == 0) {
        __syncthreads();
        const unsigned int *src = reinterpret_cast<const unsigned int *>(&sm.st);
        unsigned int *dst = reinterpret_cast<unsigned int *>(a.st);
        for (int q = tid; q < (int)(sizeof(Fp64DevState) / 4); q += NT)
            if (q != (int)(offsetof(Fp64DevState, error) / 4)) dst[q] = src[q];
    }
}

// x onto the simplex, timestep by timestep
template <int K>
__global__ void __launch_bounds__(F64_NT) fp64_start_project_kernel(double *x, long T)
{
    for (long t = (long)blockIdx.x * F64_NT + threadIdx.x; t < T; t += (long)gridDim.x * F64_NT) {
        double v[K];
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = x[t * K + k];
        project_f64<K>(v);
#pragma unroll
        for (int k = 0; k < K; k++) x[t * K + k] = v[k];
    }
}

// g = A x - b
template <int K>
__global__ void __launch_bounds__(F64_NT) fp64_start_gradient_kernel(const double *x, const double *b, double *g, long T,
                                                                     double coeff, const double *kc)
{
    for (long i = (long)blockIdx.x * F64_NT + threadIdx.x; i < T * K; i += (long)gridDim.x * F64_NT) {
        const long t = i / K;
        double row;
        if (t > 0) row = t < T - 1 ? __dadd_rn(fma(2.0, x[i], -x[i - K]), -x[i + K]) : __dadd_rn(x[i], -x[i - K]);
        else row = t < T - 1 ? __dadd_rn(x[i], -x[i + K]) : 0.0;
        g[i] = __dadd_rn(__dmul_rn(2.0 * (kc ? kc[i - t * K] : coeff), row), -b[i]);
    }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
#define F64_CASES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8)

static const void *f64_kernel_of(int K, bool ordered)
{
    switch (K) {
#define PASC_CASE(KK) \
    case KK: return ordered ? (const void *)spg_fp64_kernel<KK, true> : (const void *)spg_fp64_kernel<KK, false>;
        F64_CASES(PASC_CASE)
#undef PASC_CASE
        default: return nullptr;
    }
}

size_t fp64_words(int sms)
{
    // two sets: 8 words per tree (4 * SMs trees at most), end timesteps and barrier of 4 blocks per SM
    return (size_t)2 * (4 * sms * 8 + 4 * sms * (4 * KMAX_FUSED + 2));
}

// ORDERED up to its size limit, on the shortest tiles that leave one block per SM (T = 1e4, K = 2: 128
// timesteps 8.3 us per iteration, 256 10.3), STREAM beyond on blocks of equal shares, two per SM
// (K >= 6: one).
bool fp64_plan(int K, long T, int sms, Fp64Plan *p)
{
    if (!f64_kernel_of(K, false) || T < 1) return false;
    const long most = 4L * sms;  // trees
    p->ordered = T * K <= 256L * most;
    int per_sm = 0;
    for (;;) {
        const void *fn = f64_kernel_of(K, p->ordered);
        p->trees = (int)(p->ordered ? (T * K + 255) / 256 : most);
        p->threads = p->ordered ? F64_NT_ORDERED : F64_NT;
        p->smem = sizeof(double) * 4 * (size_t)(p->ordered ? std::max(256 * K, p->trees) : p->trees);
        // (the attribute belongs to the process: one value for every handle, more than any needs)
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, p->threads, p->smem);
        if (e != cudaSuccess || per_sm < 1) {
            cudaGetLastError();
            return false;
        }
        if (!p->ordered || (T + 255) / 256 <= (long)sms * per_sm) break;
        p->ordered = false;  // one cluster only: more blocks than fit
    }
    const long nmax = (long)sms * std::min(per_sm, 2);
    long c = std::max(1L, (T + nmax - 1) / nmax);
    if (p->ordered) {
        c = 64;
        while (c < 256 && (c * K % 256 != 0 || (T + c - 1) / c > sms)) c *= 2;
    }
    if (c > (1L << 30)) return false;
    p->C = (int)c;
    p->blocks = (int)((T + c - 1) / c);
    // (a block's trees have their place in shared memory)
    return p->ordered || (p->trees + p->blocks - 1) / p->blocks <= KMAX_FUSED;
}

cudaError_t launch_fp64_start(int K, double *x, const double *b, double *g, long T, double coeff, const double *kc,
                              int sms, cudaStream_t s)
{
    const int gp = (int)std::max(1L, std::min((T + F64_NT - 1) / F64_NT, (long)sms * 8));
    const int gg = (int)std::max(1L, std::min((T * K + F64_NT - 1) / F64_NT, (long)sms * 8));
    switch (K) {
#define PASC_CASE(KK)                                                                  \
    case KK:                                                                           \
        fp64_start_project_kernel<KK><<<gp, F64_NT, 0, s>>>(x, T);                     \
        fp64_start_gradient_kernel<KK><<<gg, F64_NT, 0, s>>>(x, b, g, T, coeff, kc);   \
        break;
        F64_CASES(PASC_CASE)
#undef PASC_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_fp64_iterations(int K, const Fp64Plan &p, const Fp64Args &a, cudaStream_t s)
{
    const void *fn = f64_kernel_of(K, p.ordered);
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {const_cast<Fp64Args *>(&a)};
    return cudaLaunchCooperativeKernel(fn, dim3(p.blocks), dim3(p.threads), args, p.smem, s);
}

}  // namespace pasc
