// kernels_cg.cu -- the FP32 conjugate gradients of the adjoint and the polish in one cooperative
// launch per solve, over the timesteps that can move.
//
// The vectors of the solve on S = {v : v_tk = 0 off F_t, sum_k v_tk = 0} vanish at every timestep with
// fewer than two free clusters, which is most of them (T = 1e6, K = 3, sigma 0.5, epssqr 30: 28% can
// move).  The active timesteps are listed once per solve; r, p, q and the correction d live at them
// alone, in the shared memory of the blocks, and an iteration (r and p to q = P A p and p'q; then d,
// r and r'r) moves nothing through HBM.  Block b owns C consecutive entries of the list, thread i
// M of them; rows are padded to an odd stride.  A neighbour in time that is not active has p = 0.
// The two sums of an iteration are three FP32 terms (f3.cuh), closer than FP64 and without the chains of
// the slow FP64 pipe; a block's sum is rounded to 48 bits once, when it is published.  They travel as
// tagged words (grid_words.cuh) together with r at the block's two ends, from which the neighbours bring
// their copies of p forward themselves.  Warp 0 adds the blocks' sums and forms alpha and beta; one block
// needs no exchange, and every warp does it for itself.
//
// Measured, loss and gradient (ms): two kernels per iteration over all timesteps / float-float sums, added
// and divided in every thread / here.  T = 1e6, K = 3, 643 iterations over 280 000 active timesteps 23.6 / 6.7 /
// 6.1; T = 3e5, K = 8 39 / 7.1 / 5.2; T = 1e5, K = 2 3.1 / 1.48 / 1.08; T = 3e4, K = 3 6.4 / 3.5 / 2.35; T = 1e4, K = 2 2.3 /
// 0.74 / 0.77; T = 5000, K = 3 3.7 / 1.07 / 1.29; T = 1000, K = 2 1.8 / 0.59 / 0.59.  What bounds it: the two
// exchanges, 1.5 to 1.8 us each between the two dies, and on few entries the chain of the sums (13 steps of
// a shuffle and 14 additions each).  How the blocks' polls fall between one another moves a solve on 2 to 32
// blocks by up to a third from one GPU to another.  FP64 sums in place of the three terms: 0.9 to 1.3 us more
// per iteration.  The neighbours' r awaited before a block publishes its sum: 0.2 to 0.7 us more.
//
// The scalars follow adjoint.cu: alpha = r'r / p'q, beta the ratio of successive r'r, until r'r has
// dropped by ADJ_INNER_TOL^2, maxit, or a breakdown (p'q <= 0).
#include <algorithm>

#include "common.cuh"
#include "f3.cuh"
#include "grid_words.cuh"
#include "internal.h"
#include "adjoint.h"

namespace pasc {

constexpr int CG_NT = 512;
constexpr int CG_WORDS = 4 + 2 * KMAX_FUSED;  // a block's words: two sums (high and low parts), r at its two ends

// entry flags above the mask's bits
constexpr unsigned int CG_LEFT = 1u << 8, CG_RIGHT = 1u << 9;    // the timestep has one before / after it
constexpr unsigned int CG_LACT = 1u << 10, CG_RACT = 1u << 11;  // which is the list's previous / next entry

template <int K>
struct CgSmem {
    float hr[2][K], hp[2][K];  // r, p of the entries before and after the block
    float red[2][CG_NT / 32][3];  // the warps' sums (p'q, r'r)
    float red2[CG_NT / 32][3];    // sums over 32 blocks each
    // of several blocks, from warp 0
    float alpha, beta;
    int status;
    int gave_up;               // a wait gave up
};

// a three-term sum as the nearest FP32 number and the rest
__device__ __forceinline__ FF ff_of(F3 v)
{
    float e;
    const float hi = f3_two_sum(v.a, v.b, e), r = e + v.c, h = hi + r;
    return FF{h, r - (h - hi)};
}

// a / b rounded to FP32, inv = __frcp_rn(b.hi): a quotient of the high parts and one correction from its
// remainder, off by 2^-44 before it is rounded (b far from 1: FP64, so that inv neither overflows nor is
// subnormal)
__device__ __forceinline__ float ff_quotient(FF a, FF b, float inv)
{
    if (!(b.hi > 0x1p-100f && b.hi < 0x1p100f)) return (float)(ff_value(a) / ff_value(b));
    const float q = __fmul_rn(a.hi, inv);
    const float rem = __fadd_rn(__fadd_rn(fmaf(-q, b.hi, a.hi), a.lo), -__fmul_rn(q, b.lo));
    return fmaf(rem, inv, q);
}

// A warp's share of a grid-wide sum.
__device__ __forceinline__ void cg_warp_sum(F3 v, float (*red)[3])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) v = f3_add(v, f3_shfl_xor(v, m));
    if (lane == 0) {
        red[warp][0] = v.a;
        red[warp][1] = v.b;
        red[warp][2] = v.c;
    }
}

// the sum over the block's warps (16 at most), in every lane of a warp: lanes 8 or 16 apart hold the same
__device__ __forceinline__ F3 cg_block_sum(const float (*red)[3])
{
    const int nw = blockDim.x >> 5, w = threadIdx.x & (nw > 8 ? 15 : 7);
    F3 v = w < nw ? F3{red[w][0], red[w][1], red[w][2]} : F3{0.f, 0.f, 0.f};
    if (nw > 8) v = f3_add(v, f3_shfl_xor(v, 8));
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) v = f3_add(v, f3_shfl_xor(v, m));
    return v;
}

// Several blocks: warp 0 publishes the block's sum, the first warps ask for the others' (one block per
// lane, so that a word is read until it is there and no longer), and warp 0 returns the sum over all
// blocks.  slots: the blocks' words (CG_WORDS apart), which: the sum's place among them.  A block's sum is
// rounded to 48 bits when it is published, once.  gave_up is set where a wait gave up.
__device__ __forceinline__ F3 cg_grid_sum(const float (*red)[3], float (*red2)[3], unsigned long long *slots, int which,
                                          unsigned int tag, int &gave_up)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = gridDim.x, polling = (nb + 31) >> 5;
    if (warp == 0) {
        const FF p = ff_of(cg_block_sum(red));
        if (lane == 0)
            word_store2(slots + (size_t)blockIdx.x * CG_WORDS + 2 * which, word_of(p.hi, tag), word_of(p.lo, tag));
    }
    F3 sum{0.f, 0.f, 0.f};
    if (tid < nb) {
        const unsigned long long *w = slots + (size_t)tid * CG_WORDS + 2 * which;
        unsigned long long hi = 0, lo = 0;
        bool have = false;
        for (unsigned int it = 0; it < WORD_WAIT_LIMIT && !have; it++) {
            word_load2(w, hi, lo);
            have = word_valid(hi, tag) && word_valid(lo, tag);
        }
        if (!have) gave_up = 1;
        sum = F3{word_float(hi), word_float(lo), 0.f};
    }
    if (warp < polling) {
        const int n = min(nb - 32 * warp, 32);  // lanes with a block
        __syncwarp();
        for (int m = n > 16 ? 16 : (n > 8 ? 8 : (n > 4 ? 4 : (n > 2 ? 2 : 1))); m >= 1; m >>= 1)
            sum = f3_add(sum, f3_shfl_xor(sum, m));
        if (polling > 1) {
            if (lane == 0) {
                red2[warp][0] = sum.a;
                red2[warp][1] = sum.b;
                red2[warp][2] = sum.c;
            }
            asm volatile("bar.sync 1, %0;" ::"r"(32 * polling) : "memory");
            if (warp == 0) {
                sum = lane < polling ? F3{red2[lane][0], red2[lane][1], red2[lane][2]} : F3{0.f, 0.f, 0.f};
                for (int m = polling > 4 ? (polling > 8 ? 8 : 4) : 2; m >= 1; m >>= 1) sum = f3_add(sum, f3_shfl_xor(sum, m));
            }
        }
    }
    return sum;
}

// after an update of r (r'r = v; rr before it, inv_rr its reciprocal): beta, and whether the solve goes on
__device__ __forceinline__ int cg_step(FF v, FF rr, float inv_rr, FF lim, bool last, float &beta)
{
    beta = ff_quotient(v, rr, inv_rr);
    if (!isfinite(v.hi)) return ADJ_BREAKDOWN;
    return (v.hi - lim.hi) + (v.lo - lim.lo) <= 0.f || last ? ADJ_INNER_DONE : ADJ_RUNNING;
}

template <int K>
__global__ void __launch_bounds__(CG_NT, 1) cg_resident_kernel(const __grid_constant__ CgArgs a)
{
    extern __shared__ __align__(16) float dyn[];
    __shared__ CgSmem<K> sm;
    const int tid = threadIdx.x, nt = blockDim.x, nb = gridDim.x, M = a.M;
    const int S = (M * K) | 1, rows = (a.C + M - 1) / M;
    float *rs = dyn, *ps = rs + (size_t)rows * S, *qs = ps + (size_t)rows * S, *ds = qs + (size_t)rows * S;
    unsigned short *fs = reinterpret_cast<unsigned short *>(ds + (size_t)rows * S);  // rows * M
    const int a0 = blockIdx.x * a.C, Cb = min(a.C, a.n - a0);

    for (int e = tid; e < Cb; e += nt) {
        const int n = a0 + e, i = e / M, j = e - i * M;
        const int t = a.list[n];
        unsigned int f = a.mask[t];
        if (t > 0) f |= CG_LEFT;
        if (t < a.T - 1) f |= CG_RIGHT;
        if (n > 0 && a.list[n - 1] == t - 1) f |= CG_LACT;
        if (n < a.n - 1 && a.list[n + 1] == t + 1) f |= CG_RACT;
        fs[i * M + j] = (unsigned short)f;
#pragma unroll
        for (int k = 0; k < K; k++) {
            rs[i * S + j * K + k] = a.r[(size_t)n * K + k];
            ps[i * S + j * K + k] = a.resume ? a.p[(size_t)n * K + k] : 0.f;
            ds[i * S + j * K + k] = a.resume ? a.d[(size_t)n * K + k] : 0.f;
        }
    }
    if (tid < 2 * K) {
        const int e = tid / K, k = tid - e * K, n = e ? a0 + Cb : a0 - 1;
        const bool in = n >= 0 && n < a.n;
        sm.hr[e][k] = in ? a.r[(size_t)n * K + k] : 0.f;
        sm.hp[e][k] = in && a.resume ? a.p[(size_t)n * K + k] : 0.f;
    }
    const int m = min(M, Cb - tid * M);
    const bool last = m > 0 && tid * M + m == Cb;
    float *r = rs + tid * S, *p = ps + tid * S, *q = qs + tid * S, *d = ds + tid * S;
    const unsigned short *fl = fs + tid * M;
    const float coeff = a.coeff;
    const double rr_in = a.st->rr, stop = ADJ_INNER_TOL * ADJ_INNER_TOL * a.st->rr_in0;
    // r'r (thread 0's counts; with one block all threads hold the same)
    FF rr{(float)rr_in, (float)(rr_in - (double)(float)rr_in)};
    const FF lim{(float)stop, (float)(stop - (double)(float)stop)};
    const int maxit = a.st->maxit;
    int it = a.st->it, status = ADJ_RUNNING;
    float beta = a.resume ? (float)a.st->beta : 0.f;
    if (tid == 0) sm.gave_up = 0;
    bool ok = true;
    __syncthreads();

    for (int s = 0; s < a.iterations; s++) {
        const unsigned int tag = a.tag + (unsigned int)s;
        unsigned long long *slots = a.slots + (size_t)(tag & 1u) * nb * CG_WORDS;
        const float inv_rr = __frcp_rn(rr.hi);
        // p = r + beta p at the thread's entries and the ones beside them
        float pc[K], pl[K], pe[K];
        if (m > 0) {
            const float *rl = tid ? r - S + (M - 1) * K : sm.hr[0], *pol = tid ? p - S + (M - 1) * K : sm.hp[0];
            const float *rn = last ? sm.hr[1] : r + S, *pon = last ? sm.hp[1] : p + S;
#pragma unroll
            for (int k = 0; k < K; k++) {
                pc[k] = fmaf(beta, p[k], r[k]);
                pl[k] = fmaf(beta, pol[k], rl[k]);
                pe[k] = fmaf(beta, pon[k], rn[k]);
            }
        }
        __syncthreads();  // the neighbours' rows were read
        F3 pq{0.f, 0.f, 0.f};
        if (m > 0) {
            if (tid == 0) {
#pragma unroll
                for (int k = 0; k < K; k++) sm.hp[0][k] = pl[k];
            }
            if (last) {
#pragma unroll
                for (int k = 0; k < K; k++) sm.hp[1][k] = pe[k];
            }
#pragma unroll 1
            for (int j = 0; j < m; j++) {
                const unsigned int f = fl[j];
                const bool end = j == m - 1;
                const int nf = __popc(f & 0xffu);
                float pn[K], y[K], sum = 0.f, part = 0.f;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    pn[k] = end ? pe[k] : fmaf(beta, p[(j + 1) * K + k], r[(j + 1) * K + k]);
                    y[k] = 0.f;
                    if (f & CG_LEFT) y[k] += 2.f * (pc[k] - ((f & CG_LACT) ? pl[k] : 0.f));
                    if (f & CG_RIGHT) y[k] += 2.f * (pc[k] - ((f & CG_RACT) ? pn[k] : 0.f));
                    y[k] *= coeff;
                    sum += ((f >> k) & 1u) ? y[k] : 0.f;
                }
                const float mean = sum / (float)nf;
#pragma unroll
                for (int k = 0; k < K; k++) {
                    y[k] = ((f >> k) & 1u) ? y[k] - mean : 0.f;
                    part = fmaf(pc[k], y[k], part);
                    p[j * K + k] = pc[k];
                    q[j * K + k] = y[k];
                    pl[k] = pc[k];
                    pc[k] = pn[k];
                }
                pq = f3_add(pq, part);
            }
        }
        cg_warp_sum(pq, sm.red[0]);
        __syncthreads();
        float alpha;
        if (nb == 1) {  // every warp for itself
            const FF sum = ff_of(cg_block_sum(sm.red[0]));
            if (!(sum.hi > 0.f) || !isfinite(sum.hi)) {
                status = ADJ_BREAKDOWN;
                break;
            }
            alpha = ff_quotient(rr, sum, __frcp_rn(sum.hi));
        } else {
            const FF sum = ff_of(cg_grid_sum(sm.red[0], sm.red2, slots, 0, tag, sm.gave_up));
            if (tid == 0) {
                const bool fine = sum.hi > 0.f && isfinite(sum.hi);
                sm.alpha = fine ? ff_quotient(rr, sum, __frcp_rn(sum.hi)) : 0.f;
                sm.status = fine ? ADJ_RUNNING : ADJ_BREAKDOWN;
            }
            __syncthreads();
            ok = sm.gave_up == 0;
            if (!ok) break;
            status = sm.status;
            if (status != ADJ_RUNNING) break;
            alpha = sm.alpha;
        }
        F3 rn{0.f, 0.f, 0.f};
#pragma unroll 1
        for (int j = 0; j < m; j++) {
            float part = 0.f;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const int e = j * K + k;
                d[e] = fmaf(alpha, p[e], d[e]);
                const float v = fmaf(-alpha, q[e], r[e]);
                r[e] = v;
                part = fmaf(v, v, part);
                // r at the block's ends, for the neighbours
                if (nb > 1) {
                    unsigned long long *own = slots + (size_t)blockIdx.x * CG_WORDS + 4;
                    if (tid == 0 && j == 0) word_store(own + k, word_of(v, tag));
                    if (last && j == m - 1) word_store(own + K + k, word_of(v, tag));
                }
            }
            rn = f3_add(rn, part);
        }
        cg_warp_sum(rn, sm.red[1]);
        __syncthreads();
        it++;
        if (nb == 1) {
            const FF sum = ff_of(cg_block_sum(sm.red[1]));
            status = cg_step(sum, rr, inv_rr, lim, it >= maxit, beta);
            rr = sum;
        } else {
            // the neighbours' r at this block's ends, awaited beside the sum (by the last warp: the
            // block's own share is published first)
            if (tid >= nt - 2 * K) {
                const int e = (tid - (nt - 2 * K)) / K, k = tid - (nt - 2 * K) - e * K, ob = (int)blockIdx.x + (e ? 1 : -1);
                if (ob >= 0 && ob < nb) {
                    const unsigned long long *w = slots + (size_t)ob * CG_WORDS + 4 + (e ? 0 : K) + k;
                    unsigned long long v = 0;
                    bool have = false;
                    for (unsigned int n = 0; n < WORD_WAIT_LIMIT && !have; n++) {
                        v = word_load(w);
                        have = word_valid(v, tag);
                    }
                    if (!have) sm.gave_up = 1;
                    sm.hr[e][k] = word_float(v);
                }
            }
            const FF sum = ff_of(cg_grid_sum(sm.red[1], sm.red2, slots, 1, tag, sm.gave_up));
            if (tid == 0) sm.status = cg_step(sum, rr, inv_rr, lim, it >= maxit, sm.beta);
            rr = sum;
            __syncthreads();
            ok = sm.gave_up == 0;
            if (!ok) break;
            status = sm.status;
            beta = sm.beta;
        }
        if (status != ADJ_RUNNING) break;
    }
    if (!ok) {
        if (tid == 0) {
            a.st->status = ADJ_BREAKDOWN;
            a.st->timeout = 1;
        }
        return;
    }
    __syncthreads();
    for (int e = tid; e < Cb; e += nt) {
        const int i = e / M, j = e - i * M;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const size_t g = (size_t)(a0 + e) * K + k;
            a.d[g] = ds[i * S + j * K + k];
            if (status == ADJ_RUNNING) {  // the next launch goes on from here
                a.r[g] = rs[i * S + j * K + k];
                a.p[g] = ps[i * S + j * K + k];
            }
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.st->rr = ff_value(rr);
        a.st->beta = beta;
        a.st->it = it;
        a.st->status = status;
    }
}

// ---------------------------------------------------------------------------------------
// the list of active timesteps (two or more free clusters), in order of time
// ---------------------------------------------------------------------------------------
constexpr int LIST_NT = 256, LIST_PER = 8, LIST_SPAN = LIST_NT * LIST_PER;  // timesteps per block

// position of a warp's flagged lanes among the block's, rounds of LIST_NT timesteps
__global__ void __launch_bounds__(LIST_NT) cg_list_count_kernel(const unsigned int *mask, long T, int *counts)
{
    const long t0 = (long)blockIdx.x * LIST_SPAN;
    int n = 0;
    for (int r = 0; r < LIST_PER; r++) {
        const long t = t0 + r * LIST_NT + threadIdx.x;
        n += __syncthreads_count(t < T && __popc(mask[t]) >= 2);
    }
    if (threadIdx.x == 0) counts[blockIdx.x] = n;
}

// counts to exclusive prefix sums, total in counts[n]
__global__ void __launch_bounds__(1024) cg_list_scan_kernel(int *counts, int n)
{
    __shared__ int warp_sum[32], carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    for (int b = 0; b < n; b += 1024) {
        __syncthreads();
        const int i = b + threadIdx.x, v = i < n ? counts[i] : 0;
        int s = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
        }
        if (lane == 31) warp_sum[warp] = s;
        __syncthreads();
        int before = carry;
        for (int w = 0; w < warp; w++) before += warp_sum[w];
        if (i < n) counts[i] = before + s - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry = before + s;
    }
    __syncthreads();
    if (threadIdx.x == 0) counts[n] = carry;
}

__global__ void __launch_bounds__(LIST_NT) cg_list_fill_kernel(const unsigned int *mask, long T, const int *offsets,
                                                               int *list)
{
    __shared__ int warps[LIST_NT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long t0 = (long)blockIdx.x * LIST_SPAN;
    int base = offsets[blockIdx.x];
    for (int r = 0; r < LIST_PER; r++) {
        const long t = t0 + r * LIST_NT + threadIdx.x;
        const bool on = t < T && __popc(mask[t]) >= 2;
        const unsigned int b = __ballot_sync(0xffffffffu, on);
        if (lane == 0) warps[warp] = __popc(b);
        __syncthreads();
        int at = base, all = 0;
        for (int w = 0; w < LIST_NT / 32; w++) {
            at += w < warp ? warps[w] : 0;
            all += warps[w];
        }
        if (on) list[at + __popc(b & ((1u << lane) - 1u))] = (int)t;
        base += all;
        __syncthreads();
    }
}

size_t cg_list_counts(long T) { return (size_t)((T + LIST_SPAN - 1) / LIST_SPAN) + 1; }

cudaError_t launch_cg_list(const unsigned int *mask, long T, int *counts, int *list, cudaStream_t s)
{
    const int nb = (int)((T + LIST_SPAN - 1) / LIST_SPAN);
    cg_list_count_kernel<<<nb, LIST_NT, 0, s>>>(mask, T, counts);
    cg_list_scan_kernel<<<1, 1024, 0, s>>>(counts, nb);
    cg_list_fill_kernel<<<nb, LIST_NT, 0, s>>>(mask, T, counts, list);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static const void *cg_kernel_of(int K)
{
    switch (K) {
#define PASC_CASE(KK) case KK: return (const void *)cg_resident_kernel<KK>;
        PASC_CASE(1) PASC_CASE(2) PASC_CASE(3) PASC_CASE(4)
        PASC_CASE(5) PASC_CASE(6) PASC_CASE(7) PASC_CASE(8)
#undef PASC_CASE
        default: return nullptr;
    }
}

size_t cg_words(int sms) { return (size_t)2 * sms * CG_WORDS; }

// One block up to 512 entries (K <= 4: 1024), then 256 entries per block up to one block per SM; false where
// the entries do not fit in shared memory.
bool cg_plan(int K, long n, int sms, CgPlan *p)
{
    const void *fn = cg_kernel_of(K);
    cudaFuncAttributes fa;
    int dev = 0, optin = 0, per_sm = 0;
    if (!fn || n < 1 || cudaFuncGetAttributes(&fa, fn) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const long nb = n <= (K <= 4 ? 1024 : 512) ? 1 : std::min((long)sms, (n + 255) / 256);
    const long C = (n + nb - 1) / nb, M = (C + CG_NT - 1) / CG_NT, rows = (C + M - 1) / M;
    const size_t smem = sizeof(float) * 4 * rows * ((M * K) | 1) + sizeof(short) * rows * M, room = optin - fa.sharedSizeBytes;
    if (smem > room) return false;
    p->blocks = (int)((n + C - 1) / C);
    p->C = (int)C;
    p->M = (int)M;
    // (at least the warps that poll the blocks' words)
    p->threads = (int)std::max((rows + 31) / 32, (long)(p->blocks + 31) / 32) * 32;
    p->smem = smem;
    // (the same limit for every handle: all a block can have)
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, p->threads, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        return false;
    }
    return true;
}

cudaError_t launch_cg(int K, const CgPlan &p, const CgArgs &a, cudaStream_t s)
{
    const void *fn = cg_kernel_of(K);
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {const_cast<CgArgs *>(&a)};
    return cudaLaunchCooperativeKernel(fn, dim3(p.blocks), dim3(p.threads), args, p.smem, s);
}

}  // namespace pasc
