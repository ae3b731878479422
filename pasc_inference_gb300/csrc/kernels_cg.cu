// kernels_cg.cu -- the FP32 conjugate gradients of the adjoint and the polish in one cooperative
// launch per solve, over the timesteps that can move.
//
// The vectors of the solve on S = {v : v_tk = 0 off F_t, sum_k v_tk = 0} vanish at every timestep with
// fewer than two free clusters, which is most of them (T = 1e6, K = 3, sigma 0.5, epssqr 30: 28% can
// move).  The active timesteps are listed once per solve; r, p, q and the correction d live at them
// alone, in the shared memory of the blocks, and an iteration (r and p to q = P A p and p'q; then d,
// r and r'r) moves nothing through HBM.  Block b owns C consecutive entries of the list, thread i
// M of them; rows are padded to an odd stride.  A neighbour in time that is not active has p = 0.
// The two sums of an iteration are FP64 (three FP32 terms up to a warp, f3.cuh) and travel as tagged
// words (grid_words.cuh) together with r at the block's two ends, from which the neighbours bring their
// copies of p forward themselves.  Warp 0 adds the blocks' sums and forms alpha and beta.  Measured at
// T = 1e6, K = 3, 280 000 active timesteps: 26 us per iteration with one kernel per half iteration over all
// timesteps, 6.9 here; 4.5 on eleven blocks, about 4 on one.  What bounds it: the two exchanges, 1.5 to 1.8 us each
// between the two dies, and on few blocks warp 0's chain of FP64 operations (float-float sums and
// quotients in every thread, with fewer bits, took 0.9 to 1.3 us less there, and up to 1.1 us more where many
// entries share a block: T = 3e5, K = 8 7.1 against 5.9 ms an adjoint).
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
constexpr int CG_WORDS = 4 + 2 * KMAX_FUSED;  // a block's words: two sums (FP64), r at its two ends

// entry flags above the mask's bits
constexpr unsigned int CG_LEFT = 1u << 8, CG_RIGHT = 1u << 9;    // the timestep has one before / after it
constexpr unsigned int CG_LACT = 1u << 10, CG_RACT = 1u << 11;  // which is the list's previous / next entry

template <int K>
struct CgSmem {
    float hr[2][K], hp[2][K];  // r, p of the entries before and after the block
    float red[CG_NT / 32][3];  // the warps' sums
    // of the whole grid, from warp 0
    float alpha, beta;
    int status, it;
    int gave_up;               // a wait gave up
};

// sum over lanes 0 .. n - 1 (the others hold 0), in lane 0
__device__ __forceinline__ double warp_sum_of(double v, int n)
{
    for (int m = n > 16 ? 16 : (n > 8 ? 8 : (n > 4 ? 4 : (n > 2 ? 2 : 1))); m >= 1; m >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, m);
    return v;
}

// (float)(a / b).  A quotient of FP32 numbers and one correction from its FP64 remainder: off by 2^-46
// before it is rounded to FP32.  (An FP64 division in its place: 0.2 to 0.4 us
// more per iteration.)
__device__ __forceinline__ float cg_quotient(double a, double b)
{
    const float fa = (float)a, fb = (float)b;
    if (!(fabsf(fa) > 0x1p-60f && fabsf(fa) < 0x1p60f && fabsf(fb) > 0x1p-60f && fabsf(fb) < 0x1p60f)) return (float)(a / b);
    const float q = fa / fb;
    return q + (float)fma(-(double)q, b, a) / fb;
}

// A warp's share of a grid-wide sum: three FP32 terms within the warp (f3.cuh), FP64 beyond.
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

// Warp 0: the sum over the block's warps, published, and the sum over all blocks, in lane 0.
// slots: the blocks' words (CG_WORDS apart), which: the sum's place among them.  ok turns false
// where a wait gave up.
__device__ __forceinline__ double cg_grid_sum(const float (*red)[3], unsigned long long *slots, int which,
                                              unsigned int tag, bool &ok)
{
    constexpr int POLL = 5;  // words a lane has in flight
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, nb = gridDim.x;
    const double own = warp_sum_of(lane < nw ? f3_value(F3{red[lane][0], red[lane][1], red[lane][2]}) : 0.0, nw);
    if (nb == 1) return own;
    if (lane == 0) word_store_double(slots + (size_t)blockIdx.x * CG_WORDS + 2 * which, own, tag);
    double sum = 0.0;
    for (int b0 = lane; b0 < nb; b0 += 32 * POLL) {
        unsigned long long hi[POLL], lo[POLL];
        bool have = false;
        for (unsigned int it = 0; it < WORD_WAIT_LIMIT && !have; it++) {
            have = true;
#pragma unroll
            for (int q = 0; q < POLL; q++) {
                const int b = b0 + 32 * q;
                if (b < nb) word_load2(slots + (size_t)b * CG_WORDS + 2 * which, hi[q], lo[q]);
                else hi[q] = lo[q] = word_of(0u, tag);
            }
#pragma unroll
            for (int q = 0; q < POLL; q++) have &= word_valid(hi[q], tag) && word_valid(lo[q], tag);
        }
        ok &= have;
#pragma unroll
        for (int q = 0; q < POLL; q++) sum += __hiloint2double((int)(unsigned int)hi[q], (int)(unsigned int)lo[q]);
    }
    return warp_sum_of(sum, nb);
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
    double rr = a.st->rr;  // (thread 0)
    const double stop = ADJ_INNER_TOL * ADJ_INNER_TOL * a.st->rr_in0;
    const int maxit = a.st->maxit;
    int it = a.st->it, status = ADJ_RUNNING;
    float beta = a.resume ? (float)a.st->beta : 0.f;
    if (tid == 0) sm.gave_up = 0;
    bool ok = true;
    __syncthreads();

    for (int s = 0; s < a.iterations; s++) {
        const unsigned int tag = a.tag + (unsigned int)s;
        unsigned long long *slots = a.slots + (size_t)(tag & 1u) * nb * CG_WORDS;
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
        cg_warp_sum(pq, sm.red);
        __syncthreads();
        if (tid < 32) {
            const double sum = cg_grid_sum(sm.red, slots, 0, tag, ok);
            if (!__all_sync(0xffffffffu, ok)) sm.gave_up = 1;
            if (tid == 0) {
                const bool fine = sum > 0.0 && isfinite(sum);
                sm.alpha = fine ? cg_quotient(rr, sum) : 0.f;
                sm.status = fine ? ADJ_RUNNING : ADJ_BREAKDOWN;
            }
        }
        __syncthreads();
        ok = sm.gave_up == 0;
        if (!ok) break;
        status = sm.status;
        if (status != ADJ_RUNNING) break;
        const float alpha = sm.alpha;
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
        // (the neighbours' r at this block's ends are awaited with the sum)
        if (nb > 1 && tid >= nt - 2 * K) {
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
        cg_warp_sum(rn, sm.red);
        __syncthreads();
        if (tid < 32) {
            const double sum = cg_grid_sum(sm.red, slots, 1, tag, ok);
            if (!__all_sync(0xffffffffu, ok)) sm.gave_up = 1;
            if (tid == 0) {
                sm.beta = cg_quotient(sum, rr);
                sm.it = it + 1;
                sm.status = !isfinite(sum) ? ADJ_BREAKDOWN : (sum <= stop || it + 1 >= maxit ? ADJ_INNER_DONE : ADJ_RUNNING);
            }
            rr = sum;
        }
        __syncthreads();
        ok = sm.gave_up == 0;
        if (!ok) break;
        status = sm.status;
        beta = sm.beta;
        it = sm.it;
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
        a.st->rr = rr;
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

// One block up to 512 entries, then 256 entries per block up to one block per SM; false where the
// entries do not fit in shared memory.
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
    const long nb = n <= 512 ? 1 : std::min((long)sms, (n + 255) / 256);
    const long C = (n + nb - 1) / nb, M = (C + CG_NT - 1) / CG_NT, rows = (C + M - 1) / M;
    const size_t smem = sizeof(float) * 4 * rows * ((M * K) | 1) + sizeof(short) * rows * M, room = optin - fa.sharedSizeBytes;
    if (smem > room) return false;
    p->blocks = (int)((n + C - 1) / C);
    p->C = (int)C;
    p->M = (int)M;
    p->threads = (int)((rows + 31) / 32) * 32;
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
