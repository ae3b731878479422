// image.cu -- the fused mixed-precision SPG sweep for image data: one timestep (T = 1) on the
// 4-neighbour pixel grid (BGMGraphGrid2D, include/general/algebra/graph/bgmgraphgrid2D.h:88-142)
// with the operator of blockgraphsparse.cpp:48-103 at T = 1: (A_hat x)_p = sum over the
// in-image neighbours n of p of (x_p - x_n).
//
// The general graph path (graph.cu) makes two passes per iteration over x and d in HBM; on the grid
// one pass does: a sweep reads x^c and d_{c+1}, applies x^{c+1} = x^c + beta d_{c+1}, and forms
// g^{c+1}, d_{c+2} and its sums from the neighbours' x^{c+1}, which it recomputes in a halo (read x, d
// and data, write x and d: (16 K + 4) bytes per pixel).  Recomputing d_{c+1} from x^c instead of
// storing it moves (8 K + 4) bytes but takes a second projection and stencil per pixel and a
// halo of 3; it was issue-bound at 388 instructions per owned pixel (K = 3).
//
// Each warp takes a strip tile: 32 columns (one per lane; 29 owned, one more on the left and two on
// the right) by th + 3 rows (the middle th owned), walked top to bottom with everything in registers:
//   row i      x^{c+1} = x^c + beta d (INIT: the projected start point);
//   row i - 1  g^{c+1}, d_{c+2} = P(x^{c+1} - alpha' g^{c+1}) - x^{c+1}; on owned pixels the objective,
//              d'd, g'd, the pair with the right neighbour, and the store of x^{c+1} and d_{c+2}; the
//              pair with the row above belongs to that row.
// Left and right neighbours come from the adjacent lanes (shuffles), up and down from the
// three-row windows; there is no block barrier in the sweep.  Strip tiles
// away from the image border run without range checks.
// Pixels outside the image hold zeros and are no one's neighbours.  The last block applies the
// step-length / GLL / stop logic of the 1-D sweeps (sweep_common.cuh).
#include <limits.h>
#include <algorithm>

#include "common.cuh"
#include "project.cuh"
#include "sweep_common.cuh"
#include "internal.h"

namespace pasc {

constexpr int IMG_TW = 29;                   // owned columns per warp (one lane per column)

// Threads of a block (each warp on its own strip tile), blocks per SM its registers leave room for, and
// rows a warp has in flight.
// A pixel's K values lie side by side, so a store of one value per lane touches a sector per lane: 2 K
// such stores per pixel were what bounded large images with many clusters, and the 160 to 200 registers
// of K >= 5 left one block of 8 warps per SM.  Even K >= 6 moves 8 or 16
// bytes at a time, K = 5 and 7 (odd: no wider alignment) write through shared memory.  us per sweep,
// recomputed direction / stored one, a value at a time / here: K = 5, 1920 x 1080 112 / 70 / 43, 4096 x 4096
// 474 / 398 / 274; K = 6 116 / 100 / 46, 497 / 705 / 291; K = 7 148 / 131 / 69, 597 / 978 / 417; K = 8 196 / 162 /
// 57, 935 / 1180 / 386.  Shapes tried at 4096 x 4096: K = 7 4 blocks, 2 rows 459, 3 blocks, 3 rows 417; K = 8 4
// blocks, 2 rows 500, 3 blocks, 3 rows 406, 4 blocks, 1 row 386; K = 6 5 blocks, 2 rows 384.  K = 3, two blocks of
// 256: 28.4 at 1920 x 1080; the compiler's own choice 31.2, three blocks 39.0.
template <int K>
struct ImgShape {
    static constexpr int NT = K <= 4 ? 256 : 128, BLOCKS = K <= 4 ? 2 : (K == 7 ? 3 : 4);
    static constexpr int PF = K <= 4 || K == 7 ? 3 : (K == 8 ? 1 : 2);
    static constexpr int VEC = K == 8 ? 4 : (K == 6 ? 2 : 1);  // values per load and store
    static constexpr bool STAGED = K == 5 || K == 7;           // stores through shared memory
};

template <int V>
struct ImgVec;
template <>
struct ImgVec<1> {
    using type = float;
};
template <>
struct ImgVec<2> {
    using type = float2;
};
template <>
struct ImgVec<4> {
    using type = float4;
};

// the K values of one pixel (rows of K * 4 bytes: aligned to 4 VEC)
template <int K>
__device__ __forceinline__ void image_load_pixel(const float *__restrict__ p, bool in, float (&v)[K])
{
    constexpr int V = ImgShape<K>::VEC;
    using T = typename ImgVec<V>::type;
#pragma unroll
    for (int k = 0; k < K; k += V) {
        T t{};
        if (in) t = __ldg(reinterpret_cast<const T *>(p + k));
        const float *f = reinterpret_cast<const float *>(&t);
#pragma unroll
        for (int j = 0; j < V; j++) v[k + j] = f[j];
    }
}
template <int K>
__device__ __forceinline__ void image_store_pixel(float *p, const float (&v)[K])
{
    constexpr int V = ImgShape<K>::VEC;
    using T = typename ImgVec<V>::type;
#pragma unroll
    for (int k = 0; k < K; k += V) {
        T t{};
        float *f = reinterpret_cast<float *>(&t);
#pragma unroll
        for (int j = 0; j < V; j++) f[j] = v[k + j];
        *reinterpret_cast<T *>(p + k) = t;
    }
}

// The owned pixels of a row, one per lane in v, written as consecutive values (whole warp; p: lane 0's
// pixel, of which and of the two last lanes' nothing is written; cols: columns of the image from there
// on; buf: 32 * K values of shared memory).
template <int K>
__device__ __forceinline__ void image_store_row(float *p, const float (&v)[K], int cols, float *buf)
{
    const int lane = threadIdx.x & 31, n = min(IMG_TW + 1, cols) * K;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < K; k++) buf[lane * K + k] = v[k];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < K; m++) {
        const int e = lane + 32 * m;
        if (e >= K && e < n) p[e] = buf[e];
    }
}

// x^c, d and data of staged row i of a strip tile (zeros outside the image)
template <int K, bool INIT, bool EDGE>
__device__ __forceinline__ void image_load_row(const ImageSweepArgs &a, const float *__restrict__ xin,
                                               const float *__restrict__ din, int i, int oy, int gx, bool colin, int H,
                                               int W, float (&x)[K], float (&d)[K], float &v)
{
    const int gy = oy + i;
    const bool in = colin && (!EDGE || (unsigned)gy < (unsigned)H);
    const long pix = (long)gy * W + gx;
    image_load_pixel<K>(xin + pix * K, in, x);
    if (!INIT) image_load_pixel<K>(din + pix * K, in, d);
    v = in ? __ldg(a.data + pix) : 0.f;
}

template <int K>
struct ImgSmem {
    static constexpr int WARPS = ImgShape<K>::NT / 32;
    double red[4 * WARPS];
    SpgDevState snap;
    float out[ImgShape<K>::STAGED ? WARPS * 32 * K : 1];
};

// sum over the in-image neighbours of (v_c - v_n); l, r from the neighbouring lanes, u, d from
// the rows above and below.  EDGE = false: all four neighbours exist.
template <bool EDGE>
__device__ __forceinline__ float grid_diff(float c, float l, float r, float u, float d, int gx, int gy, int W,
                                           int H)
{
    if (!EDGE) return ((c - l) + (c - r)) + ((c - u) + (c - d));
    float S = 0.f;
    if (gx > 0) S += c - l;
    if (gx < W - 1) S += c - r;
    if (gy > 0) S += c - u;
    if (gy < H - 1) S += c - d;
    return S;
}

// One strip tile of a warp: columns ox .. ox+31 (lane = column; lanes 1..29 owned), staged rows
// oy .. oy+th+2 (rows 1..th owned).
template <int K, bool INIT, bool EDGE>
__device__ __forceinline__ void image_strip(const ImageSweepArgs &a, const float *__restrict__ xin,
                                            const float *__restrict__ din, float *__restrict__ xout,
                                            float *__restrict__ dout, int ox, int oy, const float (&theta)[K],
                                            float beta, float a1, float coeff, float bscale, float *stage, KahanF &acc_f,
                                            FF &acc_dd, FF &acc_gd, FF &acc_dad)
{
    constexpr int IMG_PF = ImgShape<K>::PF;
    constexpr bool STAGED = ImgShape<K>::STAGED;
    const int lane = threadIdx.x & 31;
    const int W = a.W, H = a.H, th = a.th, rows = th + 3;
    const int gx = ox + lane;
    const bool colin = !EDGE || (unsigned)gx < (unsigned)W;
    const bool colown = colin && lane >= 1 && lane <= IMG_TW;
    float Y0[K], Y1[K], Y2[K], D0[K];  // x^{c+1} of rows i-2, i-1, i; d_{c+2} of row i-2
    float datY1 = 0.f, datY2 = 0.f;
#pragma unroll
    for (int k = 0; k < K; k++) Y0[k] = Y1[k] = Y2[k] = D0[k] = 0.f;
    // rows are prefetched IMG_PF ahead (ring of registers, static slots through the unrolled
    // inner loop) so that each warp keeps several row loads in flight
    float PX[IMG_PF][K], PD[IMG_PF][K], PV[IMG_PF];
#pragma unroll
    for (int q = 0; q < IMG_PF; q++)
        image_load_row<K, INIT, EDGE>(a, xin, din, q, oy, gx, colin, H, W, PX[q], PD[q], PV[q]);
#pragma unroll 1
    for (int i0 = 0; i0 < rows; i0 += IMG_PF) {
#pragma unroll
        for (int q = 0; q < IMG_PF; q++) {
            const int i = i0 + q;
            if (i >= rows) break;  // uniform
            // row i from slot q, which is refilled with row i + IMG_PF
            {
                const bool in = colin && (!EDGE || (unsigned)(oy + i) < (unsigned)H);
                float y[K];
#pragma unroll
                for (int k = 0; k < K; k++) y[k] = INIT ? PX[q][k] : fmaf(beta, PD[q][k], PX[q][k]);
                if (INIT) project_reg<K>(y);
#pragma unroll
                for (int k = 0; k < K; k++) {
                    Y0[k] = Y1[k];
                    Y1[k] = Y2[k];
                    Y2[k] = in ? y[k] : 0.f;
                }
                datY1 = datY2;
                datY2 = PV[q];
                if (i + IMG_PF < rows)
                    image_load_row<K, INIT, EDGE>(a, xin, din, i + IMG_PF, oy, gx, colin, H, W, PX[q], PD[q], PV[q]);
            }
            // row i - 1
            const int r = i - 1, gy = oy + r;
            if (r < 1) continue;  // uniform
            const bool in = colin && (!EDGE || (unsigned)gy < (unsigned)H);
            float g1[K], d1[K], fpart = 0.f;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float l = __shfl_up_sync(0xffffffffu, Y1[k], 1), rt = __shfl_down_sync(0xffffffffu, Y1[k], 1);
                const float S = grid_diff<EDGE>(Y1[k], l, rt, Y0[k], Y2[k], gx, gy, W, H);
                const float rr = datY1 - theta[k];
                const float bk = bscale * (rr * rr);
                g1[k] = fmaf(coeff, S, -bk);
                fpart += (g1[k] - bk) * Y1[k];
                d1[k] = fmaf(-a1, g1[k], Y1[k]);
            }
            project_reg<K>(d1);
#pragma unroll
            for (int k = 0; k < K; k++) d1[k] = in ? d1[k] - Y1[k] : 0.f;
            float part = 0.f;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float dr = __shfl_down_sync(0xffffffffu, d1[k], 1) - d1[k];
                if (r <= th && (!EDGE || gx < W - 1)) part = fmaf(dr, dr, part);  // (the pair with the right neighbour)
                const float dv = d1[k] - D0[k];
                if (r > 1 && in) part = fmaf(dv, dv, part);  // (the row above's pair with this one)
                D0[k] = d1[k];
            }
            if (colown && in) {
                acc_dad = ff_acc(acc_dad, ff_make(part));
                if (r <= th) {
                    acc_f.add(fpart);
                    float dd = 0.f, gd = 0.f;
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        dd = fmaf(d1[k], d1[k], dd);
                        gd = fmaf(g1[k], d1[k], gd);
                    }
                    if (!STAGED) {
                        const long pix = (long)gy * W + gx;
                        image_store_pixel<K>(xout + pix * K, Y1);
                        image_store_pixel<K>(dout + pix * K, d1);
                    }
                    acc_dd = ff_acc(acc_dd, ff_make(dd));
                    acc_gd = ff_acc(acc_gd, ff_make(gd));
                }
            }
            if (STAGED && r <= th && (!EDGE || (unsigned)gy < (unsigned)H)) {  // uniform
                const long first = (long)gy * W + ox;
                image_store_row<K>(xout + first * K, Y1, W - ox, stage);
                image_store_row<K>(dout + first * K, d1, W - ox, stage);
            }
        }
    }
}

template <int K, bool INIT>
__global__ void __launch_bounds__(ImgShape<K>::NT, ImgShape<K>::BLOCKS) image_sweep_kernel(ImageSweepArgs a)
{
    __shared__ ImgSmem<K> sm;
    SpgDevState *st = a.st;
    if (st->status != PASC_SPG_RUNNING) return;  // uniform across the grid
    const int cur = st->cur;
    const float *__restrict__ xin = cur ? a.xb1 : a.xb0, *__restrict__ din = cur ? a.db1 : a.db0;
    float *__restrict__ xout = cur ? a.xb0 : a.xb1, *__restrict__ dout = cur ? a.db0 : a.db1;
    const float beta = (float)st->beta, a1 = (float)st->alpha_cur;
    const float coeff = (float)st->coeff, bscale = (float)st->bscale;
    const int W = a.W, H = a.H, th = a.th;
    float theta[K];
#pragma unroll
    for (int k = 0; k < K; k++) theta[k] = a.theta[k];
    const int tiles_x = (W + IMG_TW - 1) / IMG_TW, tiles_y = (H + th - 1) / th;
    const int ntiles = tiles_x * tiles_y;
    const int warps = ImgShape<K>::NT / 32, warp = threadIdx.x >> 5;
    float *stage = sm.out + (ImgShape<K>::STAGED ? warp * 32 * K : 0);

    // (the pixels' terms are added in float-float: the sums then hardly depend on th and the grid)
    KahanF acc_f;
    FF acc_dd{0.f, 0.f}, acc_gd{0.f, 0.f}, acc_dad{0.f, 0.f};
    for (int tile = blockIdx.x * warps + warp; tile < ntiles; tile += gridDim.x * warps) {
        const int ty = tile / tiles_x, tx = tile - ty * tiles_x;
        const int ox = tx * IMG_TW - 1, oy = ty * th - 1;  // staged origin
        if (ox >= 0 && oy >= 0 && ox + 32 <= W && oy + th + 3 <= H)
            image_strip<K, INIT, false>(a, xin, din, xout, dout, ox, oy, theta, beta, a1, coeff, bscale, stage, acc_f,
                                        acc_dd, acc_gd, acc_dad);
        else
            image_strip<K, INIT, true>(a, xin, din, xout, dout, ox, oy, theta, beta, a1, coeff, bscale, stage, acc_f,
                                       acc_dd, acc_gd, acc_dad);
    }

    // d'A_hat d = sum over pairs of (d_p - d_n)^2; the finish step takes dAd = 2 coeff w[2]
    // (the factor 1/2 is exact in FP32)
    static_assert(sizeof(SpgDevState) % 8 == 0, "state snapshot");
    double w[4];
    FF v[4] = {FF{acc_f.s, acc_f.c}, acc_dd, FF{0.5f * acc_dad.hi, 0.5f * acc_dad.lo}, acc_gd};
    if (!sweep_grid_sum4<4>(v, reinterpret_cast<float2 *>(a.partials), blockIdx.x, &st->counter, gridDim.x, 0, 1,
                            reinterpret_cast<float2 *>(sm.red), w, st, &sm.snap, (int)sizeof(SpgDevState)))
        return;
    spg_finish_sweep<INIT>(st, sm.snap, cur, w);
}

template <int K, bool INIT>
static int image_blocks_t()
{
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, image_sweep_kernel<K, INIT>, ImgShape<K>::NT, 0);
    return nb > 0 ? nb : 1;
}

// blocks per SM of the regular form, and warps of a block
static int image_blocks_per_sm(int K, int *warps)
{
    switch (K) {
#define PASC_CASE(KK)                       \
    case KK:                                \
        *warps = ImgShape<KK>::NT / 32;     \
        return image_blocks_t<KK, false>();
        PASC_CASE(1) PASC_CASE(2) PASC_CASE(3) PASC_CASE(4)
        PASC_CASE(5) PASC_CASE(6) PASC_CASE(7) PASC_CASE(8)
#undef PASC_CASE
        default: return 0;
    }
}

// Rows of a strip tile and blocks.  A warp walks th + 3 rows for th owned ones (and about three
// more to fill its windows), all resident warps at once, in waves: the th whose whole waves cost
// least.  Measured at 1920 x 1080, K = 3: 15 (1.98 waves of 2432 warps) 31.0 us, 33 (0.91) 33.7, 9 (3.3)
// 32.6, 24 (1.24) 36.4, 63 (0.5) 40.6; at 640 x 480: 6 13.5, 15 14.9, 63 35.
void image_sweep_plan(int K, int W, int H, int sms, int *th, int *blocks)
{
    const int cols = (W + IMG_TW - 1) / IMG_TW;
    int warps = 1;
    const int per_sm = image_blocks_per_sm(K, &warps);
    const long resident = std::max(1L, (long)per_sm * sms * warps);
    long best = LONG_MAX, tiles = 1;
    for (int t = 3; t <= 63; t += 3) {
        const long n = (long)cols * ((H + t - 1) / t), cost = (n + resident - 1) / resident * (t + 6);
        if (cost < best) {
            best = cost;
            *th = t;
            tiles = n;
        }
    }
    *blocks = (int)std::max(1L, std::min((tiles + warps - 1) / warps, resident / warps));
}

cudaError_t launch_image_sweep(int K, bool init, int grid, const ImageSweepArgs &a, cudaStream_t s)
{
    switch (K) {
#define PASC_CASE(KK)                                                                                  \
    case KK:                                                                                           \
        if (init) image_sweep_kernel<KK, true><<<grid, ImgShape<KK>::NT, 0, s>>>(a);                   \
        else image_sweep_kernel<KK, false><<<grid, ImgShape<KK>::NT, 0, s>>>(a);                       \
        break;
        PASC_CASE(1) PASC_CASE(2) PASC_CASE(3) PASC_CASE(4)
        PASC_CASE(5) PASC_CASE(6) PASC_CASE(7) PASC_CASE(8)
#undef PASC_CASE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace pasc
