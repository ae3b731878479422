// adjoint.h -- state of the conjugate gradients, shared by adjoint.cu and kernels_cg.cu.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace pasc {

enum { ADJ_RUNNING = 0, ADJ_CONVERGED = 1, ADJ_MAXIT = 2, ADJ_BREAKDOWN = 4, ADJ_INNER_DONE = 8 };

constexpr double ADJ_INNER_TOL = 1e-4;  // residual reduction of one FP32 refinement step

struct AdjDevState {
    double rr, rr0, pq, alpha, beta, tol;
    double free_dims;
    int it, maxit, status, pcur;
    unsigned int counter;
    double rr_in0;  // FP32 refinement: r'r at the start of the current inner solve
    int outer;
    unsigned int fall;  // clusters free at every timestep (their cluster-constant, zero-sum
                        // vectors are the null space of P A P on S)
    double nullc[8];    // component of lambda along that null space, per cluster
    double rr64;        // FP32 refinement: FP64 r'r of the last residual
    double rscale;      // FP32 refinement: the residual is handed to the FP32 solve times this
                        // (its rms brought to 1: a small residual would otherwise lose its
                        // products p'q to FP32 underflow), the correction divided by it
    int timeout;        // a bounded wait gave up (kernels_cg.cu)
};

// FP32 conjugate gradients over the active timesteps (kernels_cg.cu)
struct CgPlan {
    int blocks, threads;
    int C, M;  // entries of the list per block and per thread
    size_t smem;
};
struct CgArgs {
    const int *list;           // the active timesteps, ascending
    const unsigned int *mask;  // free clusters of every timestep
    float *r, *p, *d;          // n x K: residual in; correction out (r and p where the solve is not done)
    AdjDevState *st;
    unsigned long long *slots;  // cg_words(sms) words
    unsigned int tag;
    long T;
    int n, C, M;
    int iterations;  // at most this many
    int resume;      // go on from r, p, d and the state
    float coeff;
};
size_t cg_list_counts(long T);  // ints of counts
// counts[last] holds the number of active timesteps
cudaError_t launch_cg_list(const unsigned int *mask, long T, int *counts, int *list, cudaStream_t s);
bool cg_plan(int K, long n, int sms, CgPlan *p);
size_t cg_words(int sms);
cudaError_t launch_cg(int K, const CgPlan &p, const CgArgs &a, cudaStream_t s);

}  // namespace pasc
