// FP64 Jacobi-PCG as one cooperative kernel (pcg_coop.cu).
#pragma once
#include "solve.h"

namespace phgb {

// One solve of A x = b from the initial guess in x: p (and for small systems p2
// and z) are what the product gathers, the other vectors stay on chip.
struct PcgRun {
    CsrView A;
    int64_t nnz;
    int32_t *cols;       // the blocks' copy of the matrix: pcg_coop_entries() each
    double *vals;
    double *x, *p, *p2, *z;   // n each
    const double *b, *D;
    double rtol, btol, atol;
    int maxit;
    double *hist;        // optional: ||r|| after each iteration, [0] = ||r0||
    double *exchange;    // coop_exchange_doubles(), zero before the launch
    int sms;             // multiprocessors of the stream (stream_sms)
    int max_row;         // a longer row declines the solve; set by the launch
    PcgState *st;        // out: nits, residual, status
};

int coop_exchange_doubles();

// Multiprocessors that kernels of the stream can run on: the device's, or those
// of the green context the stream belongs to (pcg_coop.cu).  A grid of more
// blocks than these hold would wait for blocks that are not resident.
int stream_sms(cudaStream_t s);

// Entries of the matrix copy a solve of n rows and nnz entries makes on sms
// multiprocessors (stream_sms), -1 when it is too large for the kernel.
int64_t pcg_coop_entries(int64_t n, int64_t nnz, int sms);
cudaError_t launch_pcg_coop(const PcgRun &R, cudaStream_t s);

}  // namespace phgb
