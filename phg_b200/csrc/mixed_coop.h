// Mixed-precision Jacobi-PCG as one cooperative kernel (mixed_coop.cu).
#pragma once
#include "solve.h"

namespace phgb {

struct MixedResult {
    double residual;             // FP64 ||b - A x||
    int nits, nupdates, status;  // PCG_*, kStatus*
};

// One solve of A x = b from the initial guess in x: u (n) is the vector the
// FP32 product gathers, the other FP32 vectors stay on chip.
struct MixedRun {
    CsrView A;
    int64_t nnz;
    int32_t *cols;       // the blocks' copy of the matrix: mixed_coop_entries() each
    float *vals32;
    double *vals64;
    double *x;
    float *u;
    const double *b, *D;
    double rtol, btol, atol, delta;
    int maxit;
    double *exchange;    // coop_exchange_doubles(), zero before the launch
    int sms;             // multiprocessors of the stream (stream_sms)
    int max_row;         // a longer row declines the solve; set by the launch
    MixedResult *out;
};

// Entries of the matrix copy a solve of n rows and nnz entries makes on sms
// multiprocessors (stream_sms), -1 when it is too large for the kernel.
int64_t mixed_coop_entries(int64_t n, int64_t nnz, int sms);
cudaError_t launch_mixed_coop(const MixedRun &R, cudaStream_t s);

}  // namespace phgb
