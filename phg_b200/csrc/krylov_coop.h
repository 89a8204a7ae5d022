// BiCGstab and GMRES as cooperative kernels (bicgstab_coop.cu, gmres_coop.cu).
#pragma once
#include "bicgstab.h"
#include "gmres.h"
#include "solve.h"

namespace phgb {

// One BiCGstab solve from the initial guess in x: ph and sh (n each) are the
// vectors the products gather, the others stay on chip.
struct BicgRun {
    CsrView A;
    int64_t nnz;
    int32_t *cols;       // the blocks' copy of the matrix: bicg_coop_entries() each
    double *vals;
    double *x, *ph, *sh;
    const double *b, *D;
    double rtol, btol, atol;
    int maxit;
    double *hist;        // optional: ||r|| after each iteration
    double *exchange;    // coop_exchange_doubles(), zero before the launch
    int sms;             // multiprocessors of the stream (stream_sms)
    int max_row;         // a longer row declines the solve; set by the launch
    BicgState *st;       // out: nits, residual, status (BICG_*)
};

// One GMRES_r or FLGMRES_r solve (augk < 0: GMRES_r), basis vectors at
// distance `stride` as GmresBuffers keeps them.
struct GmresRun {
    CsrView A;
    int64_t nnz;
    int32_t *cols;       // the blocks' copy of the matrix: gmres_coop_entries() each
    double *vals;
    double *x;
    const double *b, *D;
    double *V, *F, *Z;   // V_0..; F_1.., Z_0.. for FLGMRES_r
    int64_t stride;
    double rtol, btol, atol;
    int maxit, mk, augk; // steps of the first cycle, augmenting corrections
    double *exchange;
    int sms;             // multiprocessors of the stream (stream_sms)
    int max_row;         // a longer row declines the solve; set by the launch
    GmresState *st;      // out: nits, residual, status (GMRES_*, kStatus*)
};

// Entries of the matrix copy a solve makes on sms multiprocessors (stream_sms),
// -1 when it is too large for the kernel.
int64_t bicg_coop_entries(int64_t n, int64_t nnz, int sms);
int64_t gmres_coop_entries(int64_t n, int64_t nnz, int restart, int sms);
cudaError_t launch_bicg_coop(const BicgRun &R, cudaStream_t s);
cudaError_t launch_gmres_coop(const GmresRun &R, cudaStream_t s);

}  // namespace phgb
