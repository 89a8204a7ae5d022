// FP64 Jacobi-PCG (solver_pcg, solver-phg.c:485-604) as one cooperative
// kernel: the initial residual, every iteration and the stopping rule.
//
// Each block (one an SM) owns every gridDim-th slice of 32 rows and keeps their
// part of the vectors in shared memory; only the direction p, which the other
// blocks' products gather, and x go through L2.  An iteration is three phases
// between grid barriers:
//   direction  p = z + beta p
//   product    w = A p, and p.w                              (sum)
//   update     r -= alpha w, z = r / diag, ||r||^2 and r.z    (sum; x += alpha p
//              runs behind the barrier)
// Where a barrier costs more than gathers (FUSED, small systems), z goes through
// L2 too and the product gathers z + beta p from z and the last direction, so
// that the direction needs no barrier of its own; the values are the same.
// What bounds it: up to 40,000 rows the barriers, about 1.4 us each (two in the
// FUSED form, which systems of that size take up to 1.5 million entries, three
// otherwise), and the latency of the phases between them: at P1 36k rows a warp
// waits at a barrier 27 of the 38 cycles it spends on an instruction.  From
// 100,000 rows on the product, which reads the matrix from L2 (up to some 10
// million entries) at the rate its gathers allow: at P2 531k rows 42% of the DRAM
// rate, 55% of L1's, 10 of 21 cycles waiting for loads and 4 at barriers.  Time
// per iteration against the same recurrence as three launches in a graph loop: P1
// 1,331 rows 6.7 us (16.3), P1 36k 6.9 (18.9), P1 133k 10.4 (20.7), P1 389k 18.5
// (33.3), P2 69k 11.3 (23.4), P2 250k 22.5 (37.4), P2 531k 38.5 (58.5), P3 227k
// 30.8 (52.2); and a solve needs no tuned layout, no graph and one host wait: 71
// us instead of 180 before the first iteration.  (Measured and left: the rows in one contiguous run per block, as
// CSR rows of 4 to 16 lanes, as a stream over the entries, or sorted by length:
// 25 to 29 us on P1 389k and over 100 on P2 531k, whose vertex rows then sit on
// a third of the blocks.)
#include "coop_rows.cuh"
#include "grid_sync.cuh"
#include "pcg_coop.h"

#include <cudaTypedefs.h>
#include <float.h>
#include <math.h>

namespace phgb {

namespace {

struct PcgScalars {
    double alpha, beta;
    double rb, tol, rz, residual;
    int nits, status, run, nonzero, declined;
};

__device__ __forceinline__ bool is_zero(double a) { return fabs(a) < 10.0 * DBL_MIN; }   // utils.h:451

template <int H, bool FUSED>
__global__ void __launch_bounds__(kCoopThreads, 1)
pcg_coop_kernel(const PcgRun R) {
    extern __shared__ double s_vec[];
    __shared__ CoopShared sh;
    __shared__ PcgScalars S;
    __shared__ int next_unit;
    CoopGrid<> G(R.exchange, &sh);
    const int t = threadIdx.x;
    const unsigned n = (unsigned)R.A.n;
    const int m = coop_places(n);
    double *sr = s_vec, *sw = sr + m, *sp = sw + m, *sD = sp + m;   // of the block's places
    CoopRows<H> L(n, sD + m, &next_unit, R.cols);
    const bool first = blockIdx.x == 0;

    // ||b|| and |x|_1 (solver-phg.c:498-518)
    double v[2], d[1], v3[3] = {0.0, 0.0, 0.0};
    for (int i = t; i < m; i += kCoopThreads) {
        const unsigned row = L.row(i);
        const bool in = row < n;
        const double bi = in ? R.b[row] : 0.0;
        sr[i] = bi;
        sw[i] = 0.0;
        sp[i] = 0.0;
        sD[i] = in ? R.D[row] : 1.0;
        if (in) {
            v3[0] += fabs(R.x[row]);
            v3[1] += bi * bi;
            if (R.A.rp[row + 1] - R.A.rp[row] > R.max_row) v3[2] = 1.0;
        }
    }
    if (!G.sum(v3, [&](const double *s) {
            S.rb = sqrt(s[1]);
            S.nonzero = !is_zero(s[0] / (double)n);
            S.nits = 0;
            S.status = PCG_RUNNING;
            S.residual = 0.0;
            S.run = !is_zero(S.rb);
            S.declined = s[2] != 0.0;
            if (first && S.declined) {
                R.st->status = kStatusDeclined;
            } else if (first && !S.run) {
                if (R.hist != nullptr) R.hist[0] = 0.0;
                R.st->nits = 0;
                R.st->residual = 0.0;
                R.st->status = PCG_RUNNING;
            }
        })) {
        if (t == 0) R.st->status = kStatusPassLimit;
        return;
    }
    if (S.declined) return;
    if (!S.run) {
        for (int i = t; i < m; i += kCoopThreads)
            if (L.row(i) < n) R.x[L.row(i)] = 0.0;
        return;
    }
    L.build(R.A, [&](int q, double value) { R.vals[q] = value; });
    __syncthreads();
    // r = b - A x, or b when x = 0
    if (S.nonzero) {
        L.template product<false>(R.vals, (const double *)R.x, sw);
        for (int i = t; i < m; i += kCoopThreads) sr[i] -= sw[i];
    }
    v[0] = v[1] = 0.0;
    for (int i = t; i < m; i += kCoopThreads) {
        const double ri = sr[i], zi = ri / sD[i];
        sw[i] = zi;
        if (FUSED && L.row(i) < n) {
            R.z[L.row(i)] = zi;
            R.p[L.row(i)] = 0.0;
        }
        v[0] += ri * ri;
        v[1] += ri * zi;
    }
    bool ok = G.sum(v, [&](const double *s) {
        const double res = sqrt(s[0]);
        double tol = res * R.rtol;   // get_tol (solver-phg.c:104-115)
        if (tol < S.rb * R.btol) tol = S.rb * R.btol;
        if (tol < R.atol) tol = R.atol;
        S.tol = tol;
        S.rz = s[1];
        S.residual = res;
        S.beta = 0.0;
        if (first && R.hist != nullptr) R.hist[0] = res;
        if (!isfinite(s[1])) S.status = kStatusBadStart;
        S.run = S.status == PCG_RUNNING && res > tol && R.maxit > 0;
    });
    // (`start` with a beta of 0 would do as in FUSED, but the compiler then orders
    // the product's gathers worse: P2 531k rows 45.9 us instead of 38.4)
    bool start = true;
    double *from = R.p, *to = R.p2;   // FUSED: the last direction and the next
    while (ok && S.run) {
        const double beta = S.beta;
        if constexpr (FUSED) {
            const double *pold = from, *zold = R.z;
            for (int i = t; i < m; i += kCoopThreads) {
                const double pi = beta * sp[i] + sw[i];
                sp[i] = pi;
                if (L.row(i) < n) to[L.row(i)] = pi;
            }
            __syncthreads();
            L.template product<false>(R.vals, [=](int32_t c) { return beta * pold[c] + zold[c]; }, sw);
            double *other = from;
            from = to;
            to = other;
        } else {
            for (int i = t; i < m; i += kCoopThreads) {
                const double pi = start ? sw[i] : beta * sp[i] + sw[i];
                sp[i] = pi;
                if (L.row(i) < n) R.p[L.row(i)] = pi;
            }
            start = false;
            if (!(ok = G.sync())) break;
            L.template product<false>(R.vals, (const double *)R.p, sw);
        }
        d[0] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) d[0] += sp[i] * sw[i];
        ok = G.sum(d, [&](const double *s) {
            if (s[0] == 0.0) {
                S.status = PCG_BREAKDOWN;
                S.nits += 1;
                S.run = 0;
            }
            S.alpha = S.rz / s[0];
        });
        if (!ok || !S.run) break;
        const double alpha = S.alpha;
        v[0] = v[1] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) {
            const double ri = sr[i] - alpha * sw[i], zi = ri / sD[i];
            sr[i] = ri;
            sw[i] = zi;
            if (FUSED && L.row(i) < n) R.z[L.row(i)] = zi;
            v[0] += ri * ri;
            v[1] += ri * zi;
        }
        ok = G.sum(v,
                   [&](const double *s) {
                       const int k = S.nits + 1;
                       const double res = sqrt(s[0]);
                       S.nits = k;
                       S.residual = res;
                       if (first && R.hist != nullptr) R.hist[k] = res;
                       if (!isfinite(res)) {
                           S.status = PCG_NONFINITE;
                           S.run = 0;
                       } else if (!(res > S.tol) || k >= R.maxit) {
                           S.run = 0;
                       } else if (S.rz == 0.0) {   // the next step's beta would divide by it
                           S.status = PCG_BREAKDOWN;
                           S.nits = k + 1;
                           S.run = 0;
                       } else {
                           S.beta = s[1] / S.rz;
                       }
                       S.rz = s[1];
                   },
                   [&](int i0, int nt) {   // warp 0 is waiting for the sum
                       for (int i = i0; i < m; i += nt)
                           if (L.row(i) < n) R.x[L.row(i)] += alpha * sp[i];
                   });
    }
    if (t == 0 && (first || !ok)) {
        R.st->nits = S.nits;
        R.st->residual = S.residual;
        R.st->status = ok ? S.status : kStatusPassLimit;
    }
}

constexpr int kSpare = 72;   // coop_max_row
// Shared memory takes 601,472 rows on 148 SMs (127 slices of 1,092 bytes a block).
constexpr int64_t kRowBytes = 4 * sizeof(double);   // r, w / z, p, diagonal
// Entries up to which the product forms the direction from the two vectors it
// gathers, saving a barrier: us per iteration with / without, P1 9k rows 6.8 /
// 7.7, P1 36k (430,000 entries) 6.9 / 7.9, P2 9k 8.5 / 9.2, P1 133k (1.7 million)
// 10.3 / 10.6, P2 69k (1.6 million) 11.4 / 11.3, P3 51k (1.9 million) 16.1 / 15.2.
constexpr int64_t kFusedEntries = 1500000;

}  // namespace

int coop_exchange_doubles() { return kCoopDoubles; }

int stream_sms(cudaStream_t s) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    struct Driver {
        PFN_cuStreamGetGreenCtx_v12040 context = nullptr;
        PFN_cuGreenCtxGetDevResource_v12040 resource = nullptr;
        static void *entry(const char *name) {
            void *f = nullptr;
            cudaDriverEntryPointQueryResult found;
            if (cudaGetDriverEntryPointByVersion(name, &f, 12040, cudaEnableDefault, &found) != cudaSuccess) {
                cudaGetLastError();
                return nullptr;
            }
            return found == cudaDriverEntryPointSuccess ? f : nullptr;
        }
        Driver() {
            context = (PFN_cuStreamGetGreenCtx_v12040)entry("cuStreamGetGreenCtx");
            resource = (PFN_cuGreenCtxGetDevResource_v12040)entry("cuGreenCtxGetDevResource");
        }
    };
    static const Driver driver;
    CUgreenCtx green = nullptr;
    CUdevResource r{};
    if (driver.context != nullptr && driver.resource != nullptr &&
        driver.context((CUstream)s, &green) == CUDA_SUCCESS && green != nullptr &&
        driver.resource(green, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS && (int)r.sm.smCount < sms)
        sms = (int)r.sm.smCount;
    return sms;
}

int64_t pcg_coop_entries(int64_t n, int64_t nnz, int sms) {
    CoopSplit sp;
    return coop_split(n, nnz, kRowBytes, 0, 4, kSpare, sms, &sp) ? nnz : -1;
}

cudaError_t launch_pcg_coop(const PcgRun &R, cudaStream_t s) {
    CoopSplit sp;
    if (!coop_split(R.A.n, R.nnz, kRowBytes, 0, 4, kSpare, R.sms, &sp)) return cudaErrorCooperativeLaunchTooLarge;
    if (R.nnz <= kFusedEntries) {
        switch (sp.lanes) {
        case 1: return coop_launch(pcg_coop_kernel<1, true>, R, sp, s);
        case 2: return coop_launch(pcg_coop_kernel<2, true>, R, sp, s);
        default: return coop_launch(pcg_coop_kernel<4, true>, R, sp, s);
        }
    }
    switch (sp.lanes) {
    case 1: return coop_launch(pcg_coop_kernel<1, false>, R, sp, s);
    case 2: return coop_launch(pcg_coop_kernel<2, false>, R, sp, s);
    default: return coop_launch(pcg_coop_kernel<4, false>, R, sp, s);
    }
}

}  // namespace phgb
