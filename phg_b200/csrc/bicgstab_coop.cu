// Jacobi-BiCGstab (solver_BiCGstab, solver-phg.c:606-781) as one cooperative
// kernel: the recurrence and stopping rule of bicgstab.cu, rows and barriers as
// in pcg_coop.cu.  Only p^ and s^, which the products gather, and x go through
// L2.  An iteration is five phases between grid barriers:
//   dir      p = r + beta (p - omega v), p^ = p / diag
//   product  v = A p^, rh.v -> alpha                            (sum)
//   s        s = r - alpha v (in r's place), s^ = s / diag, ||s||  (sum)
//   product  t = A s^, t.s and t.t -> omega                     (sum)
//   update   r = s - omega t, ||r|| and r.rh                    (sum; x += alpha
//            p^ + omega s^ runs behind the barrier)
#include "coop_rows.cuh"
#include "grid_sync.cuh"
#include "krylov_coop.h"

#include <float.h>
#include <math.h>

namespace phgb {

namespace {

struct BicgScalars {
    double rho0, rho1, alpha, beta, omega, rb, tol, residual;
    int nits, status, run, nonzero, declined;
};

__device__ __forceinline__ bool is_zero(double a) { return fabs(a) < 10.0 * DBL_MIN; }   // utils.h:451

template <int H>
__global__ void __launch_bounds__(kCoopThreads, 1)
bicg_coop_kernel(const BicgRun R) {
    extern __shared__ double s_mem[];
    __shared__ CoopShared sh;
    __shared__ BicgScalars S;
    __shared__ int next_unit;
    CoopGrid<> G(R.exchange, &sh);
    const int t = threadIdx.x;
    const unsigned n = (unsigned)R.A.n;
    const int m = coop_places(n);
    double *sr = s_mem, *srh = sr + m, *sp = srh + m, *sv = sp + m, *st = sv + m, *sD = st + m;   // of the block's places
    CoopRows<H> L(n, sD + m, &next_unit, R.cols);
    const bool first = blockIdx.x == 0;

    // ||b|| and |x|_1
    double v3[3] = {0.0, 0.0, 0.0}, v[2], d[1];
    for (int i = t; i < m; i += kCoopThreads) {
        const unsigned row = L.row(i);
        const bool in = row < n;
        const double bi = in ? R.b[row] : 0.0;
        sr[i] = bi;
        sp[i] = 0.0;
        sv[i] = 0.0;
        sD[i] = in ? R.D[row] : 1.0;
        if (in) {
            v3[0] += fabs(R.x[row]);
            v3[1] += bi * bi;
            if (R.A.rp[row + 1] - R.A.rp[row] > R.max_row) v3[2] = 1.0;
        }
    }
    bool ok = G.sum(v3, [&](const double *s) {
        S.rb = sqrt(s[1]);
        S.nonzero = !is_zero(s[0] / (double)n);
        S.declined = s[2] != 0.0;
        S.nits = 0;
        S.status = S.declined ? BICG_DECLINED : BICG_OK;
        S.residual = 0.0;
        S.run = !is_zero(S.rb) && !S.declined;
    });
    if (ok && !S.run) {   // solver-phg.c:630-633
        if (!S.declined)
            for (int i = t; i < m; i += kCoopThreads)
                if (L.row(i) < n) R.x[L.row(i)] = 0.0;
        if (first && t == 0) {
            if (R.hist != nullptr && !S.declined) R.hist[0] = 0.0;
            R.st->nits = 0;
            R.st->residual = 0.0;
            R.st->status = S.status;
        }
        return;
    }
    if (ok) {
        L.build(R.A, [&](int q, double value) { R.vals[q] = value; });
        __syncthreads();
        // r = b - A x, or b when x = 0 (solver-phg.c:645-653)
        if (S.nonzero) L.template product<false>(R.vals, (const double *)R.x, st);
        d[0] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) {
            const double ri = S.nonzero ? sr[i] - st[i] : sr[i];
            sr[i] = ri;
            srh[i] = ri;
            d[0] += ri * ri;
        }
        ok = G.sum(d, [&](const double *s) {
            const double r0 = sqrt(s[0]);
            double tol = r0 * R.rtol;   // get_tol (solver-phg.c:104-115)
            if (tol < S.rb * R.btol) tol = S.rb * R.btol;
            if (tol < R.atol) tol = R.atol;
            S.tol = tol;
            S.residual = r0;
            S.rho1 = s[0];   // r.rh with rh = r
            S.rho0 = S.alpha = S.omega = 0.0;
            S.beta = 0.0;
            if (first && R.hist != nullptr) R.hist[0] = r0;
            S.run = r0 > tol && R.maxit > 0;
            if (S.run && s[0] == 0.0) {   // solver-phg.c:676-680: counted, then the loop ends
                S.status = BICG_RHO_ZERO;
                S.nits = 1;
                S.run = 0;
            }
        });
    }
    bool start = true;
    while (ok && S.run) {
        {
            const double beta = S.beta, mo = -S.omega;
            for (int i = t; i < m; i += kCoopThreads) {
                const double p = start ? sr[i] : sr[i] + beta * (sp[i] + mo * sv[i]);
                sp[i] = p;
                if (L.row(i) < n) R.ph[L.row(i)] = p / sD[i];
            }
        }
        start = false;
        if (!(ok = G.sync())) break;
        L.template product<false>(R.vals, (const double *)R.ph, sv);
        d[0] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) d[0] += srh[i] * sv[i];
        ok = G.sum(d, [&](const double *s) {
            if (s[0] == 0.0 || !isfinite(s[0])) {
                S.status = s[0] == 0.0 ? BICG_BREAKDOWN : BICG_NONFINITE;
                S.nits += 1;
                S.run = 0;
            } else {
                S.alpha = S.rho1 / s[0];
                S.rho0 = S.rho1;
            }
        });
        if (!ok || !S.run) break;
        const double alpha = S.alpha, ma = -alpha;
        d[0] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) {
            const double s = sr[i] + ma * sv[i];
            sr[i] = s;
            if (L.row(i) < n) R.sh[L.row(i)] = s / sD[i];
            d[0] += s * s;
        }
        ok = G.sum(d, [&](const double *s) {
            if (sqrt(s[0]) <= 1e-60) {   // solver-phg.c:717-729
                S.status = BICG_SMALL_S;
                S.nits += 1;
                S.run = 0;
            }
        });
        if (!ok || !S.run) break;
        L.template product<false>(R.vals, (const double *)R.sh, st);
        v[0] = v[1] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) {
            v[0] += sr[i] * st[i];
            v[1] += st[i] * st[i];
        }
        ok = G.sum(v, [&](const double *s) {
            if (s[1] == 0.0 || !isfinite(s[0]) || !isfinite(s[1])) {
                S.status = s[1] == 0.0 ? BICG_BREAKDOWN : BICG_NONFINITE;
                S.nits += 1;
                S.run = 0;
            } else {
                S.omega = s[0] / s[1];
            }
        });
        if (!ok || !S.run) break;
        const double omega = S.omega, mo = -omega;
        v[0] = v[1] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) {
            const double r = sr[i] + mo * st[i];
            sr[i] = r;
            v[0] += r * r;
            v[1] += r * srh[i];
        }
        ok = G.sum(v,
                   [&](const double *s) {
                       const int k = S.nits + 1;
                       const double res = sqrt(s[0]);
                       S.residual = res;
                       S.rho1 = s[1];
                       S.nits = k;
                       if (first && R.hist != nullptr) R.hist[k] = res;
                       if (!isfinite(res)) {
                           S.status = BICG_NONFINITE;
                           S.run = 0;
                       } else if (!(res > S.tol) || k >= R.maxit) {
                           S.run = 0;
                       } else if (s[1] == 0.0) {   // the next step's start finds rho = 0
                           S.status = BICG_RHO_ZERO;
                           S.nits = k + 1;
                           S.run = 0;
                       } else {
                           S.beta = (s[1] * S.alpha) / (S.rho0 * S.omega);
                       }
                   },
                   [&](int i0, int nt) {   // warp 0 is waiting for the sum
                       for (int i = i0; i < m; i += nt) {
                           const unsigned row = L.row(i);
                           if (row < n) R.x[row] = R.x[row] + (alpha * R.ph[row] + omega * R.sh[row]);
                       }
                   });
    }
    if (ok && S.status == BICG_SMALL_S) {   // x += alpha p^, then the residual of b - A x
        const double alpha = S.alpha;
        for (int i = t; i < m; i += kCoopThreads)
            if (L.row(i) < n) R.x[L.row(i)] += alpha * R.ph[L.row(i)];
        if ((ok = G.sync())) {
            L.template product<false>(R.vals, (const double *)R.x, st);
            d[0] = 0.0;
            for (int i = t; i < m; i += kCoopThreads) {
                const double r = L.row(i) < n ? R.b[L.row(i)] - st[i] : 0.0;
                d[0] += r * r;
            }
            ok = G.sum(d, [&](const double *s) {
                S.residual = sqrt(s[0]);
                if (first && R.hist != nullptr) R.hist[S.nits] = S.residual;
            });
        }
    }
    if (t == 0 && (first || !ok)) {
        R.st->nits = S.nits;
        R.st->residual = S.residual;
        R.st->status = ok ? S.status : BICG_PASS_LIMIT;
    }
}

constexpr int kSpare = 64;   // coop_max_row
// Shared memory takes 407,296 rows on 148 SMs (86 slices of 1,604 bytes a block).
constexpr int64_t kRowBytes = 6 * sizeof(double);   // r / s, rh, p, v, t, diagonal

}  // namespace

int64_t bicg_coop_entries(int64_t n, int64_t nnz, int sms) {
    CoopSplit sp;
    return coop_split(n, nnz, kRowBytes, 0, 4, kSpare, sms, &sp) ? nnz : -1;
}

cudaError_t launch_bicg_coop(const BicgRun &R, cudaStream_t s) {
    CoopSplit sp;
    if (!coop_split(R.A.n, R.nnz, kRowBytes, 0, 4, kSpare, R.sms, &sp)) return cudaErrorCooperativeLaunchTooLarge;
    switch (sp.lanes) {
    case 1: return coop_launch(bicg_coop_kernel<1>, R, sp, s);
    case 2: return coop_launch(bicg_coop_kernel<2>, R, sp, s);
    default: return coop_launch(bicg_coop_kernel<4>, R, sp, s);
    }
}

}  // namespace phgb
