// Mixed-precision Jacobi-PCG as one cooperative kernel: the recurrence, the
// reliable updates and the stopping rule of mixed.cu, for systems whose FP32
// vectors fit the SMs' shared memory (rows and barriers as in pcg_coop.cu).
//
// Only u = D^-1 r, which the products of the other blocks gather, and the FP64
// x go through L2.  An iteration is two phases between grid barriers, both of
// which carry a sum:
//   product  w = A u, delta = w.u -> alpha, beta
//   update   p, s = A p, the correction y, r, u; gamma = r.u and r.r
// A reliable update (x += y, then r and u from the explicit FP64 residual) adds
// two.  Each row's products are summed in CSR order, one by one, in FP32 and
// FP64, as the launched SELL and pair products do: the recurrence's last
// iterations depend on every rounding, so the same roundings give the same
// iterates and iteration counts as there.
// What bounds it: the two barriers (some 1.4 us each) and the phases' latency up
// to 40,000 rows, then the product's reads of the matrix from L2 at the rate its
// gathers allow.  Time per iteration against the same recurrence as two launches
// in a graph loop: P1 36k rows 7.2 us (21.4), P1 389k 16.1 (30.5), P2 69k 11.1
// (29.0), P2 250k 18.7 (40.8), P3 227k 25.6 (66.5).
#include "coop_rows.cuh"
#include "grid_sync.cuh"
#include "mixed_coop.h"

#include <float.h>
#include <math.h>

namespace phgb {

namespace {

struct MixedScalars {
    double gamma, gamma_prev, alpha_prev, rb, tol, maxr, residual;
    float alpha, beta;
    int nits, nupdates, status, run, first, nonzero, declined, due;
};

__device__ __forceinline__ bool is_zero(double a) { return fabs(a) < 10.0 * DBL_MIN; }   // utils.h:451

template <int H>
__global__ void __launch_bounds__(kCoopThreads, 1)
mixed_coop_kernel(const MixedRun R) {
    extern __shared__ double s_mem[];
    __shared__ CoopShared sh;
    __shared__ MixedScalars S;
    __shared__ int next_unit;
    CoopGrid<> G(R.exchange, &sh);
    const int t = threadIdx.x;
    const unsigned n = (unsigned)R.A.n;
    const int m = coop_places(n);
    CoopRows<H> L(n, s_mem, &next_unit, R.cols);
    float *sr = (float *)((char *)s_mem + coop_rows_bytes(L.slices, H));   // of the block's places
    float *su = sr + m, *sw = su + m, *sp = sw + m, *ss = sp + m, *sy = ss + m, *sD = sy + m;
    const bool first = blockIdx.x == 0;

    // ||b|| and |x|_1 (solver-phg.c:498-518)
    double v3[3] = {0.0, 0.0, 0.0}, v2[2], d[1];
    for (int i = t; i < m; i += kCoopThreads) {
        const unsigned row = L.row(i);
        if (row < n) {
            const double bi = R.b[row];
            v3[0] += fabs(R.x[row]);
            v3[1] += bi * bi;
            if (R.A.rp[row + 1] - R.A.rp[row] > R.max_row) v3[2] = 1.0;
        }
    }
    bool ok = G.sum(v3, [&](const double *s) {
        S.rb = sqrt(s[1]);
        S.nonzero = !is_zero(s[0] / (double)n);
        S.declined = s[2] != 0.0;
        S.nits = S.nupdates = 0;
        S.status = PCG_RUNNING;
        S.residual = 0.0;
        S.run = !is_zero(S.rb) && !S.declined;
        if (S.declined) S.status = kStatusDeclined;
    });
    if (ok && !S.run) {
        if (!S.declined)
            for (int i = t; i < m; i += kCoopThreads)
                if (L.row(i) < n) R.x[L.row(i)] = 0.0;
        if (first && t == 0) *R.out = MixedResult{0.0, 0, 0, S.status};
        return;
    }
    if (ok) {
        L.build(R.A, [&](int q, double value) {
            R.vals32[q] = (float)value;
            R.vals64[q] = value;
        });
        __syncthreads();
    }
    // the FP64 residual of a row, and the FP32 recurrence started from it
    auto restart_row = [&](int i, double rt) {
        const float rf = (float)rt, uf = rf / sD[i];
        sr[i] = rf;
        su[i] = uf;
        if (L.row(i) < n) R.u[L.row(i)] = uf;
        v3[0] += rt * rt;
        v3[1] += (double)rf * (double)uf;
        v3[2] += (double)rf * (double)rf;
    };
    // b - A x
    auto residual_from_x = [&] {
        L.product_each(R.vals64, (const double *)R.x, [&](int i, double acc) {
            restart_row(i, L.row(i) < n ? R.b[L.row(i)] - acc : 0.0);
        });
    };
    v3[0] = v3[1] = v3[2] = 0.0;
    if (ok) {
        for (int i = t; i < m; i += kCoopThreads) {
            const unsigned row = L.row(i);
            sD[i] = row < n ? (float)R.D[row] : 1.0f;
            sp[i] = 0.0f;
            ss[i] = 0.0f;
        }
        __syncthreads();
        if (S.nonzero) {
            residual_from_x();
        } else {
            for (int i = t; i < m; i += kCoopThreads) restart_row(i, L.row(i) < n ? R.b[L.row(i)] : 0.0);
        }
        ok = G.sum(v3, [&](const double *s) {
            const double res = sqrt(s[0]);
            double tol = res * R.rtol;   // get_tol (solver-phg.c:104-115)
            if (tol < S.rb * R.btol) tol = S.rb * R.btol;
            if (tol < R.atol) tol = R.atol;
            S.tol = tol;
            S.residual = res;
            S.maxr = res;
            S.gamma = s[1];
            S.first = 1;
            if (!isfinite(s[1])) S.status = kStatusBadStart;
            S.run = S.status == PCG_RUNNING && res > tol && R.maxit > 0;
        });
    }
    bool fresh = true;   // y holds nothing: the last reliable update folded it into x
    while (ok && S.run) {
        // w = A u and the step from gamma = r.u and delta = w.u
        L.template product<true>(R.vals32, (const float *)R.u, sw);
        d[0] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) d[0] += (double)sw[i] * (double)su[i];
        ok = G.sum(d, [&](const double *s) {
            const double gamma = S.gamma, delta = s[0];
            double alpha = 0.0, beta = 0.0, den = delta;
            if (!(isfinite(gamma) && isfinite(delta))) {
                S.status = PCG_NONFINITE;
            } else if (!S.first) {
                if (S.gamma_prev == 0.0) {
                    den = 0.0;
                } else {
                    beta = gamma / S.gamma_prev;
                    den = delta - beta * gamma / S.alpha_prev;
                }
            }
            if (S.status == PCG_RUNNING) {
                S.nits += 1;   // the reference counts the step it breaks down in (solver-phg.c:537)
                if (den == 0.0) S.status = PCG_BREAKDOWN;
                else alpha = gamma / den;
            }
            S.run = S.status == PCG_RUNNING;
            S.alpha = (float)alpha;
            S.beta = (float)beta;
            S.gamma_prev = gamma;
            S.alpha_prev = alpha;
            S.first = 0;
        });
        if (!ok || !S.run) break;
        const float a = S.alpha, b = S.beta;
        v2[0] = v2[1] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) {
            const float p = su[i] + b * sp[i], s = sw[i] + b * ss[i];
            sp[i] = p;
            ss[i] = s;
            sy[i] = (fresh ? 0.0f : sy[i]) + a * p;
            const float r = sr[i] - a * s, u = r / sD[i];
            sr[i] = r;
            su[i] = u;
            if (L.row(i) < n) R.u[L.row(i)] = u;
            v2[0] += (double)r * (double)u;
            v2[1] += (double)r * (double)r;
        }
        fresh = false;
        ok = G.sum(v2, [&](const double *s) {
            const double res = sqrt(s[1]);
            S.gamma = s[0];
            S.residual = res;
            S.due = 0;
            if (!isfinite(res)) {
                S.status = PCG_NONFINITE;
                S.run = 0;
            } else {
                S.due = !(res > S.tol) || S.nits >= R.maxit || res < R.delta * S.maxr;
            }
        });
        if (!ok || !S.run || !S.due) continue;
        // reliable update
        for (int i = t; i < m; i += kCoopThreads)
            if (L.row(i) < n) R.x[L.row(i)] += (double)sy[i];
        fresh = true;
        if (!(ok = G.sync())) break;
        v3[0] = v3[1] = v3[2] = 0.0;
        residual_from_x();
        ok = G.sum(v3, [&](const double *s) {
            const double res = sqrt(s[0]);
            S.residual = res;
            S.maxr = res;
            S.gamma = s[1];
            S.nupdates += 1;
            if (!isfinite(res)) {
                S.status = PCG_NONFINITE;
                S.run = 0;
            } else if (!(res > S.tol) || S.nits >= R.maxit) {
                S.run = 0;
            }
        });
    }
    // a breakdown ends between reliable updates: fold y, report the FP64 residual
    if (ok && !fresh && S.status == PCG_BREAKDOWN) {
        for (int i = t; i < m; i += kCoopThreads)
            if (L.row(i) < n) R.x[L.row(i)] += (double)sy[i];
        ok = G.sync();
        if (ok) {
            v3[0] = v3[1] = v3[2] = 0.0;
            residual_from_x();
            ok = G.sum(v3, [&](const double *s) { S.residual = sqrt(s[0]); });
        }
    }
    if (t == 0 && (first || !ok))
        *R.out = MixedResult{S.residual, S.nits, S.nupdates, ok ? S.status : kStatusPassLimit};
}

constexpr int64_t kRowBytes = 7 * sizeof(float);   // r, u, w, p, s, y, diagonal
// Entries up to which the FP32 copy (8 bytes each) stays in L2 beside the
// vectors; beyond, the products on the 16-bit-column layout move a quarter fewer
// bytes from memory.  A careful line, the kernel is faster beyond it too where
// its vectors fit: us per iteration in one kernel / on the layouts, P2 9.9 million
// entries 26.4 / 47.4, and with the limit raised P1 10.4 million 26.6 / 30.9, P2
// 13.7 million 33.3 / 41.6, P3 10.9 million 29.5 / 67.3, 16.5 million 39.9 / 79.3.
constexpr int64_t kMaxEntries = 10000000;

}  // namespace

int64_t mixed_coop_entries(int64_t n, int64_t nnz, int sms) {
    CoopSplit sp;
    return nnz <= kMaxEntries && coop_split(n, nnz, kRowBytes, 0, 2, 0, sms, &sp) ? nnz : -1;
}

cudaError_t launch_mixed_coop(const MixedRun &R, cudaStream_t s) {
    CoopSplit sp;
    if (!coop_split(R.A.n, R.nnz, kRowBytes, 0, 2, 0, R.sms, &sp)) return cudaErrorCooperativeLaunchTooLarge;
    return sp.lanes == 1 ? coop_launch(mixed_coop_kernel<1>, R, sp, s) : coop_launch(mixed_coop_kernel<2>, R, sp, s);
}

}  // namespace phgb
