// GMRES_r and FLGMRES_r (solver-phg.c:1050-1260, 2063-2340) with the Jacobi
// preconditioner as one cooperative kernel: the cycles, rotations and stopping
// rule of gmres.cu, rows and barriers as in pcg_coop.cu.  A step i is
//   pc       v_i = w / h_(i-1,i) (z / ||z|| first), V_0 or F_i = v_i / diag
//   product  w = A V_0, h_(i,1) = w.v_1                        (sum)
//   mgs k    w -= h_(i,k-1) v_(k-1), h_(i,k) = w.v_k, k = 2..i  (sum each)
//   norm     w -= h_(i,i) v_i, ||w||, rotations                (sum)
// so its modified Gram-Schmidt steps cost a barrier each instead of a launch.
// w, z and the diagonal of a block's rows stay in shared memory, the basis in
// L2: a block reads only its own rows of it.  Every block keeps the small
// dense arrays and does the rotations and the back substitution itself, in one
// thread with the reference's operation order.
#include "coop_rows.cuh"
#include "grid_sync.cuh"
#include "krylov_coop.h"

#include <float.h>
#include <math.h>

namespace phgb {

namespace {

struct GmresScalars {
    double r_norm, tol, residual, b_norm;
    int nits, restart, ninner, run, cycle_done, finished, status, itr_out, zi, ak, declined, first;
};

__device__ __forceinline__ bool is_zero(double a) { return fabs(a) < 10.0 * DBL_MIN; }   // utils.h:451

// Step i is complete (h_(i,i+1)^2 = `sum`): solver-phg.c:1147-1182.
__device__ __forceinline__ void arnoldi_end(GmresScalars &S, const GmresRun &R, int R2, double *H, double *c1, double *c2,
                                            double *s, int i, double sum) {
    double *h = H + i * R2;
    S.nits += 1;
    const double hn = sqrt(sum);
    h[i + 1] = hn;
    if (is_zero(hn)) {   // happy breakdown: step i is not used
        S.ninner = i - 1;
        S.cycle_done = 1;
        return;
    }
    for (int j = 1; j < i; j++) {
        const double a = h[j], b = h[j + 1];
        h[j] = rn_add(rn_mul(c1[j], a), rn_mul(c2[j], b));
        h[j + 1] = rn_add(rn_mul(-c2[j], a), rn_mul(c1[j], b));
    }
    const double hii = h[i], hi1 = h[i + 1];
    double tmp = sqrt(rn_add(rn_mul(hii, hii), rn_mul(hi1, hi1)));
    if (is_zero(tmp)) tmp = 1.e-16;
    c1[i] = __ddiv_rn(hii, tmp);
    c2[i] = __ddiv_rn(hi1, tmp);
    s[i + 1] = rn_mul(-c2[i], s[i]);
    s[i] = rn_mul(c1[i], s[i]);
    h[i] = rn_add(rn_mul(c1[i], hii), rn_mul(c2[i], hi1));
    const double rn = fabs(s[i + 1]);
    S.r_norm = rn;
    S.ninner = i;
    if (!isfinite(rn)) {
        S.status = GMRES_NONFINITE;
        S.cycle_done = 1;
        return;
    }
    if (rn <= S.tol || i >= S.restart || S.nits >= R.maxit) S.cycle_done = 1;
}

// H y = s by back substitution (solver-phg.c:1201-1207), and whether the solve
// ends after this cycle's update.
__device__ __forceinline__ void cycle_end(GmresScalars &S, const GmresRun &R, int R2, const double *H, double *s, double *y) {
    for (int j = S.ninner; j > 0; j--) {
        y[j] = __ddiv_rn(s[j], H[j * R2 + j]);
        for (int k = j - 1; k > 0; k--) s[k] = rn_sub(s[k], rn_mul(H[j * R2 + k], y[j]));
    }
    if (R.augk >= 0) {
        S.zi = S.itr_out % R.augk;
        S.ak = S.itr_out < R.augk ? S.itr_out : R.augk;
        S.itr_out += 1;
    }
    if (S.status != GMRES_OK) {
        S.finished = 1;
    } else if (S.r_norm <= S.tol) {
        S.residual = S.r_norm;
        S.finished = 1;
    } else if (S.nits >= R.maxit) {
        S.finished = 1;
    }
}

constexpr int64_t dense_doubles(int most) { return (int64_t)(most + 2) * (most + 2) + 4 * (most + 2); }

template <int H>
__global__ void __launch_bounds__(kCoopThreads, 1)
gmres_coop_kernel(const GmresRun R) {
    extern __shared__ double s_mem[];
    __shared__ CoopShared sh;
    __shared__ GmresScalars S;
    __shared__ int next_unit;
    CoopGrid<> G(R.exchange, &sh);
    const int t = threadIdx.x;
    const unsigned n = (unsigned)R.A.n;
    const int m = coop_places(n);
    const bool flex = R.augk >= 0;
    const int most = R.mk + (flex ? R.augk : 0), R2 = most + 2;   // the most steps a cycle takes
    double *sH = s_mem, *c1 = sH + R2 * R2, *c2 = c1 + R2, *ss = c2 + R2, *sy = ss + R2;
    double *sw = sy + R2, *sz = sw + m, *sD = sz + m;   // of the block's places
    CoopRows<H> L(n, sD + m, &next_unit, R.cols);
    const bool first = blockIdx.x == 0;
    auto Vi = [&](int i) { return R.V + (int64_t)i * R.stride; };

    double d[1], v2[2] = {0.0, 0.0};
    for (int i = t; i < m; i += kCoopThreads) {
        const unsigned row = L.row(i);
        sD[i] = row < n ? R.D[row] : 1.0;
        if (row < n) {
            v2[0] += R.b[row] * R.b[row];
            if (R.A.rp[row + 1] - R.A.rp[row] > R.max_row) v2[1] = 1.0;
        }
    }
    for (int i = t; i < R2 * R2 + 4 * R2; i += kCoopThreads) sH[i] = 0.0;
    bool ok = G.sum(v2, [&](const double *s) {
        S.b_norm = sqrt(s[0]);
        S.declined = s[1] != 0.0;
        S.status = S.declined ? kStatusDeclined : GMRES_OK;
        S.nits = S.itr_out = S.finished = 0;
        S.residual = 0.0;
        S.first = 1;
        S.restart = R.mk;
        S.run = !(S.declined || is_zero(S.b_norm));
    });
    if (ok && !S.run) {   // solver-phg.c:1071-1075
        if (!S.declined)
            for (int i = t; i < m; i += kCoopThreads)
                if (L.row(i) < n) R.x[L.row(i)] = 0.0;
        if (first && t == 0) {
            R.st->nits = 0;
            R.st->residual = 0.0;
            R.st->status = S.status;
        }
        return;
    }
    if (ok) {
        L.build(R.A, [&](int q, double value) { R.vals[q] = value; });
        __syncthreads();
    }
    while (ok) {
        // z = b - A x (solver-phg.c:1104-1106, 1244-1245) and ||z||
        L.template product<false>(R.vals, (const double *)R.x, sz);
        d[0] = 0.0;
        for (int i = t; i < m; i += kCoopThreads) {
            const double z = L.row(i) < n ? rn_sub(R.b[L.row(i)], sz[i]) : 0.0;
            sz[i] = z;
            d[0] += z * z;
        }
        ok = G.sum(d, [&](const double *s) {
            const double rn = sqrt(s[0]);
            S.r_norm = rn;
            ss[1] = rn;
            ss[0] = 1.0;
            if (S.first) {   // get_tol (solver-phg.c:104-115) with ||r0||
                double tol = rn * R.rtol;
                if (tol < S.b_norm * R.btol) tol = S.b_norm * R.btol;
                if (tol < R.atol) tol = R.atol;
                S.tol = tol;
                S.residual = rn;
                S.first = 0;
            }
            S.ninner = 0;
            if (flex)   // cycle k takes mk + min(k, augk) steps (solver-phg.c:2160-2164)
                S.restart = R.mk + (S.itr_out <= R.augk ? S.itr_out : R.augk);
            S.run = 1;
            if (!isfinite(rn)) {
                S.status = GMRES_NONFINITE;
                S.run = 0;
            } else if (S.nits >= R.maxit) {   // while (nits < max_its) ends
                S.run = 0;
            }
            S.cycle_done = !(rn > S.tol);
        });
        if (!ok || !S.run) break;
        for (int i = 1; ok && !S.cycle_done; i++) {   // the rotations end the cycle at step S.restart
            double *vi = Vi(i), *in = flex ? R.F + (int64_t)i * R.stride : R.V;
            {
                const double scale = __ddiv_rn(1.0, i == 1 ? S.r_norm : sH[(i - 1) * R2 + i]);
                const double *src = i == 1 ? sz : sw;
                const double *za = i > R.mk ? R.Z + (int64_t)(i - R.mk - 1) * R.stride : nullptr;
                for (int k = t; k < m; k += kCoopThreads) {
                    const unsigned row = L.row(k);
                    if (row < n) {
                        const double v = rn_mul(scale, src[k]);
                        vi[row] = v;
                        in[row] = __ddiv_rn(za != nullptr ? za[row] : v, sD[k]);
                    }
                }
            }
            if (!(ok = G.sync())) break;
            L.template product<false>(R.vals, (const double *)in, sw);
            for (int k = 1; ok && k <= i + 1; k++) {
                const double mh = k > 1 ? -sH[i * R2 + k - 1] : 0.0;
                const double *vprev = Vi(k - 1), *vk = Vi(k);
                const bool last = k == i + 1;
                d[0] = 0.0;
                for (int q = t; q < m; q += kCoopThreads) {
                    const unsigned row = L.row(q);
                    if (row < n) {
                        double w = sw[q];
                        if (k > 1) {
                            w = rn_add(w, rn_mul(mh, vprev[row]));
                            sw[q] = w;
                        }
                        d[0] += w * (last ? w : vk[row]);
                    }
                }
                ok = G.sum(d, [&](const double *s) {
                    if (last) arnoldi_end(S, R, R2, sH, c1, c2, ss, i, s[0]);
                    else sH[i * R2 + k] = s[0];
                });
            }
        }
        if (!ok) break;
        if (t == 0) cycle_end(S, R, R2, sH, ss, sy);
        __syncthreads();
        // x += (V y) / diag or sum_j y_j F_j, or z when the cycle made no step
        // (solver-phg.c:1209-1225, 2250-2290); FLGMRES_r keeps the correction
        const int i = S.ninner;
        for (int q = t; q < m; q += kCoopThreads) {
            const unsigned row = L.row(q);
            if (row >= n) continue;
            double c = sz[q];
            if (!flex) {
                if (i > 0) {
                    c = rn_mul(sy[1], Vi(1)[row]);
                    for (int j = 2; j <= i; j++) c = rn_add(c, rn_mul(sy[j], Vi(j)[row]));
                }
                R.x[row] = rn_add(R.x[row], __ddiv_rn(c, sD[q]));
            } else {
                double w = c;
                if (i > 0) {
                    const double *F = R.F + row;
                    c = rn_mul(sy[1], F[R.stride]);
                    for (int j = 2; j <= i; j++) c = rn_add(c, rn_mul(sy[j], F[(int64_t)j * R.stride]));
                    const int top = i <= R.mk ? i : R.mk;
                    w = rn_mul(sy[1], Vi(1)[row]);
                    for (int j = 2; j <= top; j++) w = rn_add(w, rn_mul(sy[j], Vi(j)[row]));
                    if (i > R.mk)
                        for (int j = 1; j <= S.ak; j++)
                            w = rn_add(w, rn_mul(sy[j + R.mk], R.Z[(int64_t)(j - 1) * R.stride + row]));
                }
                R.x[row] = rn_add(c, R.x[row]);
                R.Z[(int64_t)S.zi * R.stride + row] = w;
            }
        }
        if (S.finished) break;
        ok = G.sync();
    }
    if (t == 0 && (first || !ok)) {
        R.st->nits = S.nits;
        R.st->residual = S.residual;
        R.st->status = ok ? S.status : kStatusPassLimit;
    }
}

constexpr int kSpare = 176;   // coop_max_row
constexpr int64_t kRowBytes = 3 * sizeof(double);   // w, z, diagonal

}  // namespace

int64_t gmres_coop_entries(int64_t n, int64_t nnz, int restart, int sms) {
    CoopSplit sp;
    return coop_split(n, nnz, kRowBytes, 8 * dense_doubles(restart), 4, kSpare, sms, &sp) ? nnz : -1;
}

cudaError_t launch_gmres_coop(const GmresRun &R, cudaStream_t s) {
    CoopSplit sp;
    if (!coop_split(R.A.n, R.nnz, kRowBytes, 8 * dense_doubles(R.mk + (R.augk >= 0 ? R.augk : 0)), 4, kSpare, R.sms, &sp))
        return cudaErrorCooperativeLaunchTooLarge;
    switch (sp.lanes) {
    case 1: return coop_launch(gmres_coop_kernel<1>, R, sp, s);
    case 2: return coop_launch(gmres_coop_kernel<2>, R, sp, s);
    default: return coop_launch(gmres_coop_kernel<4>, R, sp, s);
    }
}

}  // namespace phgb
