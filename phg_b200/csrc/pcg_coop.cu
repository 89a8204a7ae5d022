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
// What bounds it: at 1,000 to 40,000 rows the three barriers, about 1.4 us each,
// and the latency of the phases between them; from 100,000 rows on the product,
// which reads the matrix from L2 (up to some 10 million entries) at the rate
// its gathers allow.  Time per iteration against the same recurrence as three
// launches in a graph loop: P1 1,331 rows 7.3 us (16.3), P1 36k 8.4 (18.9), P1
// 133k 10.8 (20.7), P1 389k 20.6 (33.3), P2 69k 11.9 (23.4), P2 250k 25.0
// (37.4), P2 531k 47.5 (58.5), P3 227k 32.2 (52.2); and a solve needs no tuned
// layout, no graph and one host wait: 71 us instead of 180 before the first
// iteration.  (Measured and left: the rows in one contiguous run per block, as
// CSR rows of 4 to 16 lanes, as a stream over the entries, or sorted by length:
// 25 to 29 us on P1 389k and over 100 on P2 531k, whose vertex rows then sit on
// a third of the blocks.)
#include "coop_rows.cuh"
#include "grid_sync.cuh"
#include "pcg_coop.h"

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

__global__ void __launch_bounds__(kCoopThreads, 1)
pcg_coop_kernel(const PcgRun R, int parts) {
    extern __shared__ double s_vec[];
    __shared__ CoopShared sh;
    __shared__ PcgScalars S;
    __shared__ int next_unit;
    CoopGrid G(R.exchange, &sh);
    const int t = threadIdx.x;
    const unsigned n = (unsigned)R.A.n;
    const int m = 32 * (int)((((int64_t)n + 31) / 32 - blockIdx.x + gridDim.x - 1) / gridDim.x);
    double *sr = s_vec, *sw = sr + m, *sp = sw + m, *sD = sp + m;   // of the block's places
    CoopRows L(n, parts, sD + m, &next_unit, R.cols, R.vals);
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
            if (R.A.rp[row + 1] - R.A.rp[row] > kCoopMaxRowLen) v3[2] = 1.0;
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
    L.build(R.A);
    __syncthreads();
    // r = b - A x, or b when x = 0
    if (S.nonzero) {
        L.product(R.x, sw);
        for (int i = t; i < m; i += kCoopThreads) sr[i] -= sw[i];
    }
    v[0] = v[1] = 0.0;
    for (int i = t; i < m; i += kCoopThreads) {
        const double ri = sr[i], zi = ri / sD[i];
        sw[i] = zi;
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
    bool start = true;
    while (ok && S.run) {
        const double beta = S.beta;
        for (int i = t; i < m; i += kCoopThreads) {
            const double pi = start ? sw[i] : beta * sp[i] + sw[i];
            sp[i] = pi;
            if (L.row(i) < n) R.p[L.row(i)] = pi;
        }
        start = false;
        if (!(ok = G.sync())) break;
        d[0] = 0.0;
        L.product(R.p, sw);
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

struct CoopDevice {
    int blocks = 0;          // SMs of a device that can launch cooperatively, else 0
    int64_t smem = 0;        // dynamic shared memory a block may use
};

CoopDevice coop_device() {
    CoopDevice d;
    int dev = 0, coop = 0, sms = 0, smem = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return d;
    }
    d.blocks = coop ? (sms < kCoopMaxBlocks ? sms : kCoopMaxBlocks) : 0;
    d.smem = smem - 4096;   // the kernel's static shared memory
    return d;
}

// Shared memory of a block with that many slices: r, w / z, p and the diagonal
// of each row, and the row bookkeeping.
constexpr int64_t coop_smem(int64_t slices, int parts) {
    return slices * 32 * 4 * (int64_t)sizeof(double) + coop_rows_bytes(slices, parts);
}

// Shared memory a solve takes at most.  What it takes the L1 cache loses, and
// the product's gathers need that: with 122 KB a block (P2, 531k rows) an
// iteration takes 47.5 us against 58.5 as separate launches, with 208 KB 71.
constexpr int64_t kCoopMaxSmem = 136 * 1024;
// A block per this many entries (a row's vector work counted as four) while
// there are SMs: below that the barriers of more blocks cost what they save.
constexpr int64_t kCoopBlockWork = 4096;

// Blocks of a solve; false when it is too large.
bool coop_split(const CoopDevice &dv, int64_t n, int64_t nnz, int *blocks, int *parts, int64_t *smem) {
    if (dv.blocks < 1) return false;
    const int64_t slices = ceil_div(n, 32);
    int64_t G = ceil_div(nnz + 4 * n, kCoopBlockWork);
    if (G > slices) G = slices;
    if (G > dv.blocks) G = dv.blocks;
    const int64_t per = ceil_div(slices, G);
    *blocks = (int)G;
    *parts = coop_parts(per, n, nnz);
    *smem = coop_smem(per, *parts);
    return *smem <= dv.smem && *smem <= kCoopMaxSmem;
}

cudaError_t launch(const PcgRun &R, int blocks, int parts, int64_t smem, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(pcg_coop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    PcgRun run = R;
    void *args[] = {(void *)&run, (void *)&parts};
    return cudaLaunchCooperativeKernel((const void *)pcg_coop_kernel, dim3(blocks), dim3(kCoopThreads), args,
                                       (size_t)smem, s);
}

}  // namespace

int coop_exchange_doubles() { return kCoopDoubles; }

int64_t pcg_coop_entries(int64_t n, int64_t nnz) {
    int b, p;
    int64_t m;
    return coop_split(coop_device(), n, nnz, &b, &p, &m) ? nnz : -1;
}

cudaError_t launch_pcg_coop(const PcgRun &R, cudaStream_t s) {
    int blocks, parts;
    int64_t smem;
    if (!coop_split(coop_device(), R.A.n, R.nnz, &blocks, &parts, &smem)) return cudaErrorCooperativeLaunchTooLarge;
    return launch(R, blocks, parts, smem, s);
}

}  // namespace phgb
