// Block Jacobi-PCG: many right-hand sides solved together.
//
// Every column runs the reference's PCG recurrence (solver-phg.c:485-604)
// with its own scalars and stopping rule; the columns share one sparse
// matrix-matrix product per iteration, so the matrix is read once per tile
// of columns instead of once per right-hand side.  Vectors are stored row
// major, X[i * K + k] (K = padded number of columns), so the lanes of a row
// group read consecutive columns of a gathered row of P.  SpMM mapping: a
// tile of T columns, each lane 16 bytes of it (4 FP32 or 2 FP64 columns), so T /
// 4 or T / 2 lanes a matrix row, the other lanes further rows (T and the tile
// count are autotuned).  What bounds an iteration: the product's gathers from
// L2 (256 bytes an entry at 64 FP32 columns) and the passes over the block
// vectors.  P2 24^3, 64 columns, FP32: product 77 us (149 with one 4-byte gather
// a lane and column), whole iteration 197 us (405, of which some 120 were the
// last block's sums and a third the element-wise kernels' index arithmetic);
// FP64 274 us (436); 5 columns on P2 12^3 35 us (123).
//
// Precision: FP64 throughout, or FP32 matrix values / Krylov vectors / SpMM
// with FP64-accumulated dot products and FP64 reliable updates of the
// solution and residual (as in the single right-hand-side mixed solver),
// applied to all columns at once when any column asks for one.
#include "common.cuh"
#include "block.h"

namespace phgb {

constexpr int kBT = 256;          // threads per block
constexpr int kBMaxBlocks = 148 * 4;

// V consecutive columns of a row as one 16-byte access (K is a multiple of 8
// and the arrays are this library's own, so rows are 16-byte aligned).
template <typename VT> struct BVec;
template <> struct BVec<float> { using T = float4; static constexpr int V = 4; };
template <> struct BVec<double> { using T = double2; static constexpr int V = 2; };
template <typename VT> struct BArr { VT v[BVec<VT>::V]; };
template <typename VT> __device__ __forceinline__ BArr<VT> bload(const VT *p) {
    BArr<VT> a;
    *reinterpret_cast<typename BVec<VT>::T *>(a.v) = *reinterpret_cast<const typename BVec<VT>::T *>(p);
    return a;
}
template <typename VT> __device__ __forceinline__ BArr<VT> bload_ro(const VT *p) {
    BArr<VT> a;
    *reinterpret_cast<typename BVec<VT>::T *>(a.v) = __ldg(reinterpret_cast<const typename BVec<VT>::T *>(p));
    return a;
}
template <typename VT> __device__ __forceinline__ void bstore(VT *p, const BArr<VT> &a) {
    *reinterpret_cast<typename BVec<VT>::T *>(p) = *reinterpret_cast<const typename BVec<VT>::T *>(a.v);
}

// The block that arrives last at a ticket (all threads get the answer).
__device__ __forceinline__ bool last_block(unsigned *ticket, unsigned blocks) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1u) == blocks - 1;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Sums of the blocks' partials part[block][NV * cols], NV values a column, by
// the last block: the threads take the blocks in turn, a column's threads
// next to each other's, and their sums are added in order, so that the loads
// of all columns are in flight together (one thread per column summing 592
// blocks took some 60 us a launch).  out(c, totals) runs in one thread a
// column; all threads call.
template <int NV, class Out>
__device__ __forceinline__ void sum_partials(const double *part, unsigned blocks, int cols, Out out) {
    __shared__ double s_sum[NV][kBT];
    const int c = threadIdx.x % cols, g = threadIdx.x / cols, ng = kBT / cols;   // cols: a power of two <= 64
    double a[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) a[v] = 0.0;
#pragma unroll 8
    for (unsigned b = g; b < blocks; b += ng)
#pragma unroll
        for (int v = 0; v < NV; v++) a[v] += __ldcg(&part[((size_t)b * cols + c) * NV + v]);
#pragma unroll
    for (int v = 0; v < NV; v++) s_sum[v][threadIdx.x] = a[v];
    __syncthreads();
    if (g == 0) {
        for (int q = 1; q < ng; q++)
#pragma unroll
            for (int v = 0; v < NV; v++) a[v] += s_sum[v][q * cols + c];
        out(c, a);
    }
    __syncthreads();
}

// Block sums of a kernel whose thread t holds NV sums of each of the V columns
// V (t mod K / V) ..: to part[blockIdx.x][K][NV].
template <int NV, int V>
__device__ __forceinline__ void store_partials(const double (&a)[NV][V], int K, double *part) {
    __shared__ double s_part[NV][V][kBT];
#pragma unroll
    for (int v = 0; v < NV; v++)
#pragma unroll
        for (int q = 0; q < V; q++) s_part[v][q][threadIdx.x] = a[v][q];
    __syncthreads();
    for (int t = threadIdx.x; t < K * NV; t += kBT) {
        const int c = t / NV, v = t % NV;
        double sum = 0.0;
        for (int u = c / V; u < kBT; u += K / V) sum += s_part[v][c % V][u];
        part[((size_t)blockIdx.x * K + c) * NV + v] = sum;
    }
}

// ---------------------------------------------------------------------------
// P = R / D + beta P.  A thread keeps its V columns over all its rows (the
// grid's threads are a multiple of K / V), so their scalars are read once.
template <typename VT>
__global__ void __launch_bounds__(kBT)
bdir_kernel(BlockPtrs B, const VT *__restrict__ R, const VT *__restrict__ D, VT *__restrict__ P) {
    if (B.flags[0]) return;
    constexpr int V = BVec<VT>::V;
    const int G = B.K / V, k0 = V * (threadIdx.x & (G - 1));
    bool open[V], begin[V], any = false;
    VT beta[V];
#pragma unroll
    for (int q = 0; q < V; q++) {
        open[q] = !B.done[k0 + q];
        begin[q] = B.nits[k0 + q] == 0;
        const double rp = B.rz_prev[k0 + q];
        beta[q] = (VT)(rp == 0.0 ? 0.0 : B.rz_cur[k0 + q] / rp);
        any = any || open[q];
    }
    if (!any) return;
    const int64_t step = (int64_t)gridDim.x * kBT / G;
#pragma unroll 2
    for (int64_t i = ((int64_t)blockIdx.x * kBT + threadIdx.x) / G; i < B.n; i += step) {
        const VT d = __ldg(&D[i]);
        const BArr<VT> r = bload_ro(R + i * B.K + k0);
        BArr<VT> p = bload(P + i * B.K + k0);
#pragma unroll
        for (int q = 0; q < V; q++) {
            const VT z = r.v[q] / d;
            if (open[q]) p.v[q] = begin[q] ? z : beta[q] * p.v[q] + z;
        }
        bstore(P + i * B.K + k0, p);
    }
}

// AP = A P for one tile of T columns; per-column partial sums of p . Ap.  T / V
// lanes a row, each V columns as one 16-byte gather; four entries in flight.
// The rows go to the blocks kRowChunk at a time: neighbouring rows gather the
// same rows of P, which the first of them leaves in L1.
constexpr int kRowChunk = 64;

template <typename VT, int T>
__global__ void __launch_bounds__(kBT, 4)
bspmm_kernel(BlockPtrs B, const VT *__restrict__ va, const VT *__restrict__ P, VT *__restrict__ AP) {
    if (B.flags[0]) return;
    constexpr int V = BVec<VT>::V, L = T / V, RPW = 32 / L, U = 4;
    __shared__ double s_dot[kBT / 32][T];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, sub = lane / L, gl = lane % L;
    const int tile = blockIdx.y, K = B.K, k0 = tile * T + V * gl;
    double dot[V];
#pragma unroll
    for (int q = 0; q < V; q++) dot[q] = 0.0;
    for (int64_t chunk = blockIdx.x; chunk * kRowChunk < B.n; chunk += gridDim.x) {
#pragma unroll 1
        for (int r = w * RPW + sub; r < kRowChunk; r += (kBT / 32) * RPW) {
            const int64_t row = chunk * kRowChunk + r;
            if (row >= B.n) break;
            const int32_t b = __ldg(&B.rp[row]), e = __ldg(&B.rp[row + 1]);
            VT acc[V];
#pragma unroll
            for (int q = 0; q < V; q++) acc[q] = (VT)0;
            for (int32_t j = b; j < e; j += U) {
                int32_t c[U];
                VT v[U];
                BArr<VT> p[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const bool in = j + u < e;
                    c[u] = in ? __ldg(&B.ci[j + u]) : 0;
                    v[u] = in ? __ldg(&va[j + u]) : (VT)0;
                }
#pragma unroll
                for (int u = 0; u < U; u++) p[u] = bload_ro(P + (int64_t)c[u] * K + k0);
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (j + u < e)
#pragma unroll
                        for (int q = 0; q < V; q++) acc[q] += v[u] * p[u].v[q];
            }
            const BArr<VT> own = bload_ro(P + row * K + k0);
            BArr<VT> out;
#pragma unroll
            for (int q = 0; q < V; q++) {
                out.v[q] = acc[q];
                dot[q] += (double)own.v[q] * (double)acc[q];
            }
            bstore(AP + row * K + k0, out);
        }
    }
    __syncwarp();
    // per-column block sums: the warp's rows, then the warps, in a fixed order
#pragma unroll
    for (int q = 0; q < V; q++) {
        double v = dot[q];
        for (int o = L; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (sub == 0) s_dot[w][V * gl + q] = v;
    }
    __syncthreads();
    double *part = B.partials + (size_t)tile * kBMaxBlocks * T;
    for (int c = threadIdx.x; c < T; c += blockDim.x) {
        double s = 0.0;
        for (int ww = 0; ww < kBT / 32; ww++) s += s_dot[ww][c];
        part[(size_t)blockIdx.x * T + c] = s;
    }
    if (!last_block(&B.tickets[tile], gridDim.x)) return;
    sum_partials<1>(part, gridDim.x, T, [&](int c, const double *a) {
        const int k = tile * T + c;
        const double s = a[0];
        if (!B.done[k]) {
            B.pAp[k] = s;
            if (s == 0.0) {
                B.alpha[k] = 0.0;
                B.done[k] = 1;
                B.status[k] = 1;   // breakdown
                B.nits[k] += 1;
            } else {
                B.alpha[k] = B.rz_cur[k] / s;
            }
        }
    });
    if (threadIdx.x == 0) B.tickets[tile] = 0u;
}

// X += alpha P (or Y = [reset ? 0 : Y] + alpha P), R -= alpha AP; per-column
// ||r||^2 and r.(r/D); the last block closes the iteration of every column.
template <typename VT, bool MIXED>
__global__ void __launch_bounds__(kBT)
bupdate_kernel(BlockPtrs B, VT *__restrict__ X, VT *__restrict__ R, const VT *__restrict__ P,
               const VT *__restrict__ AP, const VT *__restrict__ D) {
    if (B.flags[0]) return;
    constexpr int V = BVec<VT>::V;
    const int K = B.K, G = K / V, k0 = V * (threadIdx.x & (G - 1));
    const bool reset = MIXED && B.flags[3];
    double sums[2][V];
    bool open[V], any = false;
    VT a[V];
#pragma unroll
    for (int q = 0; q < V; q++) {
        sums[0][q] = sums[1][q] = 0.0;
        open[q] = !B.done[k0 + q];
        a[q] = (VT)B.alpha[k0 + q];
        any = any || open[q];
    }
    const int64_t step = (int64_t)gridDim.x * kBT / G;
    if (any)
#pragma unroll 2
        for (int64_t i = ((int64_t)blockIdx.x * kBT + threadIdx.x) / G; i < B.n; i += step) {
            const int64_t at = i * K + k0;
            const VT d = __ldg(&D[i]);
            const BArr<VT> p = bload_ro(P + at), ap = bload_ro(AP + at);
            BArr<VT> x = bload(X + at), r = bload(R + at);
#pragma unroll
            for (int q = 0; q < V; q++) {
                if (!open[q]) continue;
                x.v[q] = (reset ? (VT)0 : x.v[q]) + a[q] * p.v[q];
                const VT ri = r.v[q] - a[q] * ap.v[q];
                r.v[q] = ri;
                sums[0][q] += (double)ri * (double)ri;
                sums[1][q] += (double)ri * (double)(ri / d);
            }
            bstore(X + at, x);
            bstore(R + at, r);
        }
    double *part = B.partials + (size_t)kBMaxBlocks * 64 * 2;   // after the SpMM tiles
    store_partials<2, V>(sums, K, part);
    if (!last_block(&B.tickets[64], gridDim.x)) return;
    __shared__ int s_open, s_ru, s_final;
    if (threadIdx.x == 0) { s_open = 0; s_ru = 0; s_final = 0; }
    __syncthreads();
    sum_partials<2>(part, gridDim.x, K, [&](int c, const double *t) {
        if (B.done[c]) return;
        const double res = sqrt(t[0]);
        const int it = B.nits[c] + 1;
        B.nits[c] = it;
        B.res[c] = res;
        B.rz_prev[c] = B.rz_cur[c];
        B.rz_cur[c] = t[1];
        if (!isfinite(res)) {
            B.done[c] = 1;
            B.status[c] = 2;
        } else if (MIXED) {
            if (!(res > B.tol[c]) || it >= B.flags[4]) { atomicOr(&s_ru, 1); atomicOr(&s_final, 1); }
            else if (res < B.delta * B.maxr[c]) atomicOr(&s_ru, 1);
            atomicOr(&s_open, 1);
        } else {
            if (!(res > B.tol[c]) || it >= B.flags[4]) B.done[c] = 1;
            else atomicOr(&s_open, 1);
        }
    });
    if (threadIdx.x == 0) {
        B.tickets[64] = 0u;
        if (MIXED) {
            B.flags[3] = 0;
            if (s_ru) { B.flags[1] = 1; B.flags[2] = s_final; }
        }
        if (!s_open) B.flags[0] = 1;
    }
}

// Reliable update for all open columns: X += Y, Rt -= A Y (FP64 matrix),
// R32 = (float) Rt, per-column ||Rt||^2 and r32.(r32/D).  Rows and lanes as
// the FP32 product.
template <int T>
__global__ void __launch_bounds__(kBT)
breliable_kernel(BlockPtrs B, const double *__restrict__ va, double *__restrict__ X, const float *__restrict__ Y,
                 double *__restrict__ Rt, float *__restrict__ R32, const float *__restrict__ D) {
    if (B.flags[0] || !B.flags[1]) return;
    constexpr int V = 4, L = T / V, RPW = 32 / L, U = 4;
    __shared__ double s_a[kBT / 32][T], s_b[kBT / 32][T];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, sub = lane / L, gl = lane % L;
    const int tile = blockIdx.y, K = B.K, k0 = tile * T + V * gl;
    double s1[V], s2[V];
    bool open[V];
#pragma unroll
    for (int q = 0; q < V; q++) {
        s1[q] = s2[q] = 0.0;
        open[q] = !B.done[k0 + q];
    }
    for (int64_t chunk = blockIdx.x; chunk * kRowChunk < B.n; chunk += gridDim.x) {
#pragma unroll 1
        for (int r = w * RPW + sub; r < kRowChunk; r += (kBT / 32) * RPW) {
            const int64_t row = chunk * kRowChunk + r;
            if (row >= B.n) break;
            const int32_t b = __ldg(&B.rp[row]), e = __ldg(&B.rp[row + 1]);
            double acc[V];
#pragma unroll
            for (int q = 0; q < V; q++) acc[q] = 0.0;
            for (int32_t j = b; j < e; j += U) {
                int32_t c[U];
                double v[U];
                BArr<float> y[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const bool in = j + u < e;
                    c[u] = in ? __ldg(&B.ci[j + u]) : 0;
                    v[u] = in ? __ldg(&va[j + u]) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; u++) y[u] = bload_ro(Y + (int64_t)c[u] * K + k0);
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (j + u < e)
#pragma unroll
                        for (int q = 0; q < V; q++) acc[q] += v[u] * (double)y[u].v[q];
            }
            const int64_t at = row * K + k0;
            const float d = __ldg(&D[row]);
#pragma unroll
            for (int q = 0; q < V; q++) {
                if (!open[q]) continue;
                X[at + q] += (double)Y[at + q];
                const double rt = Rt[at + q] - acc[q];
                Rt[at + q] = rt;
                const float rf = (float)rt;
                R32[at + q] = rf;
                s1[q] += rt * rt;
                s2[q] += (double)rf * (double)(rf / d);
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < V; q++) {
        double a = s1[q], c2 = s2[q];
        for (int o = L; o < 32; o <<= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            c2 += __shfl_xor_sync(0xffffffffu, c2, o);
        }
        if (sub == 0) { s_a[w][V * gl + q] = a; s_b[w][V * gl + q] = c2; }
    }
    __syncthreads();
    double *part = B.partials + (size_t)tile * kBMaxBlocks * T * 2;
    for (int c = threadIdx.x; c < T; c += blockDim.x) {
        double a = 0.0, c2 = 0.0;
        for (int ww = 0; ww < kBT / 32; ww++) { a += s_a[ww][c]; c2 += s_b[ww][c]; }
        part[((size_t)blockIdx.x * T + c) * 2] = a;
        part[((size_t)blockIdx.x * T + c) * 2 + 1] = c2;
    }
    if (!last_block(&B.tickets[65 + tile], gridDim.x)) return;
    sum_partials<2>(part, gridDim.x, T, [&](int c, const double *t) {
        const int k = tile * T + c;
        if (B.done[k]) return;
        const double res = sqrt(t[0]);
        B.res[k] = res;
        B.rz_cur[k] = t[1];
        B.maxr[k] = res;
        if (B.flags[2] && (!(res > B.tol[k]) || B.nits[k] >= B.flags[4])) B.done[k] = 1;
    });
    if (threadIdx.x == 0) B.tickets[65 + tile] = 0u;
    // the tiles finish independently; the last tile to finish closes the update
    __shared__ bool lastTile;
    if (threadIdx.x == 0) {
        __threadfence();
        lastTile = atomicAdd(&B.tickets[130], 1u) == gridDim.y - 1;
    }
    __syncthreads();
    if (lastTile && threadIdx.x == 0) {
        __threadfence();
        B.tickets[130] = 0u;
        int open_cols = 0;
        for (int k = 0; k < K; k++) open_cols |= !*reinterpret_cast<volatile int *>(&B.done[k]);
        B.flags[1] = 0;
        B.flags[2] = 0;
        B.flags[3] = 1;
        if (!open_cols) B.flags[0] = 1;
    }
}

// ---------------------------------------------------------------------------
static int blocks_for(int64_t work) {
    int64_t b = (work + kBT - 1) / kBT;
    if (b > kBMaxBlocks) b = kBMaxBlocks;
    return (int)(b < 1 ? 1 : b);
}

static dim3 spmm_grid(const BlockPtrs &B, int T) {
    const int64_t chunks = ceil_div(B.n, kRowChunk);
    return dim3((unsigned)(chunks < kBMaxBlocks ? chunks : kBMaxBlocks), B.K / T);
}

template <typename VT>
static void spmm_launch(int T, const BlockPtrs &B, const VT *va, const VT *P, VT *AP, cudaStream_t s) {
    const dim3 grid = spmm_grid(B, T);
    switch (T) {
    case 8: bspmm_kernel<VT, 8><<<grid, kBT, 0, s>>>(B, va, P, AP); break;
    case 16: bspmm_kernel<VT, 16><<<grid, kBT, 0, s>>>(B, va, P, AP); break;
    case 32: bspmm_kernel<VT, 32><<<grid, kBT, 0, s>>>(B, va, P, AP); break;
    default: bspmm_kernel<VT, 64><<<grid, kBT, 0, s>>>(B, va, P, AP); break;
    }
}

cudaError_t launch_block_iteration(const BlockPtrs &B, int T, bool mixed, const BlockVecs &V, cudaStream_t s) {
    if (!mixed) {
        const int vb = blocks_for(B.n * (B.K / 2));   // 16 bytes a thread and row
        bdir_kernel<double><<<vb, kBT, 0, s>>>(B, V.R, V.D, V.P);
        spmm_launch<double>(T, B, V.va, V.P, V.AP, s);
        bupdate_kernel<double, false><<<vb, kBT, 0, s>>>(B, V.X, V.R, V.P, V.AP, V.D);
    } else {
        const int vb = blocks_for(B.n * (B.K / 4));
        bdir_kernel<float><<<vb, kBT, 0, s>>>(B, V.R32, V.D32, V.P32);
        spmm_launch<float>(T, B, V.va32, V.P32, V.AP32, s);
        bupdate_kernel<float, true><<<vb, kBT, 0, s>>>(B, V.Y32, V.R32, V.P32, V.AP32, V.D32);
        const dim3 grid = spmm_grid(B, T);
        switch (T) {
        case 8: breliable_kernel<8><<<grid, kBT, 0, s>>>(B, V.va, V.X, V.Y32, V.R, V.R32, V.D32); break;
        case 16: breliable_kernel<16><<<grid, kBT, 0, s>>>(B, V.va, V.X, V.Y32, V.R, V.R32, V.D32); break;
        case 32: breliable_kernel<32><<<grid, kBT, 0, s>>>(B, V.va, V.X, V.Y32, V.R, V.R32, V.D32); break;
        default: breliable_kernel<64><<<grid, kBT, 0, s>>>(B, V.va, V.X, V.Y32, V.R, V.R32, V.D32); break;
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_block_spmm64(const BlockPtrs &B, int T, const double *va, const double *P, double *AP,
                                cudaStream_t s) {
    spmm_launch<double>(T, B, va, P, AP, s);
    return cudaGetLastError();
}

cudaError_t launch_block_spmm32(const BlockPtrs &B, int T, const float *va, const float *P, float *AP,
                                cudaStream_t s) {
    spmm_launch<float>(T, B, va, P, AP, s);
    return cudaGetLastError();
}

size_t block_partials_doubles() { return (size_t)kBMaxBlocks * 64 * 2 * 2 + 64; }
size_t block_ticket_count() { return 131; }

// Initial state of every column from R (= B - A X0, FP64): tolerance
// rtol * ||r0||, r.(r/D), and for the mixed solver the FP32 copies.
template <bool MIXED>
__global__ void __launch_bounds__(kBT)
binit_kernel(BlockPtrs B, const double *__restrict__ R, const double *__restrict__ D, float *__restrict__ R32,
             float *__restrict__ D32, float *__restrict__ Y32, double rtol) {
    const int K = B.K;
    const int k = threadIdx.x % K;
    const int64_t rows_per_step = ((int64_t)gridDim.x * blockDim.x) / K;
    double rr = 0.0, rz = 0.0;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / K; i < B.n; i += rows_per_step) {
        const int64_t t = i * K + k;
        const double r = R[t];
        if (MIXED) {
            const float rf = (float)r, df = (float)D[i];
            R32[t] = rf;
            Y32[t] = 0.0f;
            if (k == 0) D32[i] = df;
            rr += r * r;
            rz += (double)rf * (double)(rf / df);
        } else {
            rr += r * r;
            rz += r * (r / D[i]);
        }
    }
    __shared__ double s_rr[kBT], s_rz[kBT];
    s_rr[threadIdx.x] = rr;
    s_rz[threadIdx.x] = rz;
    __syncthreads();
    double *part = B.partials + (size_t)kBMaxBlocks * 64 * 2;
    for (int c = threadIdx.x; c < K; c += blockDim.x) {
        double a1 = 0.0, a2 = 0.0;
        for (int t = c; t < (int)blockDim.x; t += K) { a1 += s_rr[t]; a2 += s_rz[t]; }
        part[((size_t)blockIdx.x * K + c) * 2] = a1;
        part[((size_t)blockIdx.x * K + c) * 2 + 1] = a2;
    }
    if (!last_block(&B.tickets[64], gridDim.x)) return;
    sum_partials<2>(part, gridDim.x, K, [&](int c, const double *t) {
        const double a2 = t[1], r0 = sqrt(t[0]);
        B.res[c] = r0;
        B.maxr[c] = r0;
        B.tol[c] = r0 * rtol;
        B.rz_cur[c] = a2;
        B.rz_prev[c] = 0.0;
        B.nits[c] = 0;
        B.status[c] = 0;
        B.done[c] = !(r0 > r0 * rtol) || B.flags[4] <= 0 || !isfinite(a2);
        if (!isfinite(a2)) B.status[c] = 2;
    });
    __syncthreads();
    if (threadIdx.x == 0) {
        B.tickets[64] = 0u;
        int open = 0;
        for (int c = 0; c < K; c++) open |= !B.done[c];
        B.flags[0] = !open;
        B.flags[1] = 0;
        B.flags[2] = 0;
        B.flags[3] = 1;
    }
}

cudaError_t launch_block_init(const BlockPtrs &B, bool mixed, const double *R, const double *D, float *R32,
                              float *D32, float *Y32, double rtol, cudaStream_t s) {
    const int nb = blocks_for(B.n * B.K);
    if (mixed) binit_kernel<true><<<nb, kBT, 0, s>>>(B, R, D, R32, D32, Y32, rtol);
    else binit_kernel<false><<<nb, kBT, 0, s>>>(B, R, D, R32, D32, Y32, rtol);
    return cudaGetLastError();
}

// R[i*K + k] = k < m ? Bin[i*m + k] : 0  (and the reverse for the output)
__global__ void pack_kernel(int64_t n, int m, int K, const double *__restrict__ in, double *__restrict__ out) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n * K; t += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(t % K);
        out[t] = k < m ? in[(t / K) * m + k] : 0.0;
    }
}
__global__ void unpack_kernel(int64_t n, int m, int K, const double *__restrict__ in, double *__restrict__ out) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n * m; t += (int64_t)gridDim.x * blockDim.x)
        out[t] = in[(t / m) * K + t % m];
}
__global__ void sub_kernel(int64_t total, const double *__restrict__ a, double *__restrict__ b) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x)
        b[t] = a[t] - b[t];
}
__global__ void to_float_kernel(int64_t n, const double *__restrict__ a, float *__restrict__ b) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        b[t] = (float)a[t];
}

cudaError_t launch_block_pack(int64_t n, int m, int K, const double *in, double *out, cudaStream_t s) {
    pack_kernel<<<blocks_for(n * K), kBT, 0, s>>>(n, m, K, in, out);
    return cudaGetLastError();
}
cudaError_t launch_block_unpack(int64_t n, int m, int K, const double *in, double *out, cudaStream_t s) {
    unpack_kernel<<<blocks_for(n * m), kBT, 0, s>>>(n, m, K, in, out);
    return cudaGetLastError();
}
cudaError_t launch_block_sub(int64_t total, const double *a, double *b, cudaStream_t s) {
    sub_kernel<<<blocks_for(total), kBT, 0, s>>>(total, a, b);
    return cudaGetLastError();
}
cudaError_t launch_to_float(int64_t n, const double *a, float *b, cudaStream_t s) {
    to_float_kernel<<<blocks_for(n), kBT, 0, s>>>(n, a, b);
    return cudaGetLastError();
}

}  // namespace phgb
