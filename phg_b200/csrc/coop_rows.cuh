// Rows and products of the one-kernel solvers (grid_sync.cuh): how the rows
// of a matrix are dealt to the blocks of a cooperative grid, and the product of
// a block's rows.
//
// The rows go in slices of 32 consecutive ones, a lane a row, slice s to block
// s mod gridDim: the long rows of a numbering (vertices before edges and
// faces) and the short ones spread over all blocks, and everything a slice
// touches of a vector is one 256-byte segment.  The matrix is copied slice by
// slice into the order the product reads it: step j holds entry j of the rows
// that have one, packed, so a slice fills the same places as its CSR rows and
// its loads are coalesced.  The 32 gathers of a step are the same neighbour of
// consecutive rows and share cache lines.
//
// A block with fewer slices than warps splits each slice's steps into `parts`
// ranges for as many warps, whose sums are added in order; where there are more
// (slice, part) units than warps, the warps take them as they come free, so
// that long slices do not queue behind one another.
#pragma once
#include "common.cuh"
#include "grid_sync.cuh"
#include "solve.h"

namespace phgb {

constexpr int kCoopMaxRowLen = 1024;   // longer rows would be a lane's serial work

// Parts per slice for a matrix of n rows and nnz entries whose blocks have at
// most that many slices: enough units for the 32 warps, and where rows are
// long up to six units a warp, so that the longest slice (a P2 vertex row has
// 65 entries against 25 on average, a P3 one 175 against 41) does not outlast
// the rest; each part keeps four steps or more.  Measured per iteration, parts
// 1 / 2 / 4: P1 36k rows (8 slices) 9.2 / 8.3 / 8.5 us, P1 133k (28) 10.8 / 11.7
// / 14.1, P2 69k (15) 19.4 / 14.6 / 11.9, P2 250k (53) 28.1 / 24.9 / 25.2, P2
// 531k (113) 47.6 / 47.4 / 70.8, P3 227k (48) 51.3 / 35.7 / 32.2.
inline int coop_parts(int64_t slices, int64_t n, int64_t nnz) {
    const int64_t units = nnz >= 16 * n ? 192 : kCoopWarps;
    int p = 1;
    while (p < 4 && 2 * p * slices <= units && nnz >= 8 * p * n) p *= 2;
    return p;
}

// Shared memory of the row bookkeeping of a block with that many slices: the
// sums of all parts but the first, each unit's first entry, and the rows'
// lengths.
constexpr int64_t coop_rows_bytes(int64_t slices, int parts) {
    return slices * (32 * 8 * (parts - 1) + 4 * parts + 32 * 2);
}

struct CoopRows {
    int slices, parts;      // of the block; its slice k is slice blockIdx.x + gridDim.x * k
    unsigned n;             // rows of the matrix
    double *extra;          // shared, [parts - 1][32 slices]
    int32_t *off;           // shared, [slices][parts] first entry of each unit
    uint16_t *len;          // shared, [32 slices] row lengths
    int *next;              // shared, the next unit to take
    int32_t *cols;          // global, the matrix in step order
    double *vals;

    // Places 0 .. places() - 1 are the block's rows, in slice order; row()
    // gives the matrix row, which is n or more for the last slice's padding.
    __device__ __forceinline__ int places() const { return 32 * slices; }
    __device__ __forceinline__ unsigned row(int place) const {
        return 32u * (blockIdx.x + gridDim.x * (unsigned)(place >> 5)) + (place & 31);
    }

    __device__ __forceinline__ CoopRows(int64_t rows, int slice_parts, void *shared, int *next_unit, int32_t *c,
                                        double *v) {
        const int64_t all = (rows + 31) / 32;
        n = (unsigned)rows;
        slices = (int)((all - blockIdx.x + gridDim.x - 1) / gridDim.x);
        parts = slice_parts;
        extra = (double *)shared;
        off = (int32_t *)(extra + (parts - 1) * 32 * slices);
        len = (uint16_t *)(off + parts * slices);
        next = next_unit;
        cols = c;
        vals = v;
    }

    // Steps [j0, j1) of a unit of a slice of `width` steps.
    __device__ __forceinline__ int first_step(int part, int width) const { return (width * part) / parts; }

    // Copies the CSR rows of the block into step order.  All threads call it,
    // the block's next barrier completes it.
    __device__ __forceinline__ void build(const CsrView &A) const {
        constexpr int U = 4;
        const int lane = threadIdx.x & 31;
        const unsigned lt = (1u << lane) - 1u;
        if (threadIdx.x == 0) *next = kCoopWarps;
        for (int k = threadIdx.x >> 5; k < slices; k += kCoopWarps) {
            const unsigned r = row(32 * k + lane);
            const int32_t b = A.rp[min(r, n)], e = A.rp[min(r + 1, n)];
            const int l = e - b, width = __reduce_max_sync(0xffffffffu, (unsigned)l);
            int at = __shfl_sync(0xffffffffu, b, 0), part = 0;
            len[32 * k + lane] = (uint16_t)l;
            for (int j = 0; j < width || part < parts; j += U) {   // one more turn starts parts at the end
                int32_t c[U];
                double v[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    c[u] = j + u < l ? __ldg(&A.ci[b + j + u]) : 0;
                    v[u] = j + u < l ? __ldg(&A.va[b + j + u]) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    for (; part < parts && first_step(part, width) == j + u; part++)
                        if (lane == 0) off[k * parts + part] = at;
                    const unsigned m = __ballot_sync(0xffffffffu, j + u < l);
                    if (j + u < l) {
                        cols[at + __popc(m & lt)] = c[u];
                        vals[at + __popc(m & lt)] = v[u];
                    }
                    at += __popc(m);
                }
            }
        }
    }

    // y[place] = (A x)_row for the block's places (shared memory, zero in the
    // padding).  x is read with plain loads: other blocks write it between
    // barriers.  All threads call it, with y and the parts free to write; y is
    // complete when it returns.
    __device__ __forceinline__ void product(const double *x, double *y) const {
        constexpr int U = 8;
        const int lane = threadIdx.x & 31, units = slices * parts;
        const unsigned lt = (1u << lane) - 1u;
        for (int unit = threadIdx.x >> 5; unit < units;) {
            const int k = unit / parts, part = unit % parts;
            const int l = len[32 * k + lane], width = __reduce_max_sync(0xffffffffu, (unsigned)l);
            const int j1 = first_step(part + 1, width), le = min(l, j1);
            int at = off[unit];
            double acc = 0.0;
            for (int j = first_step(part, width); j < j1; j += U) {
                int32_t c[U];
                double v[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const unsigned m = __ballot_sync(0xffffffffu, j + u < le);
                    c[u] = -1;
                    v[u] = 0.0;
                    if (j + u < le) {
                        const int q = at + __popc(m & lt);
                        c[u] = load_once(cols + q);
                        v[u] = load_once(vals + q);
                    }
                    at += __popc(m);
                }
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (c[u] >= 0) acc += v[u] * x[c[u]];
            }
            (part == 0 ? y : extra + (part - 1) * 32 * slices)[32 * k + lane] = acc;
            unit = units;
            if (units > kCoopWarps) {
                if (lane == 0) unit = atomicAdd(next, 1);
                unit = __shfl_sync(0xffffffffu, unit, 0);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) *next = kCoopWarps;   // before the next product: every caller has a barrier between
        if (parts > 1) {
            for (int i = threadIdx.x; i < 32 * slices; i += kCoopThreads) {
                double s = y[i];
                for (int q = 0; q < parts - 1; q++) s += extra[q * 32 * slices + i];
                y[i] = s;
            }
            __syncthreads();
        }
    }

private:
    // Matrix words are read once per product: they stay out of L1, which the
    // gathers need.
    static __device__ __forceinline__ int32_t load_once(const int32_t *p) {
        int32_t v;
        asm volatile("ld.global.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
        return v;
    }
    static __device__ __forceinline__ double load_once(const double *p) {
        double v;
        asm volatile("ld.global.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
        return v;
    }
};

}  // namespace phgb
