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
// Where slices are few or rows long, H = 2 or 4 lanes share a row (its entries
// in turn), so that a slice is the work of H warps; where there are more such
// units than warps, the warps take them as they come free, so that long units
// do not queue behind one another.
#pragma once
#include "common.cuh"
#include "grid_sync.cuh"
#include "solve.h"

namespace phgb {

constexpr int kCoopMaxRowLen = 1024;   // of any of these solvers (coop_max_row)

// Shared memory of the row bookkeeping of a block with that many slices: the
// rows' lengths and each unit's first entry.
__host__ __device__ constexpr int64_t coop_rows_bytes(int64_t slices, int lanes) {
    return slices * (4 * lanes + 32 * 2);
}

// Places of the calling block: 32 for each of its slices.
__device__ __forceinline__ int coop_places(int64_t n) {
    return 32 * (int)(((n + 31) / 32 - blockIdx.x + gridDim.x - 1) / gridDim.x);
}

// Entry c of a vector: a pointer (read with plain loads: other blocks write it
// between barriers) or a function of the column.
template <class V> __device__ __forceinline__ V entry_of(const V *x, int32_t c) { return x[c]; }
template <class F> __device__ __forceinline__ auto entry_of(const F &f, int32_t c) -> decltype(f(c)) { return f(c); }

template <int H>
struct CoopRows {
    int slices;             // of the block; its slice k is slice blockIdx.x + gridDim.x * k
    unsigned n;             // rows of the matrix
    int32_t *off;           // shared, [H slices] first entry of each unit
    uint16_t *len;          // shared, [32 slices] row lengths
    int *next;              // shared, the next unit to take
    int32_t *cols;          // global, the matrix's columns in step order

    // Places 0 .. 32 slices - 1 are the block's rows, in slice order; row()
    // gives the matrix row, which is n or more for the last slice's padding.
    __device__ __forceinline__ unsigned row(int place) const {
        return 32u * (blockIdx.x + gridDim.x * (unsigned)(place >> 5)) + (place & 31);
    }

    __device__ __forceinline__ CoopRows(int64_t rows, void *shared, int *next_unit, int32_t *c) {
        n = (unsigned)rows;
        slices = coop_places(rows) / 32;
        off = (int32_t *)shared;
        len = (uint16_t *)(off + H * slices);
        next = next_unit;
        cols = c;
    }

    // Unit u is 32 / H consecutive places, lane `lane` at this one.
    __device__ __forceinline__ int place_of(int unit, int lane) const { return (32 * unit + lane) / H; }
    // Entries of a row of l the lane takes: lane % H, lane % H + H, ...
    __device__ __forceinline__ int own(int l, int lane) const { return (l + H - 1 - lane % H) / H; }

    // Copies the CSR rows of the block into step order: columns to cols, and
    // put(place, value) the values.  All threads call it, the block's next
    // barrier completes it.
    template <class Put>
    __device__ __forceinline__ void build(const CsrView &A, Put put) const {
        constexpr int U = 4;
        const int lane = threadIdx.x & 31;
        const unsigned lt = (1u << lane) - 1u;
        if (threadIdx.x == 0) *next = kCoopWarps;
        for (int unit = threadIdx.x >> 5; unit < H * slices; unit += kCoopWarps) {
            const int place = place_of(unit, lane);
            const unsigned r = row(place);
            const int32_t b = A.rp[min(r, n)], e = A.rp[min(r + 1, n)];
            const int mine = own(e - b, lane), width = __reduce_max_sync(0xffffffffu, (unsigned)mine);
            int at = __shfl_sync(0xffffffffu, b, 0);
            if (lane % H == 0) len[place] = (uint16_t)(e - b);
            if (lane == 0) off[unit] = at;
            for (int j = 0; j < width; j += U) {
                int32_t c[U];
                double v[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const bool in = j + u < mine;
                    const int32_t q = b + (j + u) * H + lane % H;
                    c[u] = in ? __ldg(&A.ci[q]) : 0;
                    v[u] = in ? __ldg(&A.va[q]) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const unsigned m = __ballot_sync(0xffffffffu, j + u < mine);
                    if (j + u < mine) {
                        const int q = at + __popc(m & lt);
                        cols[q] = c[u];
                        put(q, v[u]);
                    }
                    at += __popc(m);
                }
            }
        }
    }

    // y[place] = (A x)_row for the block's places (shared memory, zero in the
    // padding), values `vals` in step order, x a vector or a function of the column
    // (entry_of).  All threads call it, with y free to write; y is complete
    // when it returns.  ORDERED: each row's sum takes its
    // entries in CSR order, one by one, whatever H (the sums of the launched
    // SELL products); otherwise the lanes' sums are added.
    template <bool ORDERED, class V, class X>
    __device__ __forceinline__ void product(const V *vals, X x, V *y) const {
        const int lane = threadIdx.x & 31, units = H * slices;
        for (int unit = threadIdx.x >> 5; unit < units;) {
            const int place = place_of(unit, lane);
            const V acc = row_sum<ORDERED>(vals, x, off[unit], len[place]);
            if (lane % H == 0) y[place] = acc;
            unit = units;
            if (units > kCoopWarps) {
                if (lane == 0) unit = atomicAdd(next, 1);
                unit = __shfl_sync(0xffffffffu, unit, 0);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) *next = kCoopWarps;   // before the next product: every caller has a barrier between
    }

    // f(place, (A x)_row) in one lane for each of the block's places: the
    // product (ordered) without a place to keep it, the units dealt to the
    // warps in turn.
    template <class V, class X, class F>
    __device__ __forceinline__ void product_each(const V *vals, X x, F f) const {
        const int lane = threadIdx.x & 31;
        for (int unit = threadIdx.x >> 5; unit < H * slices; unit += kCoopWarps) {
            const int place = place_of(unit, lane);
            const V acc = row_sum<true>(vals, x, off[unit], len[place]);
            if (lane % H == 0) f(place, acc);
        }
    }

private:
    // Sum of the lane's row, of length l, in every lane of the row; the
    // unit's entries start at `at`.  FP32 entries are loaded a batch ahead of
    // the gathers they feed (FP64 ones would not fit the registers).
    template <bool ORDERED, class V, class X>
    __device__ __forceinline__ V row_sum(const V *vals, X x, int at, int l) const {
        constexpr int U = 8;
        constexpr bool ahead = sizeof(V) == 4;
        const int lane = threadIdx.x & 31, mine = own(l, lane);
        const int width = __reduce_max_sync(0xffffffffu, (unsigned)mine);
        const unsigned lt = (1u << lane) - 1u;
        V acc = (V)0;
        int32_t c[U], cn[ahead ? U : 1];
        V v[U], vn[ahead ? U : 1];
        auto load = [&](int j, int32_t *cc, V *vv) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const unsigned m = __ballot_sync(0xffffffffu, j + u < mine);
                cc[u] = -1;
                vv[u] = (V)0;
                if (j + u < mine) {
                    const int q = at + __popc(m & lt);
                    cc[u] = load_once(cols + q);
                    vv[u] = load_once(vals + q);
                }
                at += __popc(m);
            }
        };
        if (ahead) load(0, cn, vn);
        for (int j = 0; j < width; j += U) {
            if (ahead) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    c[u] = cn[ahead ? u : 0];
                    v[u] = vn[ahead ? u : 0];
                }
                load(j + U, cn, vn);
            } else {
                load(j, c, v);
            }
            V xv[U];
#pragma unroll
            for (int u = 0; u < U; u++) xv[u] = c[u] >= 0 ? entry_of(x, c[u]) : (V)0;
            if constexpr (ORDERED && H > 1) {
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int h = 0; h < H; h++) {
                        const bool in = (j + u) * H + h < l;
                        if constexpr (sizeof(V) == 4) {
                            const V p = __shfl_sync(0xffffffffu, __fmul_rn(v[u], xv[u]), h, H);
                            if (in) acc = __fadd_rn(acc, p);
                        } else {
                            const V vh = __shfl_sync(0xffffffffu, v[u], h, H), xh = __shfl_sync(0xffffffffu, xv[u], h, H);
                            if (in) acc = fma(vh, xh, acc);
                        }
                    }
            } else {
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (c[u] >= 0) {
                        if constexpr (sizeof(V) == 4) acc = fma_free(acc, v[u], xv[u]);   // as the launched FP32 products
                        else acc = fma(v[u], xv[u], acc);
                    }
            }
        }
        if constexpr (!ORDERED)
#pragma unroll
            for (int o = H / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, H);
        return acc;
    }

    // Matrix words are read once per product: they stay out of L1, which the
    // gathers need.
    static __device__ __forceinline__ int32_t load_once(const int32_t *p) {
        int32_t v;
        asm volatile("ld.global.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
        return v;
    }
    static __device__ __forceinline__ float load_once(const float *p) {
        float v;
        asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
        return v;
    }
    static __device__ __forceinline__ double load_once(const double *p) {
        double v;
        asm volatile("ld.global.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
        return v;
    }
};

// Lanes per row (at most `most`) for a matrix of n rows and nnz entries whose
// blocks have at most that many slices: enough units for the 32 warps, two a
// warp where rows have 16 entries or more and six where they have 32 or more
// (P3's vertex rows, 175 entries against 41 on average, outlast the rest
// otherwise), while a lane keeps four entries or more.  Measured us per
// iteration with 1 / 2 / 4 lanes: FP64 PCG P1 36k rows (8 slices) 8.7 / 7.9 /
// 8.0, P1 133k (28) 10.4 / 10.9 / 13.2, P2 69k (15) 16.1 / 13.9 / 11.3, P2 250k
// (53) 22.5 / 23.9 / 24.5, P2 531k (113) 38.5 / 44.6 / 47.3, P3 227k (48) 39.9 /
// 31.5 / 30.8; mixed PCG, whose ordered sums cost more lanes more, P1 36k 7.5 /
// 7.2 / 8.4, P2 69k 12.6 / 11.1 / 12.2, P2 250k 18.7 / 21.4 / 26.6, P3 227k 29.6 /
// 25.6 / 30.7.
inline int coop_lanes(int64_t slices, int64_t n, int64_t nnz, int most) {
    const int64_t units = nnz >= 32 * n ? 192 : nnz >= 16 * n ? 64 : kCoopWarps;
    int h = 1;
    while (h < most && 2 * h * slices <= units && nnz >= 8 * h * n) h *= 2;
    return h;
}

// The longest row an FP64 solver takes.  A row is its lanes' serial work, some
// 0.14 us an entry and lane while the other blocks wait, where the launched
// products share it among up to 32 lanes: so it may cost what the launches cost
// and what the blocks' average product hides.  `spare` is the first in entries
// a lane, an entry of a block's product counts 1/128 of one.  Measured us per
// iteration, 7 entries a row and one row of L, one kernel / launched:
// PCG (spare 72)          L = 7        100         200         500
//   2.2k rows         6.5 / 15.8  20.6 / 16.0  34.6 / 17.1  80.4 / 19.5
//   39k               6.6 / 15.1  18.8 / 17.8  32.1 / 19.8  71.7 / 23.3
//   373k             12.8 / 23.2  19.9 / 28.0  30.0 / 33.3  59.2 / 46.3
// BiCGstab (64, two products an iteration)
//   39k              14.1 / 29.8  33.0 / 30.5  53.1 / 34.4   114 / 47.7
//   373k             24.3 / 48.4  40.6 / 57.7  63.6 / 65.8   131 / 77.2
// GMRES, restart 10 (176)
//   2.2k             20.5 / 40.8  31.6 / 42.9  44.0 / 41.6  82.7 / 45.5
//   39k              20.7 / 43.0  31.1 / 45.5  42.6 / 45.6  77.2 / 53.0
//   373k             33.2 / 58.2  42.2 / 63.3  54.5 / 68.8  95.0 / 76.2
// Meshes of random points stay below it: PCG, P3 on 3,000 points (rows of up to 371
// entries, 47 on average, four lanes) 22.8 / 29.4, on 9,000 (two lanes) 49.3 / 65.9.
// The mixed solver's launched FP32 products give a row one lane too, and it has
// no limit but kCoopMaxRowLen: L = 1000, 2.2k rows 72.6 / 93.7, 373k 87.8 / 237.
inline int coop_max_row(int64_t nnz, int blocks, int lanes, int spare) {
    const int64_t most = lanes * (spare + nnz / blocks / 128);
    return most < kCoopMaxRowLen ? (int)most : kCoopMaxRowLen;
}

// The launch of a one-kernel solver on that many multiprocessors: blocks, lanes a row, longest row and shared
// memory (`fixed_bytes`, `row_bytes` of vectors a row, and the row bookkeeping);
// false when it is too large.  `spare`: see coop_max_row, 0 for no limit of the
// kind.
//
// Shared memory a solve takes at most: what it takes the L1 cache loses, and
// the product's gathers need that.  A careful line, the kernels are faster some
// way beyond it: FP64 PCG, us per iteration in one kernel / launched, 121 KB a
// block (P2 531k rows) 38.5 / 58.0, 125 KB (P3 551k) 59.0 / 91.5, and with the
// limit raised 154 KB (P3 681k) 74.6 / 107, 159 KB (P1 705k) 28.2 / 44.4, (P2 705k)
// 51.0 / 72.7, 188 KB (P3 831k) 105 / 125, 194 KB (P2 857k) 69.7 / 72.2, 206 KB (P1
// 913k) 51.0 / 48.2; BiCGstab 130 KB (P3 389k) 96.7 / 169, 183 KB (P3 551k) 154 / 220.
constexpr int64_t kCoopMaxSmem = 136 * 1024;
// A block per this many entries (a row's vector work counted as four) while
// there are SMs.  Us per iteration with 1024 / 2048 / 4096 / 8192: FP64 PCG P1 343
// rows 6.6 / 6.5 / 3.3 / 3.4 (one block, no barriers, from 4096 on), P1 729 6.6 /
// 6.6 / 6.8 / 4.6, P1 3.4k 6.3 / 6.4 / 6.6 / 7.8, P1 36k 6.7 / 6.7 / 6.7 / 8.3, P2
// 6.9k 8.1 / 8.0 / 8.4 / 9.5, P3 15.6k 12.7 / 12.8 / 12.3 / 13.2; mixed P1 9.3k 6.7 /
// 6.7 / 7.3 / 7.7; GMRES P1 343 18.4 / 18.2 / 8.1 / 8.0, P1 3.4k 20.3 / 20.3 / 20.5 /
// 21.8: more blocks than 4096 gives save next to nothing, and cost the smallest
// systems their barriers.
constexpr int64_t kCoopBlockWork = 4096;

struct CoopSplit {
    int blocks = 0, lanes = 1, max_row = 0;
    int64_t smem = 0;
};

inline bool coop_split(int64_t n, int64_t nnz, int64_t row_bytes, int64_t fixed_bytes, int most_lanes, int spare,
                       int sms, CoopSplit *out) {
    int dev = 0, coop = 0, most = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (!coop || sms < 1) return false;
    if (sms > kCoopMaxBlocks) sms = kCoopMaxBlocks;
    const int64_t slices = ceil_div(n, 32);
    int64_t G = ceil_div(nnz + 4 * n, kCoopBlockWork);
    if (G > slices) G = slices;
    if (G > sms) G = sms;
    const int64_t per = ceil_div(slices, G);
    out->blocks = (int)G;
    out->lanes = coop_lanes(per, n, nnz, most_lanes);
    out->max_row = spare > 0 ? coop_max_row(nnz, out->blocks, out->lanes, spare) : kCoopMaxRowLen;
    out->smem = fixed_bytes + 32 * per * row_bytes + coop_rows_bytes(per, out->lanes);
    return out->smem <= kCoopMaxSmem && out->smem <= most - 4096;   // 4 KB of static shared memory at most
}

// Cooperative launch of kernel(run) with that split, whose longest row goes to
// run.max_row.
template <class Run>
inline cudaError_t coop_launch(void (*kernel)(Run), const Run &run, const CoopSplit &sp, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoopMaxSmem);
    if (e != cudaSuccess) return e;
    Run r = run;
    r.max_row = sp.max_row;
    void *args[] = {(void *)&r};
    return cudaLaunchCooperativeKernel((const void *)kernel, dim3(sp.blocks), dim3(kCoopThreads), args, (size_t)sp.smem, s);
}

}  // namespace phgb
