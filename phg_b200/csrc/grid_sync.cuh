// Barriers and sums of a cooperative grid, for the solvers that run as one
// kernel with their vectors on chip (pcg_coop.cu).
//
// An iteration of a Krylov solver is a product and a few passes over vectors,
// separated by sums over all rows.  As separate launches each pass pays a
// launch, the ramp and drain of a grid, and a tree of tickets for its sum;
// inside one resident grid it pays an exchange of a few words.
//
// sum(): each block leaves its partial sums in L2 and counts itself in
// (release); one lane of each block polls the count (acquire), then its warp
// adds all blocks' partials in block order, the same in every block.  The
// scalars that follow from the totals (divisions, square roots) are computed
// once per block, by that warp's lane 0, while the other warps may do work
// that does not depend on them.  (Partials that carry the sum's number, polled
// directly or after the count without a fence, were no faster: 148 blocks
// polling 148 words each cost 5 us an iteration, after the count nothing.)
// sync(): the barrier alone, before a vector that other blocks read.
//
// While such a grid runs it holds the SMs it has blocks on: 1024 threads of up
// to 64 registers are an SM's whole register file, so a solve that has a block on
// every SM (from 606,000 entries on, a row counted as four) lets nothing of
// another stream run until it ends.  A small kernel of another stream waits up to
// the whole solve (2000 iterations of P2 250k rows: 42 ms, 0.05 ms beside the
// launched ones).  Two threads solving at once: P2 250k rows, 100 iterations each,
// 4.65 ms a pair (6.58 as launches), P1 36k 1.40 (2.24), P1 9k, whose grids fit
// side by side, 0.74 (1.95).
//
// The kernels are launched cooperatively (all blocks resident), so a poll
// ends; a bound on the polls turns a fault elsewhere into an error status
// instead of a hang.
#pragma once
#include "common.cuh"
#include "solve.h"

namespace phgb {

constexpr int kCoopThreads = 1024;   // one block an SM: 64 registers a thread
constexpr int kCoopWarps = kCoopThreads / 32;
constexpr int kCoopMaxBlocks = 160;  // of the solvers with a block an SM
constexpr int kCoopMostBlocks = 320; // of any grid
constexpr int kCoopSums = 3;         // sums exchanged at once, at most
// Doubles of exchange memory, zero before the launch: two buffers of partials
// (a block may be writing the next sum while another still reads the last),
// then two 32-bit words, the arrivals and the give-up flag.
constexpr int kCoopDoubles = 2 * kCoopSums * kCoopMostBlocks + 1;
// Polls before a wait gives up (each is an L2 round trip, about half a
// microsecond: some ten seconds).
constexpr int kCoopPolls = 1 << 24;

struct CoopShared {
    double part[kCoopSums][kCoopWarps];
    int failed;
};

// MAXB: blocks of the grid at most (MAXB / 32 partials a lane of the adding warp).
template <int MAXB = kCoopMaxBlocks>
struct CoopGrid {
    double *mem;        // kCoopDoubles
    CoopShared *sh;
    unsigned epoch;

    __device__ __forceinline__ CoopGrid(double *m, CoopShared *s) : mem(m), sh(s), epoch(0) {}

    // Barrier: every write of the grid before it is visible after it.
    // False (in every thread of the block) when the wait gave up.
    __device__ __forceinline__ bool sync() {
        epoch++;
        __syncthreads();
        if (gridDim.x == 1) return true;
        if (threadIdx.x == 0) sh->failed = arrive_wait() ? 0 : 1;
        __syncthreads();
        return sh->failed == 0;
    }

    // Barrier that sums v[0..K) over the grid and calls fin(totals) in lane 0
    // of warp 0 of every block; what it leaves in shared memory is visible to
    // the block when sum returns.  The other warps call over(thread, threads)
    // meanwhile.
    template <int K, class Fin, class Over>
    __device__ __forceinline__ bool sum(double (&v)[K], Fin fin, Over over) {
        epoch++;
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
        for (int k = 0; k < K; k++) {
            v[k] = warp_sum(v[k]);
            if (lane == 0) sh->part[k][w] = v[k];
        }
        __syncthreads();
        if (w == 0) {
            double t[K];
#pragma unroll
            for (int k = 0; k < K; k++) t[k] = warp_sum(sh->part[k][lane]);
            int ok = 1;
            if (gridDim.x > 1) {
                double *P = mem + (epoch & 1u) * (kCoopSums * MAXB);   // [sum][block]
                if (lane == 0) {
#pragma unroll
                    for (int k = 0; k < K; k++) P[k * MAXB + blockIdx.x] = t[k];
                    ok = arrive_wait() ? 1 : 0;
                }
                __syncwarp();   // the lanes' loads below come after lane 0's acquire
                double a[K][MAXB / 32];
#pragma unroll
                for (int k = 0; k < K; k++)
#pragma unroll
                    for (int j = 0; j < MAXB / 32; j++) {
                        const unsigned b = lane + 32 * j;
                        a[k][j] = b < gridDim.x ? fetch(&P[k * MAXB + b]) : 0.0;
                    }
#pragma unroll
                for (int k = 0; k < K; k++) {
                    t[k] = a[k][0];
#pragma unroll
                    for (int j = 1; j < MAXB / 32; j++) t[k] += a[k][j];
                    t[k] = warp_sum(t[k]);
                }
            }
            if (lane == 0) {
                sh->failed = !ok;
                fin(t);
            }
        } else {
            over((int)threadIdx.x - 32, kCoopThreads - 32);
        }
        __syncthreads();
        return sh->failed == 0;
    }
    template <int K, class Fin>
    __device__ __forceinline__ bool sum(double (&v)[K], Fin fin) {
        return sum(v, fin, [](int, int) {});
    }

private:
    // One thread of the block: arrive and wait for every block.  False when
    // the wait gave up here or elsewhere.
    __device__ __forceinline__ bool arrive_wait() const {
        unsigned *bar = reinterpret_cast<unsigned *>(mem + kCoopDoubles - 1);
        const unsigned target = epoch * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        for (int i = 0; i < kCoopPolls; i++) {
            unsigned c;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(bar) : "memory");
            if ((int)(c - target) >= 0) return true;
            if ((i & 1023) == 1023 && *reinterpret_cast<volatile unsigned *>(bar + 1) != 0) break;
        }
        atomicExch(bar + 1, 1u);
        return false;
    }

    // A load of another block's word that stays where it is written (__ldcg
    // is an asm statement the compiler may move above the wait before it).
    static __device__ __forceinline__ double fetch(const double *p) {
        double v;
        asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
        return v;
    }
};

}  // namespace phgb
