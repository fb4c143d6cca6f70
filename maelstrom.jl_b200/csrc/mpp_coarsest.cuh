// The coarsest level's red-black Gauss-Seidel in one CTA (coarse_kernel!, src/flip.jl:935-962;
// the sparse hierarchy's coarsest_kernel!, src/sflip.jl:1627-1660): up to 1024 cells, 2 * sweeps
// sweeps of two half-sweeps each, every half-sweep reading what the one before it wrote.
//
// Bound: the latency of one half-sweep (shared-memory store -> barrier -> loads -> six ordered
// sums -> division -> store), times 4 * sweeps of them; there is nothing to overlap it with. So
// everything that does not change between half-sweeps is in registers: a thread owns the t-th
// unknown of each colour, with its right-hand side, its (reciprocal) diagonal and its six
// neighbours' places in shared memory. The unknowns are stored colour by colour in list order
// (cells that are none take no thread and no place), so a warp's stores and most of its loads
// are consecutive words, and a neighbour that is no unknown is the place of a zero: no test is
// left in the loop. Division is div_small / div_rn. Only the warps that own an unknown meet at
// the barrier. An 8^3 level, 160 half-sweeps in Float32: 330 -> 122 cycles each.
#pragma once

#include "mpp_common.cuh"
#include "mpp_div.cuh"

namespace mpp {

constexpr int RB_CELLS = 1024, RB_HALF = RB_CELLS / 2;

// Shared memory of the solve: x by colour (RB_HALF places each, then a zero and a spare place), each cell's place
// and the lists of each colour's cells.
template <class CC>
struct RbShared {
    CC x[RB_CELLS + 2];
    uint16_t place[RB_CELLS], cell[2][RB_HALF];
    int cnt[2][33];
};

// The lists. on(c): whether cell c (< N) is an unknown; col(c): its colour. A block of whole warps,
// 512 threads or more for N above 512; all threads call; three barriers. Returns the threads that
// own an unknown, rounded up to whole warps.
template <class CC, class On, class Col>
__device__ __forceinline__ int rb_lists(RbShared<CC>& sh, int N, On&& on, Col&& col) {
    const int tid = (int)threadIdx.x, T = (int)blockDim.x, lane = tid & 31, w = tid >> 5, nw = T >> 5;
    bool o[2];
    int cl[2];
    unsigned m[2][2];
#pragma unroll
    for (int u = 0; u < 2; u++) {  // cells tid and tid + T (none when T covers the level)
        const int c = tid + u * T;
        o[u] = c < N && c < RB_CELLS && on(c);
        cl[u] = o[u] ? col(c) : 0;
#pragma unroll
        for (int q = 0; q < 2; q++) m[u][q] = __ballot_sync(0xffffffffu, o[u] && cl[u] == q);
        if (lane == 0 && u * nw + w < 32) {
            sh.cnt[0][u * nw + w] = __popc(m[u][0]);
            sh.cnt[1][u * nw + w] = __popc(m[u][1]);
        }
    }
    for (int p = tid; p <= RB_CELLS; p += T) sh.x[p] = (CC)0;
    __syncthreads();
    if (w < 2) {  // warp w: exclusive prefix of colour w's counts
        const int v = lane < 2 * nw ? sh.cnt[w][lane] : 0;
        int s = v;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, s, k);
            if (lane >= k) s += x;
        }
        sh.cnt[w][lane] = s - v;
        if (lane == 31) sh.cnt[w][32] = s;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int c = tid + u * T;
        if (c >= N || c >= RB_CELLS) continue;
        const int pos = o[u] ? sh.cnt[cl[u]][u * nw + w] + __popc(m[u][cl[u]] & ((1u << lane) - 1u)) : 0;
        sh.place[c] = o[u] ? (uint16_t)(cl[u] * RB_HALF + pos) : (uint16_t)RB_CELLS;
        if (o[u]) sh.cell[cl[u]][pos] = (uint16_t)c;
    }
    __syncthreads();
    const int n0 = sh.cnt[0][32], n1 = sh.cnt[1][32], n = n0 > n1 ? n0 : n1;
    return (n + 31) & ~31;
}

// `sweeps` sweeps in colour order 0, 1 and `sweeps` in order 1, 0, each half-sweep step(u, x) for
// this thread's unknown of colour u; a barrier after each for the first `nt` threads, which are
// the callers.
template <class Step>
__device__ __forceinline__ void rb_sweeps(int nt, int sweeps, Step&& step) {
    auto meet = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory"); };
#pragma unroll 1
    for (int s = 0; s < sweeps; s++) {
        step(std::integral_constant<int, 0>{});
        meet();
        step(std::integral_constant<int, 1>{});
        meet();
    }
#pragma unroll 1
    for (int s = 0; s < sweeps; s++) {
        step(std::integral_constant<int, 1>{});
        meet();
        step(std::integral_constant<int, 0>{});
        meet();
    }
}

}  // namespace mpp
