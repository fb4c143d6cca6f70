// The V-cycle's small levels as one launch: down, the coarsest solve and back up, in the shared
// memory of one thread-block cluster.
//
// From about 32^3 cells down a pass of a level is far less work than a launch costs, and most of
// a V-cycle's passes are on these levels. Here the levels ls .. L-1 run in one launch:
//   * the first one, when it is above CL_LOCAL_CELLS, is spread over the cluster, CTA r holding planes
//     [r P, r P + P) with one halo plane each side; after each pass a CTA pushes its boundary
//     planes' new values into its neighbours' halos (st.async, whose bytes complete a
//     transaction barrier there), and waits for theirs: the exchange is one one-way trip between
//     two CTAs, where a cluster barrier and a remote load cost two;
//   * the smaller levels and the coarsest solve run in CTA 0 alone, where a pass ends in a
//     __syncthreads; the others wait at the cluster barrier.
// Bound: latency (shared memory, barriers, exchange) of the chain of passes. Measured, one launch
// at clock 1.9 GHz, against the two cluster launches and the one-CTA launch between them that it
// takes the place of: 16^3 and 8^3 levels, Float32, 2 sweeps, 40 coarsest: 47 -> 23 us, of which
// the 160 half-sweeps of the coarsest are 10; 32^3 to 8^3: 67 -> 31 us; 32^3 to 8^3, FP16, 6
// sweeps, 10 coarsest: 85 -> 45 us. A pass of the 16^3 level is 650-800 cycles (its 16 warps'
// loads, about 300, then the chain load - six sums - division - store - barrier); a pass of
// the spread 32^3 level 1000-1100, of which the exchange is about 400 (a cluster barrier with a
// remote load 650-780).
//
// Layout of a level in shared memory: by colour, then planes (halo, P planes, halo), rows (a zero
// row before each plane's rows) and half-rows of H cells with a zero before them: a cell's six
// neighbours are the other colour's values at the offsets ci, ci - 1, +-RS, +-PS from its own
// place (ci the parity of its x), and everything that is not a LIQUID cell of the grid is a zero
// that nothing writes, so no test enters the sums. x, b and r hold the values the level's arrays
// hold (rounded to the storage type) in the arithmetic type. Each colour's LIQUID cells are
// listed once a projection (k_cluster_lists): place, parity, diagonal (a coarse cell's count of open
// faces, 0 .. 6), which neighbours take its value, where its restriction and its prolongation read.
// A thread owns up to CL_U cells of each colour for a whole leg of the V-cycle, their entries,
// right-hand sides and diagonals in registers: a pass is its loads of x, the sums, the store and
// the meeting. (Reading the list, b and the diagonal from shared memory in every pass, cell after
// cell, took 1000 cycles a pass of a 16^3 level.)
//
// Each pass does what the per-level kernel does for the same cell, in the same order (rbgs,
// residual, restriction's 64 terms, prolongation's 8), so the results are bit for bit those of the
// per-level launches and the one-CTA bottom solve.
//
// The exchange holds both ways whatever is wet. A pass's phase of a CTA's barrier takes, besides the
// bytes of the neighbours' listed boundary cells, an arrival from each neighbour, sent when that one
// has come through the pass before: a neighbour is at most one pass ahead, so the two barriers never
// mix passes p and p + 2, and none of its values of pass p + 1 lands before this CTA has read what
// they replace. (By bytes alone a CTA whose neighbours' facing planes are dry waits for nobody.)
// The arrivals are on their way while the pass works, sent by threads of the last warps (thread 0
// sending them before its cells: 64^3 1.8 % slower, 256^3 0.9 %). Projections, us, bytes alone and with
// the arrivals: 64^3 1022-1027 and 1015, 256^3 FP16 1.04 and 1.03 times the speed of the tree before
// k_cluster, the 96^3 rollout 1.32 and 1.30 times.
//
// Every thread of every CTA runs the same cluster barriers; waits on the exchange are bounded
// (the fault flag is set; that CTA waits, arrives and pushes no more, so its neighbours' waits give
// up in turn), and the last barrier keeps a CTA's shared memory alive until no neighbour writes to it.
#pragma once

#include "mpp_tiles.cuh"

namespace mpp {

constexpr int CL_THREADS = 512, CL_MAXLEV = 7, CL_SIZE = 16;
// A level of at most this many cells runs in one CTA: a pass over 16^3 cells takes less there than
// the spread form's exchange alone and its barriers together, and the level above the coarsest (at
// most 1024 cells) always fits.
constexpr int64_t CL_LOCAL_CELLS = 8192;
// The largest level that joins: a pass over 44 x 36 x 28 cells takes 1200-1600 cycles here, a launch
// over the whole GPU 2.1-2.6 us; above about 64 x 32 x 32 the planes do not fit the CTAs' shared
// memory in Float32.
constexpr int64_t CL_CELLS = 65536;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\n"
        "barrier.cluster.wait.acquire.aligned;\n" ::
            : "memory");
}

struct ClLev {
    int n1, n2, n3;  // the level's cells
    int P;           // planes a CTA holds (local levels: n3)
    int RS, PS, CS;  // strides of a row, a plane and a colour, in elements
    int cap;         // places in a colour's list
    unsigned ox, ob, orr, oent;  // byte offsets in shared memory
    int full;        // a level of the bottom solve: values in the arithmetic type, natural order in
                     // global memory, division by the diagonal
    int gent;        // its first list entry in the global lists (a CTA's colours one after the other)
};
// What k_cluster_lists writes and k_cluster reads.
struct ClLists {
    uint2* ent;      // every level's entries
    uint32_t* gidx;  // the top level's cells in its global arrays, in its entries' order
    int4* cnt;       // [level][CTA]: cells of each colour; of each colour that the neighbours push here
    uint4* rb;       // the coarsest's unknowns by colour, RB_HALF places each
    int* nrb;        // and their numbers
    void* share;     // the level's x below the spread one, as CTA 0 holds it
};
template <class M>
struct ClArgs {
    Lev<M> g[CL_MAXLEV];      // the levels above the coarsest
    ClLev s[CL_MAXLEV + 1];   // and the coarsest (x only)
    BotLev cl;                // the coarsest
    ClLists l;
    int nl, nd, nact;         // levels above the coarsest; 1: the first is spread; CTAs that hold planes of it
    int sweeps, coarse;
    unsigned orb, ogi;        // byte offsets of the coarsest's unknowns and of the top level's global places
    int* fault;
    int tries;                // polls of an exchange wait before it gives up
};

// A list entry. x: the place (16 bits), then these bits and the diagonal; y: where prolongation
// reads the coarse level (its lower corner's place, 16 bits) and where the restriction into the
// cell reads the finer one (16 bits).
constexpr uint32_t CL_CI = 1u << 16, CL_LO = 1u << 17, CL_HI = 1u << 18;  // x odd; pushed to the CTA before, after
constexpr uint32_t CL_CJ = 1u << 19, CL_CK = 1u << 20;                    // y, z odd
constexpr uint32_t CL_P0 = 1u << 21, CL_DH = 1u << 22;  // the lower corner's colour; its x + 1 in the next place
constexpr int CL_DG = 24;                               // the diagonal's shift (3 bits)
constexpr uint32_t CL_NONE = 1u << 31;                  // a thread's place in no list: reads zeros' neighbours, writes nothing

extern __shared__ __align__(128) unsigned char cl_sm[];
template <class T>
__device__ __forceinline__ T* cl_ptr(unsigned off) {
    return reinterpret_cast<T*>(cl_sm + off);
}
__device__ __forceinline__ uint32_t cl_mapa(const void* p, int r) {
    uint32_t o;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(smem_u32(p)), "r"(r));
    return o;
}
// B bytes (4 or 8) from global to shared memory, asynchronously
template <int B>
__device__ __forceinline__ void cl_fetch(void* sm, const void* gm) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(sm)), "l"(gm), "n"(B) : "memory");
}
// v into another CTA's shared memory, its bytes completing a transaction of the barrier there
__device__ __forceinline__ void cl_push(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
                 "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cl_push(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
// an arrival at another CTA's barrier
__device__ __forceinline__ void cl_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cl_store(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(__float_as_uint(v)) : "memory");
}
__device__ __forceinline__ void cl_store(uint32_t addr, double v) {
    asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(addr), "l"(__double_as_longlong(v)) : "memory");
}
__host__ __device__ __forceinline__ int cl_place(const ClLev& S, int kk, int j, int h) {  // kk: 1 for the first plane held
    return kk * S.PS + (j + 1) * S.RS + h + 1;
}

// ---- the lists: once a projection, after the coarse levels are built ----
template <class Pr>
__global__ void __launch_bounds__(CL_THREADS) k_cluster_lists(const __grid_constant__ ClArgs<typename Pr::M> a) {
    using CC = typename Pr::CC;
    __shared__ int cnt[CL_MAXLEV][4];
    const int tid = (int)threadIdx.x, lane = tid & 31, me = (int)blockIdx.x;
    pdl_wait();
    pdl_trigger();
    if (tid < 4 * CL_MAXLEV) (&cnt[0][0])[tid] = 0;
    __syncthreads();
    for (int q = 0; q < a.nl; q++) {
        const bool spread = q < a.nd;
        if (!spread && me > 0) continue;
        const ClLev &S = a.s[q], &D = a.s[q + 1];
        const auto& G = a.g[q];
        const int kb = spread ? me * S.P : 0, left = S.n3 - kb, np = left < 0 ? 0 : (left < S.P ? left : S.P);
        const int n = np * S.n2 * S.n1, H = S.n1 >> 1;
        const int64_t g0 = (int64_t)kb * S.n1 * S.n2;
        const bool lo = spread && me > 0, hi = spread && me + 1 < a.nact;
        uint2* ent = a.l.ent + S.gent + (spread ? (int64_t)me * 2 * S.cap : 0);
        for (int e0 = 0; e0 < n; e0 += CL_THREADS) {
            const int e = e0 + tid, row = e / S.n1, p = e - row * S.n1, kk = row / S.n2, j = row - kk * S.n2, k = kb + kk;
            bool on = false;
            int c = 0, i = p, d = 0;
            if (e < n) {
                on = (G.code[g0 + e] & SELF) != 0;
                d = S.full ? (int)G.dc[g0 + e] : (int)ld<float>(G.dg + g0 + e);
            }
            if (S.full) {
                c = (i + j + k + 1) & 1;
            } else {
                c = p >= H ? 1 : 0;
                i = 2 * (p - c * H) + ((c + j + k + 1) & 1);
            }
            // prolongation's lower corner: coarse cell (A, B, K)
            const int ci = i & 1, cj = j & 1, ck = k & 1, A = (i >> 1) - 1 + ci, B = (j >> 1) - 1 + cj, K = (k >> 1) - 1 + ck;
            uint2 w;
            w.x = (uint32_t)cl_place(S, kk + 1, j, i >> 1) | (ci ? CL_CI : 0u) | (cj ? CL_CJ : 0u) | (ck ? CL_CK : 0u) |
                  ((lo && kk == 0) ? CL_LO : 0u) | ((hi && kk + 1 == np) ? CL_HI : 0u) |
                  (((A + B + K + 1) & 1) ? CL_P0 : 0u) | ((A & 1) ? CL_DH : 0u) | ((uint32_t)d << CL_DG);
            w.y = (uint32_t)cl_place(D, K + 1, B, A >> 1);
            if (q > 0) w.y |= (uint32_t)(2 * k * a.s[q - 1].PS + 2 * j * a.s[q - 1].RS + i + 1) << 16;
#pragma unroll
            for (int cc = 0; cc < 2; cc++) {
                const unsigned m = __ballot_sync(0xffffffffu, on && c == cc);
                if (m == 0) continue;
                int base = 0;
                if (lane == 0) base = atomicAdd(&cnt[q][cc], __popc(m));
                base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1u));
                if (on && c == cc) {
                    ent[cc * S.cap + base] = w;
                    if (q == 0) a.l.gidx[(spread ? (int64_t)me * 2 * S.cap : 0) + cc * S.cap + base] = (uint32_t)(g0 + e);
                }
            }
        }
        // what the neighbours push: their boundary planes' listed cells
        const int pl = S.n1 * S.n2;
        for (int side = 0; side < 2; side++) {
            if (np == 0 || (side == 0 ? !lo : !hi)) continue;
            const uint8_t* code = G.code + g0 + (side == 0 ? -pl : np * pl);
            for (int e0 = 0; e0 < pl; e0 += CL_THREADS) {
                const int e = e0 + tid;
                const bool on = e < pl && (code[e] & SELF) != 0;
                const int c = (e % S.n1) >= H ? 1 : 0;
                const unsigned m0 = __ballot_sync(0xffffffffu, on && c == 0), m1 = __ballot_sync(0xffffffffu, on && c == 1);
                if (lane == 0) {
                    if (m0) atomicAdd(&cnt[q][2], __popc(m0));
                    if (m1) atomicAdd(&cnt[q][3], __popc(m1));
                }
            }
        }
    }
    __syncthreads();
    if (tid < a.nl) a.l.cnt[tid * CL_SIZE + me] = make_int4(cnt[tid][0], cnt[tid][1], cnt[tid][2], cnt[tid][3]);
    if (me > 0) return;
    // the coarsest: each colour's unknowns with their neighbours' places, diagonal, restriction
    // base and place in the level's x
    __shared__ RbShared<CC> rb;
    const BotLev& B = a.cl;
    const ClLev &F = a.s[a.nl - 1], &D = a.s[a.nl];
    coarsest_lists<Pr>(B, rb);
    const int step6[6] = {1, -1, B.n1, -B.n1, B.n1 * B.n2, -B.n1 * B.n2};
    for (int u = 0; u < 2; u++) {
        if (tid >= rb.cnt[u][32]) continue;
        const int c = rb.cell[u][tid], i = c % B.n1, j = (c / B.n1) % B.n2, k = c / (B.n1 * B.n2);
        const uint8_t cd = B.code[c];
        uint32_t nb[6];
#pragma unroll
        for (int m = 0; m < 6; m++) nb[m] = (cd & (1u << m)) ? rb.place[c + step6[m]] : (uint32_t)RB_CELLS;
        // (level nl - 1 is CTA 0's own, or a spread level above the coarsest does not exist)
        const uint32_t rbase = (uint32_t)(2 * k * F.PS + 2 * j * F.RS + i + 1);
        const uint32_t yp = (uint32_t)(((i + j + k + 1) & 1) * D.CS + cl_place(D, k + 1, j, i >> 1));
        a.l.rb[u * RB_HALF + tid] = make_uint4(nb[0] | (nb[1] << 11) | ((uint32_t)B.dc[c] << 22), nb[2] | (nb[3] << 11),
                                               nb[4] | (nb[5] << 11), rbase | (yp << 16));
    }
    if (tid < 2) a.l.nrb[tid] = rb.cnt[tid][32];
}

// A diagonal and its reciprocal.
template <class C>
struct alignas(2 * sizeof(C)) ClDiag {
    C d, rd;
};
template <class C>
struct ClShared {
    unsigned long long bar[2];  // the exchange: passes take them in turn
    int4 cnt[CL_MAXLEV];        // listed cells of each colour; cells of each colour that the neighbours push here
    ClDiag<C> dg[2][8];         // a diagonal 0 .. 6 with its reciprocal, [0] as it is stored, [1] not rounded
    int nrb[2];                 // the coarsest's unknowns of each colour
    int dead;                   // an exchange wait gave up
};

// A thread's cells of a level: CL_U of each colour at a time.
constexpr int CL_U = 4;
template <class C>
struct ClCells {
    uint32_t e[2][CL_U];
    C b[2][CL_U];
};

template <class Pr>
struct ClRun {
    using C = typename Pr::C;
    using M = typename Pr::M;
    const ClArgs<M>& a;
    ClShared<C>& sh;
    int me;
    int ph;    // exchanges so far
    bool off;  // an exchange wait of this CTA gave up
    // the level at work
    int q, full, RS, PS, CS, n[2], in[2];
    bool spread, one;      // one: a thread's cells are all in its registers
    C *X, *B, *R;
    const uint2* ent;
    int cap;
    uint32_t far[2], bars[2];  // the CTAs before and after: x shifted onto their halo, the exchange barriers
    unsigned xr;               // from x to r
    const ClDiag<C>* dg;
    ClCells<C> cl;

    __device__ static __forceinline__ C rnd(C v, int full) {
        if (full) return v;
        M m;
        st(&m, v);
        return ld<C>(&m);
    }

    // Level q's constants and this thread's cells. top_b: b comes from the level's global array.
    __device__ __forceinline__ void enter(int q_) {
        q = q_;
        const ClLev& S = a.s[q];
        full = S.full;
        RS = S.RS;
        PS = S.PS;
        CS = S.CS;
        cap = S.cap;
        spread = q < a.nd;
        X = cl_ptr<C>(S.ox);
        B = cl_ptr<C>(S.ob);
        R = cl_ptr<C>(S.orr);
        ent = cl_ptr<uint2>(S.oent);
        const int4 c = sh.cnt[q];
        n[0] = c.x;
        n[1] = c.y;
        in[0] = c.z;
        in[1] = c.w;
        one = n[0] <= CL_U * CL_THREADS && n[1] <= CL_U * CL_THREADS;
        dg = sh.dg[(Pr::scaled && !full) ? 0 : 1];
        xr = S.orr - S.ox;
        if (spread) {
            const int by = S.P * S.PS * (int)sizeof(C), lo = me > 0 ? me - 1 : me, hi = me + 1 < a.nact ? me + 1 : me;
            far[0] = cl_mapa(X, lo) + (uint32_t)by;
            far[1] = cl_mapa(X, hi) - (uint32_t)by;
            bars[0] = cl_mapa(&sh.bar[0], lo);
            bars[1] = cl_mapa(&sh.bar[0], hi);
        }
    }
    // This thread's cells from base on, NU of each colour (b from shared memory when with_b).
    template <int NU>
    __device__ __forceinline__ void load(int base, bool with_b) {
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int u = 0; u < NU; u++) {
                const int t = base + u * CL_THREADS + (int)threadIdx.x;
                const uint32_t e = t < n[c] ? ent[c * cap + t].x : CL_NONE | (uint32_t)(PS + RS + 1);
                cl.e[c][u] = e;
                if (with_b) cl.b[c][u] = B[c * CS + (int)(e & 0xffffu)];
            }
    }

    // ---- the exchange ----
    // the start of a pass in which the neighbours push `cells` values here: this CTA's own arrival, and
    // the one it owes each neighbour (see above)
    __device__ __forceinline__ void expect(int cells) {
        if (!spread || off) return;
        const uint32_t b = 8u * (uint32_t)(ph & 1);
        if (threadIdx.x == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&sh.bar[ph & 1])),
                         "r"(cells * (int)sizeof(C))
                         : "memory");
        // (the last warps: theirs are the fewest cells)
        if (threadIdx.x == CL_THREADS - 32 && me > 0) cl_arrive(bars[0] + b);
        if (threadIdx.x == CL_THREADS - 64 && me + 1 < a.nact) cl_arrive(bars[1] + b);
    }
    // a listed cell's value to the neighbours that hold it in their halos (r: its residual, else x)
    __device__ __forceinline__ void push(uint32_t e, bool r, int idx, C v) const {
        if (!spread || off || !(e & (CL_LO | CL_HI))) return;
        const uint32_t at = (uint32_t)(idx * (int)sizeof(C)) + (r ? xr : 0u), b = 8u * (uint32_t)(ph & 1);
        if (e & CL_LO) cl_push(far[0] + at, v, bars[0] + b);
        if (e & CL_HI) cl_push(far[1] + at, v, bars[1] + b);
    }
    // the end of a pass
    __device__ __forceinline__ void meet() {
        __syncthreads();
        if (!spread) return;
        const uint32_t bar = smem_u32(&sh.bar[ph & 1]);
        const unsigned par = (unsigned)(ph >> 1) & 1u;
        ph++;
        if (*(volatile int*)&sh.dead) {
            off = true;
            return;
        }
        unsigned done = 0;
        for (int tries = 0; !done && tries < a.tries; tries++)
            asm volatile(
                "{\n.reg .pred p;\n"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                "selp.u32 %0, 1, 0, p;\n}\n"
                : "=r"(done)
                : "r"(bar), "r"(par)
                : "memory");
        if (!done) {
            off = true;
            *(volatile int*)&sh.dead = 1;
            *a.fault = FAULT_CLUSTER;
        }
    }

    // ---- passes ----
    __device__ __forceinline__ C divide(C v, uint32_t e) const {  // by the cell's diagonal, as the level does
        const ClDiag<C> g = dg[(e >> CL_DG) & 7u];
        if (Pr::scaled && !full) return v * g.rd;
        if constexpr (std::is_same<C, float>::value) return div_small(v, g.d, g.rd);  // (d = 0: rd = 0 gives 0)
        else return g.d > (C)0 ? v / g.d : (C)0;
    }
    // f(): one pass over NU cells of each colour a thread at a time (which are in its registers
    // already when they are all).
    template <int NU, class F>
    __device__ __forceinline__ void chunks(F&& f) {
        if (NU < CL_U || one) {
            f();
        } else {
            const int m = n[0] > n[1] ? n[0] : n[1];
#pragma unroll 1
            for (int base = 0; base < m; base += CL_U * CL_THREADS) {
                load<NU>(base, true);
                f();
            }
        }
    }
    // start_kernel! (src/flip.jl:965-973): the first colour's first sweep from x = 0
    template <int NU>
    __device__ __forceinline__ void start() {
        expect(in[0]);
        chunks<NU>([&]() {
#pragma unroll
            for (int u = 0; u < NU; u++) {
                const uint32_t e = cl.e[0][u];
                const C v = rnd(divide(cl.b[0][u], e), full);
                if (e & CL_NONE) continue;
                X[e & 0xffffu] = v;
                push(e, false, (int)(e & 0xffffu), v);
            }
        });
        meet();
    }
    // liquidsum (src/flip.jl:852-857) around the places of this thread's cells of colour c
    template <int c, int NU>
    __device__ __forceinline__ void around(C (&s)[NU]) const {
        C v[NU][6];
#pragma unroll
        for (int u = 0; u < NU; u++) {
            const uint32_t e = cl.e[c][u];
            const C *o = X + (1 - c) * CS + (int)(e & 0xffffu), *ox = o + ((e & CL_CI) ? 1 : 0);
            v[u][0] = ox[0];
            v[u][1] = ox[-1];
            v[u][2] = o[RS];
            v[u][3] = o[-RS];
            v[u][4] = o[PS];
            v[u][5] = o[-PS];
        }
#pragma unroll
        for (int u = 0; u < NU; u++) s[u] = ((((v[u][0] + v[u][1]) + v[u][2]) + v[u][3]) + v[u][4]) + v[u][5];
    }
    // rbgs_kernel! (src/flip.jl:870-877), one colour
    template <int c, int NU>
    __device__ __forceinline__ void rbgs() {
        expect(in[c]);
        chunks<NU>([&]() {
            C s[NU];
            around<c, NU>(s);
#pragma unroll
            for (int u = 0; u < NU; u++) {
                const uint32_t e = cl.e[c][u];
                const C v = rnd(divide(cl.b[c][u] + s[u], e), full);
                const int i = c * CS + (int)(e & 0xffffu);
                if (e & CL_NONE) continue;
                X[i] = v;
                push(e, false, i, v);
            }
        });
        meet();
    }
    // residual_kernel! (src/flip.jl:859-863)
    template <int c, int NU>
    __device__ __forceinline__ void residual_of() {
        C s[NU];
        around<c, NU>(s);
#pragma unroll
        for (int u = 0; u < NU; u++) {
            const uint32_t e = cl.e[c][u];
            const int i = c * CS + (int)(e & 0xffffu);
            const C v = rnd(cl.b[c][u] - (dg[(e >> CL_DG) & 7u].d * X[i] - s[u]), full);
            if (e & CL_NONE) continue;
            R[i] = v;
            push(e, true, i, v);
        }
    }
    template <int NU>
    __device__ __forceinline__ void residual() {
        expect(in[0] + in[1]);
        chunks<NU>([&]() {
            residual_of<0, NU>();
            residual_of<1, NU>();
        });
        meet();
    }
    // restrict_kernel! (src/flip.jl:894-906) of level q's residual, the 64 terms in its order (x
    // fastest); r0: the place of the 4 x 4 x 4 cells' first row. Terms off the grid or off the
    // liquid are zeros. Fine row (jf, kf) holds x = 2I-1 .. 2I+2 at the places I-1, I, I, I+1 of
    // alternating colours, the first one's (jf + kf) & 1, which is (b + c) & 1 for term row (b, c).
    __device__ __forceinline__ C restricted(int r0) const {
        const C *E = R + r0, *O = E + CS;  // where rows of even and odd b start
        C s = (C)0;
#pragma unroll 1
        for (int c3 = 0; c3 < 4; c3++) {
            const C wc = (c3 == 1 || c3 == 2) ? (C)0.375f : (C)0.125f;
            C v[4][4];
#pragma unroll
            for (int b3 = 0; b3 < 4; b3++) {
                const C *A = ((b3 & 1) ? O : E) + b3 * RS, *Bc = ((b3 & 1) ? E : O) + b3 * RS;
                v[b3][0] = A[-1];
                v[b3][1] = Bc[0];
                v[b3][2] = A[0];
                v[b3][3] = Bc[1];
            }
#pragma unroll
            for (int b3 = 0; b3 < 4; b3++)
#pragma unroll
                for (int a3 = 0; a3 < 4; a3++)  // (w_a w_b) w_c: exact dyadic products
                    s = macc<Pr::scaled>(s, wB<C>(a3) * wB<C>(b3) * wc, v[b3][a3]);
            const C* t = E + PS;
            E = O + PS;
            O = t;
        }
        return Pr::scaled ? s : (C)4 * s;
    }
    // into level q + 1, both in this CTA
    __device__ __forceinline__ void restrict_into() {
        const ClLev& S = a.s[q + 1];
        const int4 c = sh.cnt[q + 1];
        const uint2* en = cl_ptr<uint2>(S.oent);
        C* Bn = cl_ptr<C>(S.ob);
        for (int t = (int)threadIdx.x; t < c.x + c.y; t += CL_THREADS) {
            const int col = t >= c.x ? 1 : 0;
            const uint2 e = en[col * S.cap + t - (col ? c.x : 0)];
            Bn[col * S.CS + (int)(e.x & 0xffffu)] = rnd(restricted((int)(e.y >> 16)), S.full);
        }
        __syncthreads();
    }
    // into the next level, in CTA 0, from the spread one: this CTA's share of its planes
    __device__ __forceinline__ void restrict_out(int planes) {
        const ClLev& S = a.s[q + 1];
        const auto& G = a.g[q + 1];
        const int kb = me * a.s[q].P, K0 = kb / 2, m = planes / 2 * S.n2 * S.n1;
        const uint32_t to = cl_mapa(cl_ptr<C>(S.ob), 0);
        for (int t = (int)threadIdx.x; t < m; t += CL_THREADS) {
            const int row = t / S.n1, I = t - row * S.n1, kk = row / S.n2, J = row - kk * S.n2, K = K0 + kk;
            const int c = (I + J + K + 1) & 1;
            const uint8_t cd = S.full ? G.code[G.nat(I, J, K)] : G.code[G.pos(I, J, K)];
            if (!(cd & SELF)) continue;
            const C v = rnd(restricted((2 * K - kb) * PS + 2 * J * RS + I + 1), S.full);
            cl_store(to + (uint32_t)((c * S.CS + cl_place(S, K + 1, J, I >> 1)) * (int)sizeof(C)), v);
        }
    }
    // prolong_kernel! (src/flip.jl:914-929): the eight coarse cells around each of this thread's
    // cells, x fastest; cells off the coarse grid are zeros around it
    // Only the first colour's values are pushed: the pass that follows reads that colour and pushes the
    // other one anew (and two pushes of one place in passes that follow each other have no order).
    __device__ __forceinline__ void prolong() {
        const ClLev& D = a.s[q + 1];
        const C* Y = cl_ptr<C>(D.ox);
        const int dRS = D.RS, dPS = D.PS, dCS = D.CS, m0 = n[0], m = n[0] + n[1];
        expect(in[0]);
        for (int t = (int)threadIdx.x; t < m; t += CL_THREADS) {
            const int c = t >= m0 ? 1 : 0;
            const uint2 w = ent[c * cap + t - (c ? m0 : 0)];
            const uint32_t e = w.x;
            const int i = c * CS + (int)(e & 0xffffu), dh = (e & CL_DH) ? 1 : 0;
            // corners of the lower corner's colour parity, and of the other one
            const C* low = Y + (w.y & 0xffffu);
            const C *E = low + ((e & CL_P0) ? dCS : 0), *O = low + ((e & CL_P0) ? 0 : dCS);
            const C v[8] = {E[0], O[dh], O[dRS], E[dRS + dh], O[dPS], E[dPS + dh], E[dPS + dRS], O[dPS + dRS + dh]};
            const C wa[2] = {(e & CL_CI) ? (C)0.75f : (C)0.25f, (e & CL_CI) ? (C)0.25f : (C)0.75f};
            const C wb[2] = {(e & CL_CJ) ? (C)0.75f : (C)0.25f, (e & CL_CJ) ? (C)0.25f : (C)0.75f};
            const C wc[2] = {(e & CL_CK) ? (C)0.75f : (C)0.25f, (e & CL_CK) ? (C)0.25f : (C)0.75f};
            C s = (C)0;
#pragma unroll
            for (int k = 0; k < 8; k++)
                s = macc<Pr::scaled>(s, wa[k & 1] * wb[(k >> 1) & 1] * wc[k >> 2], rnd(v[k], full));
            const C x = rnd(X[i] + (Pr::scaled ? (C)4 * s : s), full);
            X[i] = x;
            if (c == 0) push(e, false, i, x);
        }
        meet();
    }
    // the V-cycle's legs of the level at work (vcycle!, src/flip.jl:992-1014).
    template <int NU>
    __device__ __forceinline__ void down_n() {
        load<NU>(0, true);
        start<NU>();
        rbgs<1, NU>();
#pragma unroll 1
        for (int i = 1; i < a.sweeps; i++) {
            rbgs<0, NU>();
            rbgs<1, NU>();
        }
        residual<NU>();
    }
    template <int NU>
    __device__ __forceinline__ void sweeps_up() {
        load<NU>(0, true);
#pragma unroll 1
        for (int i = 0; i < a.sweeps; i++) {
            rbgs<1, NU>();
            rbgs<0, NU>();
        }
    }
    __device__ __forceinline__ void down() {
        const int m = n[0] > n[1] ? n[0] : n[1];
        if (m <= CL_THREADS) down_n<1>();
        else if (m <= 2 * CL_THREADS) down_n<2>();
        else down_n<CL_U>();
    }
    __device__ __forceinline__ void up() {
        prolong();
        const int m = n[0] > n[1] ? n[0] : n[1];
        if (m <= CL_THREADS) sweeps_up<1>();
        else if (m <= 2 * CL_THREADS) sweeps_up<2>();
        else sweeps_up<CL_U>();
    }
};

template <class Pr>
__device__ __forceinline__ void cluster_dev(const ClArgs<typename Pr::M>& a) {
    using C = typename Pr::C;
    using CC = typename Pr::CC;
    using M = typename Pr::M;
    __shared__ ClShared<C> sh;
    __shared__ CC rbx[RB_CELLS + 2];  // the coarsest's x by colour, a zero, a place for threads without a cell
    const int tid = (int)threadIdx.x;
    ClRun<Pr> r{a, sh, (int)blockIdx.x, 0, false};
    const bool spread = a.nd > 0, first = r.me == 0;
    const int kb = spread ? r.me * a.s[0].P : 0, left = a.s[0].n3 - kb;
    const int np = left < 0 ? 0 : (left < a.s[0].P ? left : a.s[0].P);  // planes of the top level
    const bool holds = spread ? np > 0 : first;
    // Before the programmatic-dependent-launch wait: zeros, lists and constants, which the operator
    // alone decides. The preceding kernel writes only the top level's b.
    if (tid < a.nl) sh.cnt[tid] = a.l.cnt[tid * CL_SIZE + (tid < a.nd ? r.me : 0)];
    if (tid < 2) sh.nrb[tid] = a.l.nrb[tid];
    if (tid < 8) {
        M m;
        st(&m, tid ? 1.f / (float)tid : 0.f);
        sh.dg[0][tid] = ClDiag<C>{(C)tid, ld<C>(&m)};
        sh.dg[1][tid] = ClDiag<C>{(C)tid, tid ? (C)1 / (C)tid : (C)0};
    }
    if (tid == 0) {
        sh.dead = 0;
        const int arrivals = 1 + (r.me > 0 ? 1 : 0) + (r.me + 1 < a.nact ? 1 : 0);  // its own, its neighbours'
        for (int i = 0; i < 2; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&sh.bar[i])), "r"(arrivals) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // (every copy in flight at once: one latency for the lot)
    uint32_t* gi = cl_ptr<uint32_t>(a.ogi);  // the top level's cells in its global arrays
    for (int q = 0; q < a.nl; q++) {
        if (q >= a.nd && !first) break;
        const ClLev& S = a.s[q];
        const int64_t mine = q < a.nd ? (int64_t)r.me * 2 * S.cap : 0;
        const uint2* g = a.l.ent + S.gent + mine;
        uint2* en = cl_ptr<uint2>(S.oent);
        const int4 c = sh.cnt[q];
#pragma unroll
        for (int cc = 0; cc < 2; cc++)
            for (int t = tid; t < (cc ? c.y : c.x); t += CL_THREADS) {
                cl_fetch<8>(en + cc * S.cap + t, g + cc * S.cap + t);
                if (q == 0) cl_fetch<4>(gi + cc * S.cap + t, a.l.gidx + mine + cc * S.cap + t);
            }
    }
    // the coarsest's unknowns, a thread one of each colour
    const int nrb0 = first ? sh.nrb[0] : 0, nrb1 = first ? sh.nrb[1] : 0;
    uint4* rbe = cl_ptr<uint4>(a.orb);
    if (tid < nrb0) cp_async16(rbe + tid, a.l.rb + tid);
    if (tid < nrb1) cp_async16(rbe + RB_HALF + tid, a.l.rb + RB_HALF + tid);
    cp_async_commit();
    // zeros while they fly (the levels in CTA 0 alone: only x elsewhere, of the one prolongation reads)
    auto zero = [&](unsigned off, int elems) {
        uint4* z = cl_ptr<uint4>(off);
        for (int u = tid; u < (int)((elems * sizeof(C) + 15) / 16); u += CL_THREADS) z[u] = make_uint4(0, 0, 0, 0);
    };
    for (int q = 0; q <= a.nl; q++) {
        if (q <= a.nd || first) zero(a.s[q].ox, 2 * a.s[q].CS);
        if (q < a.nl && (q < a.nd || first)) zero(a.s[q].orr, 2 * a.s[q].CS);
    }
    for (int p = tid; p < RB_CELLS + 2; p += CL_THREADS) rbx[p] = (CC)0;
    cp_async_wait<0>();
    __syncthreads();
    if (spread) cluster_barrier();  // every CTA's barriers and zeros are ready for its neighbours
    if (holds) r.enter(0);
    pdl_wait();
    pdl_trigger();
    if (holds) {  // the top level's right-hand side
        const M* gb = a.g[0].b;
#pragma unroll
        for (int c = 0; c < 2; c++) {
            for (int t0 = tid; t0 < r.n[c]; t0 += CL_U * CL_THREADS) {
                M v[CL_U];
#pragma unroll
                for (int u = 0; u < CL_U; u++)
                    if (t0 + u * CL_THREADS < r.n[c]) v[u] = gb[gi[c * r.cap + t0 + u * CL_THREADS]];
#pragma unroll
                for (int u = 0; u < CL_U; u++)
                    if (t0 + u * CL_THREADS < r.n[c])
                        r.B[c * r.CS + (int)(r.ent[c * r.cap + t0 + u * CL_THREADS].x & 0xffffu)] = ld<C>(&v[u]);
            }
        }
        __syncthreads();
    }
    // down
#pragma unroll 1
    for (int q = 0; q < a.nl; q++) {
        if (spread && q == 1) cluster_barrier();  // level 1's right-hand side is in CTA 0
        if (q < a.nd ? !holds : !first) continue;
        if (q > 0) r.enter(q);
        r.down();
        if (spread && q == 0) r.restrict_out(np);
        else if (q + 1 < a.nl) r.restrict_into();
    }
    // coarse_kernel! (src/flip.jl:935-962), the right-hand side restricted into registers
    if (first) {
        int own[2], nb[2][6], yp[2];
        CC bi[2], d[2], rd[2];
        const int n = nrb0 > nrb1 ? nrb0 : nrb1, nt = (n + 31) & ~31;
#pragma unroll
        for (int u = 0; u < 2; u++) {  // a thread without a cell solves 0 = 0 in the place after the zero
            const bool is = tid < (u ? nrb1 : nrb0);
            const uint4 w = is ? rbe[u * RB_HALF + tid]
                               : make_uint4(RB_CELLS | (RB_CELLS << 11) | (1u << 22), RB_CELLS | (RB_CELLS << 11),
                                            RB_CELLS | (RB_CELLS << 11), 0u);
            own[u] = is ? u * RB_HALF + tid : RB_CELLS + 1;
            nb[u][0] = (int)(w.x & 2047u);
            nb[u][1] = (int)((w.x >> 11) & 2047u);
            nb[u][2] = (int)(w.y & 2047u);
            nb[u][3] = (int)((w.y >> 11) & 2047u);
            nb[u][4] = (int)(w.z & 2047u);
            nb[u][5] = (int)((w.z >> 11) & 2047u);
            d[u] = (CC)(int)(w.x >> 22);
            rd[u] = (CC)1 / d[u];
            bi[u] = is ? (CC)r.restricted((int)(w.w & 0xffffu)) : (CC)0;
            yp[u] = (int)(w.w >> 16);
        }
        if (tid < nt) {
            rb_sweeps(nt, a.coarse, [&](auto uc) {
                constexpr int u = decltype(uc)::value;
                CC v[6];
#pragma unroll
                for (int m = 0; m < 6; m++) v[m] = rbx[nb[u][m]];
                CC acc = bi[u];
#pragma unroll
                for (int m = 0; m < 6; m++) acc += v[m];
                if constexpr (std::is_same<CC, float>::value) rbx[own[u]] = div_small(acc, d[u], rd[u]);
                else rbx[own[u]] = acc * rd[u];  // FP64 coarsest of the 16-bit forms
            });
            C* Y = cl_ptr<C>(a.s[a.nl].ox);
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (own[u] <= RB_CELLS) Y[yp[u]] = (C)rbx[own[u]];
        }
        __syncthreads();
    }
    // up
#pragma unroll 1
    for (int q = a.nl - 1; q >= 0; q--) {
        if (spread && q == 0) {
            if (first) {  // level 1's x as it lies here, for the other CTAs
                const uint4* x = reinterpret_cast<const uint4*>(r.X);
                for (int u = tid; u < (int)((2 * r.CS * sizeof(C) + 15) / 16); u += CL_THREADS)
                    static_cast<uint4*>(a.l.share)[u] = x[u];
            }
            cluster_barrier();
            if (holds && !first) {  // the planes that this CTA's cells read, at their places
                const ClLev& D = a.s[1];
                const int k0 = kb / 2, m = (np / 2 + 2) * D.PS + D.RS;
                const C* x = static_cast<const C*>(a.l.share);
                C* Y = cl_ptr<C>(D.ox);
                for (int t = tid; t < 2 * m; t += CL_THREADS) {
                    const int c = t >= m ? 1 : 0, o = k0 * D.PS + t - c * m;
                    if (o < D.CS) Y[c * D.CS + o] = __ldcg(x + c * D.CS + o);
                }
                __syncthreads();
            }
        }
        if (q < a.nd ? !holds : !first) continue;
        r.enter(q);
        r.up();
    }
    if (holds) {
        const Lev<M>& G = a.g[0];
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll 4
            for (int t = tid; t < r.n[c]; t += CL_THREADS)
                st(G.x + gi[c * r.cap + t], r.X[c * r.CS + (int)(r.ent[c * r.cap + t].x & 0xffffu)]);
    }
    if (spread) {
        cluster_barrier();  // (a CTA leaves when no neighbour pushes to it any more)
        if (*(volatile int*)&sh.dead)  // what it did not wait for may still be on its way
            for (int i = 0; i < 64; i++) __nanosleep(1000);
    }
}
template <class Pr>
__global__ void __launch_bounds__(CL_THREADS, 1) k_cluster(const __grid_constant__ ClArgs<typename Pr::M> a) {
    cluster_dev<Pr>(a);
}

}  // namespace mpp
