// The level-set passes step! runs before the projection (sm_100a): redistance! (Jacobi
// sweeps of reinit_kernel!), classify! (fused into the last sweep) and filltrapped! (the
// trapped-air fill), src/flip.jl:608-760.
//
// Redistancing: a thread takes 4 consecutive cells of a row (16-byte loads of the row and
// of the rows at -+y and -+z, one element each side for -+x). The arithmetic is the
// reference's, in its order, with Julia's min/max (the sign of a zero counts) and clamp;
// the library is built without FMA contraction, so every cell is bit-identical to the
// reference's Float32 code. The last sweep also writes the cell classes (classify!).
// A sweep is bound by its instructions, not by its 8 bytes a cell, so the common cells
// take few: the wall test of issolidcell is a range of open cells a row (Walls), four
// cells with no wall beside them take a minimum and a maximum of their neighbours each
// (which decide whether the surface passes, and whether the distance is beyond phimax), and
// only a cell near the surface goes through Godunov's update. 256^3, a sweep: 138 us with
// the Float32 wall geometry of seven cells and Julia's min on every pair, 61 here.
//
// Trapped air: the reference reaches air from the grid's top layer by rounds of sweeps of
// one thread per line along z, x and y, until a round reaches nothing (a host read per
// round). A sweep fills every run of air along a line that holds a reached cell (a walk
// there and back with a carry). Here the AIR cells and the reached cells are bit masks,
// 32 cells of a row per word: a sweep along x is a carry through the words of a row with
// a 5-step shift-and-mask fill inside each word; a sweep along y or z moves 32 lines at
// once (one word column) and splits the line over a warp's lanes, each lane filling its
// segment and the carries joined by a warp scan of (generate, propagate) masks. The round
// loop is a conditional WHILE node of a CUDA graph whose last kernel ends it when a round
// reached nothing or maxrounds is done: no host round trip. The masks (a bit a cell each)
// stay in L2 through the rounds.
#pragma once

#include "mpp_base.cuh"
#include "mpp_div.cuh"

namespace mpp {

// ---- Julia's Float32 min/max/clamp (Base: diff = x - y, its sign bit picks) ----
__device__ __forceinline__ float jmin(float x, float y) {
    const float d = x - y;
    if (isnan(x) || isnan(y)) return d;
    return signbit(d) ? x : y;
}
__device__ __forceinline__ float jmax(float x, float y) {
    const float d = x - y;
    if (isnan(x) || isnan(y)) return d;
    return signbit(d) ? y : x;
}

// eikonal (src/flip.jl:611-623): Godunov's upwind update from the smallest neighbour
// distance along each axis.
__device__ __forceinline__ float eikonal(float a, float b, float c, float h) {
    float t0 = jmin(a, b), t1 = jmax(a, b);
    a = t0;
    b = t1;
    t0 = jmin(b, c);
    t1 = jmax(b, c);
    b = t0;
    c = t1;
    t0 = jmin(a, b);
    t1 = jmax(a, b);
    a = t0;
    b = t1;
    float d = a + h;
    if (d > b) {
        const float ab = a - b;
        d = 0.5f * (a + b + sqrtf(jmax(2.0f * h * h - ab * ab, 0.0f)));
        if (d > c) {
            const float t = a + b + c;
            d = (t + sqrtf(jmax(t * t - 3.0f * (a * a + b * b + c * c - h * h), 0.0f))) / 3.0f;
        }
    }
    return d;
}

// eikonal for three numbers of the same sign (no NaN), where the hardware's min and max are Julia's;
// the division by 3 as div_small rounds it.
__device__ __forceinline__ float eikonal_ord(float a, float b, float c, float h) {
    float t0 = fminf(a, b), t1 = fmaxf(a, b);
    a = t0;
    b = t1;
    t0 = fminf(b, c);
    t1 = fmaxf(b, c);
    b = t0;
    c = t1;
    t0 = fminf(a, b);
    t1 = fmaxf(a, b);
    a = t0;
    b = t1;
    float d = a + h;
    if (d > b) {
        const float ab = a - b;
        d = 0.5f * (a + b + sqrtf(fmaxf(2.0f * h * h - ab * ab, 0.0f)));
        if (d > c) {
            const float t = a + b + c;
            d = div_small(t + sqrtf(fmaxf(t * t - 3.0f * (a * a + b * b + c * c - h * h), 0.0f)), 3.0f, 1.0f / 3.0f);
        }
    }
    return d;
}
// The walls as ranges (the context's build_walls): row (j, k)'s open (not SOLID) cells are x from
// rows[j].x to rows[j].y when k >= rows[n2].x, none below.
struct Walls {
    // a quad (cells 4 q .. 4 q + 3 of row j): open with all cells around it in the plane, inside the
    // walls likewise, or neither
    enum : uint8_t { CLEAR = 0, SHUT = 1, MIXED = 2 };
    const int2* rows;
    const uint8_t* quad;   // [n2][n1 / 4], when n1 is a multiple of 4
    const uint32_t* list;  // j << 16 | q of the MIXED quads, then of the CLEAR ones
    int nlist, nclear;
    __device__ __forceinline__ bool open(int2 r, int i) const { return i >= r.x && i <= r.y; }
};

// min and max that hand a NaN on
__device__ __forceinline__ float nmin(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float nmax(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// reinit_kernel!'s value of a cell from its neighbours f (+x, -x, +y, -y, +z, -z; ok: in range and not
// SOLID) in any case: walls beside it, NaN.
__device__ __forceinline__ float reinit_cell(float cm, const float (&f)[6], unsigned ok, bool solid, float phimax, float h,
                                             float far) {
    if (solid) {
        // a wall cell takes the lowest value of the water next to it
        float lowest = cm;
        bool found = false;
#pragma unroll
        for (int e = 0; e < 6; e++)
            if (ok & (1u << e)) {
                lowest = found ? jmin(lowest, f[e]) : f[e];
                found = true;
            }
        return found ? lowest : (cm > phimax ? phimax : (cm < -phimax ? -phimax : cm));
    }
    const bool inside = cm < 0.0f;
    bool frozen = false;
    float ax = phimax, ay = phimax, az = phimax;
#pragma unroll
    for (int e = 0; e < 6; e++)
        if (ok & (1u << e)) {
            if ((f[e] < 0.0f) != inside) frozen = true;
            const float d = fabsf(f[e]);
            if (e < 2) ax = jmin(ax, d);
            else if (e < 4) ay = jmin(ay, d);
            else az = jmin(az, d);
        }
    if (frozen) return cm;
    const float d = (ax == phimax && ay == phimax && az == phimax) ? far : jmin(eikonal(ax, ay, az, h), phimax);
    return inside ? -d : d;
}
// One cell of a sweep in any place.
__device__ __forceinline__ float reinit_any(const Geo& g, const Walls& wl, const float* phi, int i, int j, int k, int kf,
                                            float phimax, float far, bool& solid) {
    const int n1 = g.n[0], n2 = g.n[1], n3 = g.n[2];
    const int64_t sy = n1, sz = (int64_t)n1 * n2, idx = i + sy * j + sz * k;
    const int2 r0 = wl.rows[j];
    const bool in = wl.open(r0, i), up = k >= kf;
    const unsigned ok = (up && i + 1 < n1 && wl.open(r0, i + 1) ? 1u : 0u) | (up && i > 0 && wl.open(r0, i - 1) ? 2u : 0u) |
                        (up && j + 1 < n2 && wl.open(wl.rows[j + 1 < n2 ? j + 1 : j], i) ? 4u : 0u) |
                        (up && j > 0 && wl.open(wl.rows[j > 0 ? j - 1 : j], i) ? 8u : 0u) |
                        (in && k + 1 < n3 && k + 1 >= kf ? 16u : 0u) | (in && k > 0 && k - 1 >= kf ? 32u : 0u);
    const float f[6] = {ok & 1u ? phi[idx + 1] : 0.f,  ok & 2u ? phi[idx - 1] : 0.f,  ok & 4u ? phi[idx + sy] : 0.f,
                        ok & 8u ? phi[idx - sy] : 0.f, ok & 16u ? phi[idx + sz] : 0.f, ok & 32u ? phi[idx - sz] : 0.f};
    solid = !(in && up);
    return reinit_cell(phi[idx], f, ok, solid, phimax, g.dx, far);
}

// reinit_kernel! (src/flip.jl:631-666), one Jacobi sweep out <- phi, four cells of a row a thread
// (n1 a multiple of 4, 16-byte aligned arrays), and classify! with it when `types` is given.
// Almost every warp's 128 cells of a row cross a wall, and the four cells there would make the
// other 31 threads wait for their longer way (113 M issued warp instructions a sweep at 256^3, 12
// threads in one). So the first loop takes the quads that are open with all around them and those
// inside the walls, told by a byte each (Walls::quad, the same for every plane), and the second
// the quads beside walls (Walls::list) of every plane and the open ones of the planes at the floor
// and the top, a cell a thread. A thread's next quad is stepped (dq, dj, dk), not divided out.
__global__ void __launch_bounds__(TPB) k_reinit4(Geo g, Walls wl, const float* __restrict__ phi, float* __restrict__ out,
                                                 float phimax, uint8_t* __restrict__ types) {
    pdl_wait();
    pdl_trigger();
    const int n1 = g.n[0], n2 = g.n[1], n3 = g.n[2], rq = n1 / 4;
    const float h = g.dx;
    const unsigned sy = (unsigned)n1, sz = (unsigned)n1 * (unsigned)n2;
    // far from the surface every neighbour distance is phimax: the same update for every such cell
    const float far = jmin(eikonal(phimax, phimax, phimax, h), phimax);
    const int kf = wl.rows[n2].x;
    const unsigned step = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned t = t0;
    int q = (int)(t % (unsigned)rq), j = (int)(t / (unsigned)rq % (unsigned)n2), k = (int)(t / (unsigned)rq / (unsigned)n2);
    const int dq = (int)(step % (unsigned)rq), dj = (int)(step / (unsigned)rq % (unsigned)n2),
              dk = (int)(step / (unsigned)rq / (unsigned)n2);
    for (; k < n3; t += step) {
        const uint8_t kind = wl.quad[j * rq + q];
        const unsigned base = 4u * t;
        const bool solid = kind == Walls::SHUT;
        if (solid || (kind == Walls::CLEAR && k > kf && k + 1 < n3)) {
            const float4 C = *reinterpret_cast<const float4*>(phi + base);
            const float c[4] = {C.x, C.y, C.z, C.w};
            float o[4];
            if (solid) {
#pragma unroll
                for (int m = 0; m < 4; m++) o[m] = c[m] > phimax ? phimax : (c[m] < -phimax ? -phimax : c[m]);
            } else {
                const float4 YP = *reinterpret_cast<const float4*>(phi + base + sy);
                const float4 YM = *reinterpret_cast<const float4*>(phi + base - sy);
                const float4 ZP = *reinterpret_cast<const float4*>(phi + base + sz);
                const float4 ZM = *reinterpret_cast<const float4*>(phi + base - sz);
                const float xl = phi[base - 1], xr = phi[base + 4];
                const float yp[4] = {YP.x, YP.y, YP.z, YP.w}, ym[4] = {YM.x, YM.y, YM.z, YM.w},
                            zp[4] = {ZP.x, ZP.y, ZP.z, ZP.w}, zm[4] = {ZM.x, ZM.y, ZM.z, ZM.w};
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    const float f[6] = {m < 3 ? c[m < 3 ? m + 1 : 0] : xr, m > 0 ? c[m > 0 ? m - 1 : 0] : xl, yp[m], ym[m],
                                        zp[m], zm[m]};
                    const float mx = nmax(nmax(nmax(f[0], f[1]), nmax(f[2], f[3])), nmax(f[4], f[5]));
                    const float mn = nmin(nmin(nmin(f[0], f[1]), nmin(f[2], f[3])), nmin(f[4], f[5]));
                    const bool inside = c[m] < 0.0f;
                    // the surface passes when a neighbour's side differs; else the nearest one's distance
                    // is that of the largest (smallest) value
                    const bool frozen = inside ? !(mx < 0.0f) : mn < 0.0f;
                    const float near = inside ? -mx : mn;
                    float v = inside ? -far : far;
                    if (frozen) v = c[m];
                    if (!frozen && !(near >= phimax)) {
                        if (!(mx == mx)) {  // (a NaN neighbour: on no side, so an inside cell was frozen)
                            v = reinit_cell(c[m], f, 63u, false, phimax, h, far);
                        } else {
                            const float d = fminf(eikonal_ord(fminf(phimax, fminf(fabsf(f[0]), fabsf(f[1]))),
                                                              fminf(phimax, fminf(fabsf(f[2]), fabsf(f[3]))),
                                                              fminf(phimax, fminf(fabsf(f[4]), fabsf(f[5]))), h), phimax);
                            v = inside ? -d : d;
                        }
                    }
                    o[m] = v;
                }
            }
            *reinterpret_cast<float4*>(out + base) = make_float4(o[0], o[1], o[2], o[3]);
            if (types) {
                uint8_t ty[4];
#pragma unroll
                for (int m = 0; m < 4; m++) ty[m] = solid ? SOLID : (o[m] < 0.0f ? LIQUID : AIR);
                *reinterpret_cast<uchar4*>(types + base) = make_uchar4(ty[0], ty[1], ty[2], ty[3]);
            }
        }
        q += dq;
        j += dj;
        k += dk;
        if (q >= rq) {
            q -= rq;
            j++;
        }
        if (j >= n2) {
            j -= n2;
            k++;
        }
    }
    // the rest, a cell a thread: quads beside walls in every plane, then the open quads of the planes
    // 0 .. kf and n3 - 1
    const unsigned walled = 4u * (unsigned)wl.nlist, nclear = 4u * (unsigned)wl.nclear;
    const unsigned low = (unsigned)(kf + 1 < n3 ? kf + 1 : n3), planes = low < (unsigned)n3 ? low + 1u : low;
    const unsigned all = walled * (unsigned)n3, end = all + nclear * planes;
    for (unsigned e = t0; e < end; e += step) {
        const bool w = e < all;
        const unsigned x = w ? e : e - all, m = w ? walled : nclear, p = x / m, c = x - p * m;
        const uint32_t jq = (w ? wl.list : wl.list + wl.nlist)[c >> 2];
        const int kk = w ? (int)p : (p < low ? (int)p : n3 - 1), jj = (int)(jq >> 16), i = 4 * (int)(jq & 0xffffu) + (int)(c & 3u);
        const int64_t idx = i + (int64_t)n1 * (jj + (int64_t)n2 * kk);
        bool solid;
        const float v = reinit_any(g, wl, phi, i, jj, kk, kf, phimax, far, solid);
        out[idx] = v;
        if (types) types[idx] = solid ? SOLID : (v < 0.0f ? LIQUID : AIR);
    }
}

// classify_kernel! (src/flip.jl:682-686), four cells a thread (as k_reinit4; types 4-byte aligned).
__global__ void __launch_bounds__(TPB) k_classify4(Geo g, Walls wl, const float* __restrict__ phi, uint8_t* __restrict__ types) {
    pdl_wait();
    pdl_trigger();
    const int n2 = g.n[1], n3 = g.n[2], rq = g.n[0] / 4, kf = wl.rows[n2].x;
    const unsigned step = gridDim.x * blockDim.x;
    unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    int q = (int)(t % (unsigned)rq), j = (int)(t / (unsigned)rq % (unsigned)n2), k = (int)(t / (unsigned)rq / (unsigned)n2);
    const int dq = (int)(step % (unsigned)rq), dj = (int)(step / (unsigned)rq % (unsigned)n2),
              dk = (int)(step / (unsigned)rq / (unsigned)n2);
    for (; k < n3; t += step) {
        const float4 C = *reinterpret_cast<const float4*>(phi + 4u * t);
        const int2 r = wl.rows[j];
        const float c[4] = {C.x, C.y, C.z, C.w};
        uint8_t ty[4];
#pragma unroll
        for (int m = 0; m < 4; m++) ty[m] = !(wl.open(r, 4 * q + m) && k >= kf) ? SOLID : (c[m] < 0.0f ? LIQUID : AIR);
        *reinterpret_cast<uchar4*>(types + 4u * t) = make_uchar4(ty[0], ty[1], ty[2], ty[3]);
        q += dq;
        j += dj;
        k += dk;
        if (q >= rq) {
            q -= rq;
            j++;
        }
        if (j >= n2) {
            j -= n2;
            k++;
        }
    }
}

// One Jacobi sweep, a cell a thread, for rows or arrays that k_reinit4 does not take.
__global__ void __launch_bounds__(TPB) k_reinit(Geo g, Walls wl, const float* __restrict__ phi, float* __restrict__ out,
                                                float phimax, uint8_t* __restrict__ types) {
    pdl_wait();
    pdl_trigger();
    const int kf = wl.rows[g.n[1]].x;
    const float far = jmin(eikonal(phimax, phimax, phimax, g.dx), phimax);
    FOR_CELLS(g.n[0], g.n[1], g.n[2], i, j, k, idx) {
        bool solid;
        const float v = reinit_any(g, wl, phi, i, j, k, kf, phimax, far, solid);
        out[idx] = v;
        if (types) types[idx] = solid ? SOLID : (v < 0.0f ? LIQUID : AIR);
    }
}

// classify_kernel! (src/flip.jl:682-686) on its own (redistance! with no sweep).
__global__ void __launch_bounds__(TPB) k_classify(Geo g, const float* __restrict__ phi, uint8_t* __restrict__ types) {
    pdl_wait();
    pdl_trigger();
    FOR_CELLS(g.n[0], g.n[1], g.n[2], i, j, k, idx) {
        types[idx] = issolidcell(g, i, j, k) ? SOLID : (phi[idx] < 0.0f ? LIQUID : AIR);
    }
}

// ---- trapped air (src/flip.jl:698-760) on bit masks ----
// Word (wx, j, k) of a mask holds cells i = 32 wx .. 32 wx + 31 of row (j, k), bit b for
// i = 32 wx + b; a row has W1 = ceil(n1 / 32) words; bits past n1 are 0 (never AIR).
struct TrapMasks {
    uint32_t* air;    // AIR cells
    uint32_t* reach;  // cells reached from the top layer's air
    int n1, n2, n3, W1;
};
// The round loop's device state.
struct TrapState {
    int changed;    // a sweep of this round reached a new cell
    int rounds;     // rounds run
    int maxrounds;
    int pad;
};

// seedair_kernel! (src/flip.jl:704-708) and the AIR mask: a thread a word.
__global__ void __launch_bounds__(TPB) k_trap_pack(TrapMasks T, const uint8_t* __restrict__ types, TrapState* st,
                                                   int maxrounds, int vec) {
    pdl_wait();
    pdl_trigger();
    const int64_t words = (int64_t)T.W1 * T.n2 * T.n3;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t0 == 0) {
        st->changed = 0;
        st->rounds = 0;
        st->maxrounds = maxrounds;
    }
    for (int64_t t = t0; t < words; t += (int64_t)gridDim.x * blockDim.x) {
        const unsigned row = (unsigned)t / (unsigned)T.W1;  // the host checks the masks fit 32 bits
        const int wx = (int)((unsigned)t - row * (unsigned)T.W1);
        const int k = (int)(row / (unsigned)T.n2);
        const int i0 = wx * 32;
        const uint8_t* p = types + row * T.n1 + i0;
        uint32_t a = 0;
        if (vec) {  // n1 a multiple of 32, types 16-byte aligned: two 16-byte loads
            const uint4 v0 = reinterpret_cast<const uint4*>(p)[0], v1 = reinterpret_cast<const uint4*>(p)[1];
            const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
            for (int q = 0; q < 8; q++)  // four classes at a time: a byte of ones each, one bit of it kept, added up
                a |= (((__vcmpeq4(w[q], 0x01010101u * AIR) & 0x08040201u) * 0x01010101u) >> 24) << (4 * q);
        } else {
            const int cnt = T.n1 - i0 < 32 ? T.n1 - i0 : 32;
            for (int b = 0; b < cnt; b++)
                if (p[b] == AIR) a |= 1u << b;
        }
        T.air[t] = a;
        T.reach[t] = k == T.n3 - 1 ? a : 0u;  // the top layer's air
    }
}

// Fill toward higher / lower bits from the seeds g through runs of set bits of p (the
// AIR mask): 5 doubling steps of a shift-and-mask carry.
__device__ __forceinline__ uint32_t fill_up(uint32_t g, uint32_t p) {
    g |= p & (g << 1);
    p &= p << 1;
    g |= p & (g << 2);
    p &= p << 2;
    g |= p & (g << 4);
    p &= p << 4;
    g |= p & (g << 8);
    p &= p << 8;
    g |= p & (g << 16);
    return g;
}
__device__ __forceinline__ uint32_t fill_down(uint32_t g, uint32_t p) {
    g |= p & (g >> 1);
    p &= p >> 1;
    g |= p & (g >> 2);
    p &= p >> 2;
    g |= p & (g >> 4);
    p &= p >> 4;
    g |= p & (g >> 8);
    p &= p >> 8;
    g |= p & (g >> 16);
    return g;
}

// sweepair_kernel! along x (src/flip.jl:715-731): a thread a row, there and back through
// its words. A run of air holding a reached cell is reached whole.
__global__ void __launch_bounds__(TPB) k_trap_sweep_x(TrapMasks T, TrapState* st) {
    pdl_wait();
    pdl_trigger();
    const int64_t rows = (int64_t)T.n2 * T.n3;
    bool ch = false;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x) {
        uint32_t* R = T.reach + r * T.W1;
        const uint32_t* A = T.air + r * T.W1;
        uint32_t carry = 0;
        for (int w = 0; w < T.W1; w++) {
            const uint32_t a = A[w], r0 = R[w];
            const uint32_t f = fill_up(r0 | (carry & a & 1u), a);
            carry = f >> 31;
            if (f != r0) {
                R[w] = f;
                ch = true;
            }
        }
        carry = 0;
        for (int w = T.W1 - 1; w >= 0; w--) {
            const uint32_t a = A[w], r0 = R[w];
            const uint32_t f = fill_down(r0 | ((carry << 31) & a), a);
            carry = f & 1u;
            if (f != r0) {
                R[w] = f;
                ch = true;
            }
        }
    }
    if (__syncthreads_or(ch) && threadIdx.x == 0) atomicOr(&st->changed, 1);
}

// sweepair_kernel! along y (axis 1) or z (axis 2): a warp takes one word column (32 lines)
// and splits it into 32 segments of S words; each lane fills its segment (a line's fill is
// F_p = A_p & (R_p | F_{p-1})), and the carries into the segments come from a warp scan of
// the segments' (generate, propagate) masks: g = the fill from a zero carry, p = the AND of
// A over the segment, so a carry c leaves the segment as g | (p & c). Lines longer than
// 32 S go chunk by chunk, the carry passed on. Forward over the chunks, then back.
constexpr int TRAP_S = 8;
__global__ void __launch_bounds__(TPB) k_trap_sweep_col(TrapMasks T, TrapState* st, int axis) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int64_t ncols = axis == 1 ? (int64_t)T.W1 * T.n3 : (int64_t)T.W1 * T.n2;
    const int len = axis == 1 ? T.n2 : T.n3;
    const int64_t step = axis == 1 ? (int64_t)T.W1 : (int64_t)T.W1 * T.n2;
    const int chunk = 32 * TRAP_S;
    const int nchunks = (len + chunk - 1) / chunk;
    bool ch = false;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t col = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); col < ncols; col += warps) {
        const int wx = (int)(col % T.W1);
        const int64_t other = col / T.W1;  // k (y sweep) or j (z sweep)
        const int64_t base = axis == 1 ? wx + (int64_t)T.W1 * T.n2 * other : wx + (int64_t)T.W1 * other;
        for (int dir = 0; dir < 2; dir++) {  // there (increasing p), then back
            __syncwarp();  // the way back reads what the other lanes wrote on the way there
            uint32_t carry = 0;
            for (int cq = 0; cq < nchunks; cq++) {
                const int cidx = dir == 0 ? cq : nchunks - 1 - cq;
                // this lane's segment of the chunk, in walking order
                const int p0 = cidx * chunk + (dir == 0 ? lane : 31 - lane) * TRAP_S;
                uint32_t a[TRAP_S], r[TRAP_S];
#pragma unroll
                for (int s = 0; s < TRAP_S; s++) {
                    const int p = dir == 0 ? p0 + s : p0 + TRAP_S - 1 - s;
                    const bool in = p < len;
                    a[s] = in ? T.air[base + (int64_t)p * step] : 0u;
                    r[s] = in ? T.reach[base + (int64_t)p * step] : 0u;
                }
                uint32_t gsum = 0, psum = 0xffffffffu;
#pragma unroll
                for (int s = 0; s < TRAP_S; s++) {
                    gsum = a[s] & (r[s] | gsum);
                    psum &= a[s];
                }
                // inclusive scan over the lanes in walking order: (g, p) then (g', p') is
                // (g' | (p' & g), p & p')
                uint32_t G = gsum, P = psum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t go = __shfl_up_sync(0xffffffffu, G, o), po = __shfl_up_sync(0xffffffffu, P, o);
                    if (lane >= o) {
                        G = G | (P & go);
                        P = P & po;
                    }
                }
                uint32_t cin = __shfl_up_sync(0xffffffffu, G, 1);
                uint32_t pin = __shfl_up_sync(0xffffffffu, P, 1);
                // the carry into this lane: from the chunks before, through lanes 0..lane-1
                cin = lane == 0 ? carry : (cin | (pin & carry));
                uint32_t f = cin;
#pragma unroll
                for (int s = 0; s < TRAP_S; s++) {
                    const int p = dir == 0 ? p0 + s : p0 + TRAP_S - 1 - s;
                    f = a[s] & (r[s] | f);
                    if (p < len && f != r[s]) {
                        T.reach[base + (int64_t)p * step] = f;
                        ch = true;
                    }
                }
                // the carry out of the chunk: the last lane's fill
                carry = __shfl_sync(0xffffffffu, f, 31);
            }
        }
    }
    if (__syncthreads_or(ch) && threadIdx.x == 0) atomicOr(&st->changed, 1);
}

// The end of a round (src/flip.jl:751-757): another round while this one reached a cell
// and fewer than maxrounds have run.
__global__ void k_trap_round(TrapState* st, cudaGraphConditionalHandle cond) {
    pdl_wait();
    const int r = st->rounds + 1;
    st->rounds = r;
    const int again = st->changed != 0 && r < st->maxrounds;
    st->changed = 0;
    cudaGraphSetConditional(cond, again ? 1u : 0u);
}

// fillair_kernel! (src/flip.jl:734-740): AIR that no sweep reached becomes LIQUID, with phi
// at most -depth (Julia's min). A thread a word of 32 cells.
__global__ void __launch_bounds__(TPB) k_trap_fill(TrapMasks T, uint8_t* __restrict__ types, float* __restrict__ phi,
                                                   float depth) {
    pdl_wait();
    pdl_trigger();
    const int64_t words = (int64_t)T.W1 * T.n2 * T.n3;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < words; t += (int64_t)gridDim.x * blockDim.x) {
        uint32_t m = T.air[t] & ~T.reach[t];
        if (!m) continue;
        const int wx = (int)(t % T.W1);
        const int64_t at = (t / T.W1) * T.n1 + (int64_t)wx * 32;
        while (m) {
            const int b = __ffs(m) - 1;
            m &= m - 1;
            types[at + b] = LIQUID;
            phi[at + b] = jmin(phi[at + b], -depth);
        }
    }
}

}  // namespace mpp
