// Short-range part of a P3M force in the periodic box, for the 3-D particle
// mesh (pm3d.cu). The mesh's Green's function -4 pi G / k^2 e^{-k^2 r_s^2} is
// the force of Gaussian clouds; what it leaves out of a pair at distance r
// is G m g(alpha r) / r^2 along the separation, alpha = 1 / (2 r_s) and
// g(x) = erfc(x) + 2 x e^{-x^2} / sqrt(pi): the real-space term of an Ewald
// sum with that alpha. With the Plummer softening of the direct sum the pair
// adds ((1 + eps^2 / r^2)^{-3/2} - 1) / r^2 as well. Both act for r < r_cut
// (g(alpha r_cut) is the truncation error of a pair at the cutoff, relative to
// its Newtonian term: 4.4e-4 for alpha r_cut = 3, 2e-5 for 3.5).
// The reference has no such term: its 2-D PM (pm_kernel.py:63-154) ends at
// the mesh force; here it is the exact short-range part of the force the
// learned correction then refines.
//
//   keys    : chaining cell (side box / M >= r_cut) of every particle
//   sort    : stable radix sort by cell (devscan.cuh), particles gathered in
//             that order as (x, y, z, m)
//   bounds  : first and last sorted particle of every cell
//   items   : one work item per group of 32 particles of a cell (cells
//             hold from none to many thousands in a clustered state), listed
//             by the power of two of its source chunks, longest first
//   pairs   : persistent warps take items from a counter (a dense cell's
//             items spread over many warps). Every pair is evaluated once
//             (the two accelerations are m_j h d and -m_i h d): an item pairs
//             its particles with each other, with the later particles of its
//             cell and with the particles of the neighbouring cells of
//             higher index (13 or so of the 26, periodic). The sources are
//             staged through the warp's shared memory in chunks of 32,
//             relative to the item's cell corner, so that f32 differences
//             keep the positions' resolution; lane l meets sources (l + k)
//             and (l + k + 16) mod 32 at step k, in packed f32x2 arithmetic,
//             and the sources' sums rotate through the lanes with them, so
//             that both sides accumulate in registers. Both go to an f32
//             accumulator per particle with atomics.
//   finish  : acceleration = mesh force (already in a) + G x accumulator, in
//             f64, through the KDK epilogue of the force passes.

#include "pm3d.cuh"
#include "devscan.cuh"

namespace {

constexpr int PP_WARPS = 4;                         // cells per block

unsigned blocks_for(long long n, int nt) { return (unsigned)((n + nt - 1) / nt); }

__global__ void k_pp_keys(const Pm3Parts s, int M, double inv_l, unsigned long long* __restrict__ keys,
                          unsigned* __restrict__ vals) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.n) return;
    int c[3];
    for (int d = 0; d < 3; ++d) {
        const double f = s.x[d][p] * inv_l;
        const int ci = f >= 0.0 ? (int)f : 0;              // NaN and negatives go to cell 0
        c[d] = min(ci, M - 1);
    }
    keys[p] = ((unsigned long long)c[2] * M + c[1]) * M + c[0];
    vals[p] = (unsigned)p;
}

__global__ void k_pp_gather(const Pm3Parts s, const unsigned* __restrict__ order, double4* __restrict__ src) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= s.n) return;
    const unsigned p = order[q];
    src[q] = make_double4(s.x[0][p], s.x[1][p], s.x[2][p], s.m ? s.m[p] : s.mass_const);
}

// first and one-past-last sorted position of every occupied cell (the
// others stay 0, 0)
__global__ void k_pp_bounds(const unsigned long long* __restrict__ keys, long long n, int* __restrict__ first,
                            int* __restrict__ last) {
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const unsigned long long k = keys[q];
    if (q == 0 || keys[q - 1] != k) first[k] = (int)q;
    if (q == n - 1 || keys[q + 1] != k) last[k] = (int)(q + 1);
}

// Work lists of items by length. An item's length is the number of source
// chunks of 32 its warp walks: the later ones of its cell and those of the
// neighbouring cells of higher index; class = floor(log2(length)). The
// warps take the longest class first: an item of a collapsed halo's cell is
// one warp's work for milliseconds, and the ones taken last set the tail. (64
// targets an item, two per lane sharing the sources' loads and rotation, halved
// the items and gained nothing: 442,368 uniform particles 2065 us a pair pass
// against 1796 before.)
constexpr int PP_CLASSES = 16;

__device__ __forceinline__ int pp_chunks(const int* first, const int* last, long long c) {
    return (last[c] - first[c] + 31) / 32;
}

// (cell, first target) of every item into the list, the classes one after
// another, the longest first (thread per cell; an item's length falls along its
// cell, so a class is one stretch). Two launches: COUNT adds up the classes'
// lengths, the other writes behind its class's cursor. (A list of full length a
// class in one launch took 16 times the memory, 128 bytes a particle.)
template <bool COUNT>
__global__ void k_pp_items(const int* __restrict__ first, const int* __restrict__ last, int M, long long cells,
                           unsigned* __restrict__ n_items, unsigned* __restrict__ cursor, int2* __restrict__ items) {
    __shared__ unsigned base[PP_CLASSES];
    if (!COUNT) {
        if (threadIdx.x < PP_CLASSES) {
            unsigned b = 0;
            for (int k = PP_CLASSES - 1; k > (int)threadIdx.x; --k) b += n_items[k];
            base[threadIdx.x] = b;
        }
        __syncthreads();
    }
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells) return;
    const int g = pp_chunks(first, last, c);
    if (g == 0) return;
    const int cx = (int)(c % M), cy = (int)((c / M) % M), cz = (int)(c / ((long long)M * M));
    const int xs[3] = {cx ? cx - 1 : M - 1, cx, cx + 1 < M ? cx + 1 : 0};
    const int ys[3] = {cy ? cy - 1 : M - 1, cy, cy + 1 < M ? cy + 1 : 0};
    const int zs[3] = {cz ? cz - 1 : M - 1, cz, cz + 1 < M ? cz + 1 : 0};
    long long near = 0;
#pragma unroll
    for (int nb = 0; nb < 27; ++nb) {
        if (nb == 13) continue;
        const long long nc = ((long long)zs[nb / 9] * M + ys[nb / 3 % 3]) * M + xs[nb % 3];
        const int q = pp_chunks(first, last, nc);
        near += nc > c ? q : 0;
    }
    for (int k = 0; k < g;) {
        const long long len = near + g - k;                 // >= 1
        const int cls = min(PP_CLASSES - 1, 63 - __clzll(len));
        // down to length 2^cls the class stays the same (class 15 is open above)
        const int run = (int)min((long long)(g - k), len - (1ll << cls) + 1);
        if (COUNT) {
            atomicAdd(n_items + cls, (unsigned)run);
        } else {
            const unsigned at = base[cls] + atomicAdd(cursor + cls, (unsigned)run);
            for (int j = 0; j < run; ++j) items[at + j] = make_int2((int)c, first[c] + 32 * (k + j));
        }
        k += run;
    }
}

struct PPArgs {
    const double4* src;             // particles in cell order: x, y, z, m
    const unsigned* order;          // cell order -> particle index
    const int* first;               // M^3
    const int* last;
    int M;
    double l;                       // chaining cell side
    double box;
    double G;
    float alpha, rc2, eps2;
    const int2* items;              // longest first
    const unsigned* n_items;        // by class
    unsigned* next;                 // work counter (zero at launch)
    float* acc;                     // 3 x n, by cell-order position (zero at launch)
    long long n;
};

// ---- packed f32x2 pair arithmetic: two sources per lane and step
typedef unsigned long long f2x;                     // two packed f32

__device__ __forceinline__ f2x pk2(float lo, float hi) {
    f2x r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void upk2(f2x v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2x add2(f2x a, f2x b) {
    f2x d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2x mul2(f2x a, f2x b) {
    f2x d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2x fma2(f2x a, f2x b, f2x c) {
    f2x d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ f2x shfl2(f2x v, int from) {
    return __shfl_sync(0xffffffffu, v, from);
}

// h(r) of a pair (a_i += m_j h d, a_j -= m_i h d, d = x_j - x_i), for
// 0 < r < r_cut: (g(x) + (1 + u)^{-3/2} - 1) / r^3 with u = eps^2 / r^2,
// evaluated as (g - 1) / r^3 + (r^2 + eps^2)^{-3/2} (its rounding is about
// 1e-7 of the pair's Newtonian term 1 / r^2 for every r). erfc(x) =
// e^{-x^2} t (a1 + a2 t + ... + a5 t^4), t = 1 / (1 + p x) (Abramowitz &
// Stegun 7.1.26, |error| <= 1.5e-7), so g shares its Gaussian with the
// second term 2 x e^{-x^2} / sqrt(pi). No branches: out of range (and for
// coincident particles, where the erfc form is not finite) the caller
// selects 0. Two pairs at a time in packed f32x2 arithmetic; the reciprocal
// square roots, the exponential and the reciprocal are f32 MUFU operations.
// (A polynomial of (1 - g) / x^3 in x^2 instead of the erfc form, one MUFU a pair
// instead of four and as exact, took a halo step from 12.3 to 9.7 ms, but its
// rounding moved the f64 state by up to 1.5e-9 of itself: left out.)
__device__ __forceinline__ f2x dup(float v) { return pk2(v, v); }

struct PPConst {
    f2x alpha, eps2;
};

__device__ __forceinline__ f2x pp_h2(f2x R2, f2x alpha, f2x eps2) {
    float r0, r1;
    upk2(R2, r0, r1);
    const f2x RI = pk2(sss_rsqrt_approx_f32(r0), sss_rsqrt_approx_f32(r1));
    const f2x INV3 = mul2(mul2(RI, RI), RI);
    const f2x X = mul2(alpha, mul2(R2, RI));
    float v0, v1;
    upk2(mul2(mul2(X, X), dup(-1.44269504f)), v0, v1);
    const f2x EX = pk2(ex2_approx(v0), ex2_approx(v1));
    float d0, d1;
    upk2(fma2(dup(0.3275911f), X, dup(1.0f)), d0, d1);
    const f2x T = pk2(rcp_approx(d0), rcp_approx(d1));
    f2x P = fma2(T, dup(1.061405429f), dup(-1.453152027f));
    P = fma2(T, P, dup(1.421413741f));
    P = fma2(T, P, dup(-0.284496736f));
    P = fma2(T, P, dup(0.254829592f));
    const f2x Gx = mul2(EX, fma2(dup(1.12837917f), X, mul2(T, P)));
    float s0, s1;
    upk2(add2(R2, eps2), s0, s1);
    const f2x SI = pk2(sss_rsqrt_approx_f32(s0), sss_rsqrt_approx_f32(s1));
    return fma2(add2(Gx, dup(-1.0f)), INV3, mul2(mul2(SI, SI), SI));
}

// Stage a chunk's sources (lane l holds source l) as the packed pairs the
// steps use: entry j = sources j and (j + da) mod 32, so that a step's operands
// are two 16-byte shared loads and no register moves.
__device__ __forceinline__ void pp_stage(ulonglong2* stage, int lane, int da, float x, float y, float z, float m) {
    const int o = (lane + da) & 31;
    const float x1 = __shfl_sync(0xffffffffu, x, o), y1 = __shfl_sync(0xffffffffu, y, o);
    const float z1 = __shfl_sync(0xffffffffu, z, o), m1 = __shfl_sync(0xffffffffu, m, o);
    __syncwarp();                                          // the previous chunk is consumed
    stage[lane] = make_ulonglong2(pk2(x, x1), pk2(y, y1));
    stage[32 + lane] = make_ulonglong2(pk2(z, z1), pk2(m, m1));
    __syncwarp();
}

// A lane's target (negated, both halves) and its sums, one half per source of a step.
struct PPTarget {
    f2x nx, ny, nz, nm;
    f2x ax, ay, az;
};

// One chunk of sources against the lanes' targets, two sources per step:
// offsets (a, a + DA) for steps a = A0 .. A1 - 1 (source (lane + offset) mod
// 32); OWN masks offset 16 on lanes 16 .. 31 (32 particles among themselves,
// whose pairs (l, l + 16) and (l + 16, l) coincide). Both sources' sums rotate
// through the lanes and end on their own lanes, then go to the accumulator.
// 35 FMA-pipe operations and four special-function ones a pair (the latter
// bound it), with the 6 shuffles and two 16-byte shared loads of a step shared
// by its 2 pairs. Two steps at a time, skipped by one vote where no pair is in range:
// particles that come in spatial order, a lattice above all, lie together in the
// chunks (1,048,576 on a lattice, r_split 2.25 cells, r_cut 3 / alpha: 3.80 ms a pass,
// 5.20 without the vote, 3.87 with one a step; uniform at random 4.53, 5.18, 4.62). A
// vote a step holds up the longest items, a halo's, which two steps' work hides again
// (262,144 particles in 192 halos 1,386 us a step, 1,594 without, 1,670 with one a
// step). 1,048,576 particles collapsed into halos (7.2e9 candidate pairs, 5.1e9 in
// range): 11.0 ms a step against 15.2 with sources packed by register moves and
// items in cell order (the last heavy items then ran on by themselves). Sorting
// particles inside a cell and testing chunk boxes saves only a fifth of these pairs.
template <bool OWN, int A0, int A1, int DA>
__device__ __forceinline__ void pp_chunk2(const ulonglong2* stage, int lane, PPTarget& t, const PPConst& k,
                                          const PPArgs& q, long long src0, int m) {
    static_assert((A1 - A0) % 2 == 0, "steps by two");
    f2x BX = 0ull, BY = 0ull, BZ = 0ull;             // sums of sources (lane + a) and (lane + a + DA)
    const int from = (lane + 1) & 31;
    auto rotate = [&]() {                            // take the next lane's sums (sources + 1)
        BX = shfl2(BX, from);
        BY = shfl2(BY, from);
        BZ = shfl2(BZ, from);
    };
#pragma unroll 1
    for (int a = A0; a < A1; a += 2) {
        f2x DX[2], DY[2], DZ[2], R2[2], M[2];
        bool in0[2], in1[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const ulonglong2 xy = stage[(lane + a + u) & 31], zm = stage[32 + ((lane + a + u) & 31)];
            DX[u] = add2(xy.x, t.nx);
            DY[u] = add2(xy.y, t.ny);
            DZ[u] = add2(zm.x, t.nz);
            M[u] = zm.y;
            R2[u] = fma2(DX[u], DX[u], fma2(DY[u], DY[u], mul2(DZ[u], DZ[u])));
            float r0, r1;
            upk2(R2[u], r0, r1);
            in0[u] = r0 < q.rc2 && r0 > 0.0f;
            in1[u] = r1 < q.rc2 && r1 > 0.0f && !(OWN && a + u + DA == 16 && lane >= 16);
        }
        if (__any_sync(0xffffffffu, in0[0] || in1[0] || in0[1] || in1[1])) {       // (warp-uniform)
            f2x H[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                float h0, h1;
                upk2(pp_h2(R2[u], k.alpha, k.eps2), h0, h1);
                H[u] = pk2(in0[u] ? h0 : 0.0f, in1[u] ? h1 : 0.0f);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const f2x HJ = mul2(H[u], M[u]), HI = mul2(H[u], t.nm);
                t.ax = fma2(HJ, DX[u], t.ax);
                t.ay = fma2(HJ, DY[u], t.ay);
                t.az = fma2(HJ, DZ[u], t.az);
                BX = fma2(HI, DX[u], BX);
                BY = fma2(HI, DY[u], BY);
                BZ = fma2(HI, DZ[u], BZ);
                if (u == 0) rotate();
            }
        } else {
            rotate();
        }
        if (a + 2 < A1) rotate();
    }
    // lane l holds sources (l + A1 - 1) and (l + A1 - 1 + DA): deliver both to their lanes
    const int fa = (lane - (A1 - 1)) & 31, fb = (lane - (A1 - 1 + DA)) & 31;
    float xa, xb, ya, yb, za, zb, t0, t1;
    upk2(shfl2(BX, fa), xa, t0);
    upk2(shfl2(BX, fb), t1, xb);
    upk2(shfl2(BY, fa), ya, t0);
    upk2(shfl2(BY, fb), t1, yb);
    upk2(shfl2(BZ, fa), za, t0);
    upk2(shfl2(BZ, fb), t1, zb);
    if (lane < m) {
        atomicAdd(q.acc + src0 + lane, xa + xb);
        atomicAdd(q.acc + q.n + src0 + lane, ya + yb);
        atomicAdd(q.acc + 2 * q.n + src0 + lane, za + zb);
    }
}

// The sources [s0, s1) (shifted by s) against the lanes' targets, chunk by chunk.
__device__ __forceinline__ void pp_walk(ulonglong2* stage, int lane, PPTarget& t, const PPConst& k, const PPArgs& q,
                                        int s0, int s1, double sx, double sy, double sz) {
    for (int j0 = s0; j0 < s1; j0 += 32) {
        const int j = j0 + lane;
        float x = 1e18f, y = 1e18f, z = 1e18f, m = 0.0f;            // padding: out of range of everything
        if (j < s1) {
            const double4 p = q.src[j];
            x = (float)(p.x + sx);
            y = (float)(p.y + sy);
            z = (float)(p.z + sz);
            m = (float)p.w;
        }
        pp_stage(stage, lane, 16, x, y, z, m);
        pp_chunk2<false, 0, 16, 16>(stage, lane, t, k, q, j0, min(32, s1 - j0));
    }
}

// An item: the 32 targets from t0 of a cell. Every target meets its sources in ascending order.
__device__ __forceinline__ void pp_item(ulonglong2* stage, int lane, const PPArgs& q, int c, int t0,
                                        const PPConst& k) {
    const int M = q.M, cl = q.last[c];
    const int cx = c % M, cy = (c / M) % M, cz = c / (M * M);
    const double ox = cx * q.l, oy = cy * q.l, oz = cz * q.l;
    const int t = t0 + lane;
    const bool act = t < cl;
    float tx = -1e18f, ty = -1e18f, tz = -1e18f, tm = 0.0f;         // padding: out of range, of padding sources too
    if (act) {
        const double4 p = q.src[t];
        tx = (float)(p.x - ox);
        ty = (float)(p.y - oy);
        tz = (float)(p.z - oz);
        tm = (float)p.w;
    }
    PPTarget T{dup(-tx), dup(-ty), dup(-tz), dup(-tm), 0ull, 0ull, 0ull};
    // the particles with each other (offsets 1 .. 16 as (j, j + 8), j = 1 .. 8)
    pp_stage(stage, lane, 8, act ? tx : 1e18f, act ? ty : 1e18f, act ? tz : 1e18f, tm);
    pp_chunk2<true, 1, 9, 8>(stage, lane, T, k, q, t0, min(32, cl - t0));
    // the later particles of the cell, then the neighbouring cells of higher index
    for (int nb = -1; nb < 27; ++nb) {
        int s0, s1;
        double sx = -ox, sy = -oy, sz = -oz;                    // source shift: periodic image - corner
        if (nb < 0) {
            s0 = t0 + 32;
            s1 = cl;
        } else {
            if (nb == 13) continue;                            // the cell itself
            int nx = cx + nb % 3 - 1, ny = cy + (nb / 3) % 3 - 1, nz = cz + nb / 9 - 1;
            if (nx < 0) { nx += M; sx -= q.box; } else if (nx >= M) { nx -= M; sx += q.box; }
            if (ny < 0) { ny += M; sy -= q.box; } else if (ny >= M) { ny -= M; sy += q.box; }
            if (nz < 0) { nz += M; sz -= q.box; } else if (nz >= M) { nz -= M; sz += q.box; }
            const int nc = (nz * M + ny) * M + nx;
            if (nc < c) continue;                              // that cell's items take these pairs
            s0 = q.first[nc];
            s1 = q.last[nc];
        }
        pp_walk(stage, lane, T, k, q, s0, s1, sx, sy, sz);
    }
    float x0, x1, y0, y1, z0, z1;
    upk2(T.ax, x0, x1);
    upk2(T.ay, y0, y1);
    upk2(T.az, z0, z1);
    if (act) {
        atomicAdd(q.acc + t, x0 + x1);
        atomicAdd(q.acc + q.n + t, y0 + y1);
        atomicAdd(q.acc + 2 * q.n + t, z0 + z1);
    }
}

__global__ void __launch_bounds__(PP_WARPS * 32) k_pp_pairs(const PPArgs q) {
    __shared__ ulonglong2 sh[PP_WARPS][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned total = __reduce_add_sync(0xffffffffu, lane < PP_CLASSES ? q.n_items[lane] : 0u);
    ulonglong2* stage = sh[w];
    PPConst k;
    k.alpha = dup(q.alpha);
    k.eps2 = dup(q.eps2);
    // no more items than warps: by the warp's place, which spreads them over all SMs (taken from the counter,
    // 4 each by the blocks that start first, 32,768 particles in 7^3 cells took 1,020 us a step, placed 727)
    const unsigned warps = gridDim.x * PP_WARPS, placed = total <= warps ? warps : 0u;
    auto take = [&]() {
        unsigned it = 0;
        if (lane == 0) it = atomicAdd(q.next, 1u);
        return __shfl_sync(0xffffffffu, it, 0);
    };
    for (unsigned it = placed ? w * gridDim.x + blockIdx.x : take(); it < total; it = placed ? total : take()) {
        const int2 item = q.items[it];
        pp_item(stage, lane, q, item.x, item.y, k);
    }
}

// acceleration = mesh force + G x pair sums, then the epilogue
__global__ void k_pp_finish(const PPArgs q, const Pm3Parts s, const Pm3Epi e) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= s.n) return;
    const unsigned i = q.order[t];
    const long long n = q.n;
    pm3_epilogue(s, e, i, s.a[0][i] + q.G * (double)q.acc[t], s.a[1][i] + q.G * (double)q.acc[n + t],
                 s.a[2][i] + q.G * (double)q.acc[2 * n + t]);
}

}  // namespace

extern "C" int sss_pm3_short(sss_pm3* p, const sss_pm3_particles* s, double G, double alpha, double r_cut,
                             double eps, int mode, double hdt, double dt, float* snap, void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    if (!s) return sss_set_err(ctx, SSS_ERR_ARG, "NULL particle state");
    if (s->n < 0) return sss_set_err(ctx, SSS_ERR_ARG, "negative particle count");
    if (mode < SSS_PM3_FORCE || mode > SSS_PM3_KICK_DRIFT) return sss_set_err(ctx, SSS_ERR_ARG, "bad mode");
    if (!(alpha > 0.0)) return sss_set_err(ctx, SSS_ERR_ARG, "alpha must be > 0");
    if (!(r_cut > 0.0) || !(eps >= 0.0)) return sss_set_err(ctx, SSS_ERR_ARG, "r_cut must be > 0, eps >= 0");
    const double mf = floor(p->box / r_cut);
    if (!(mf >= 3.0)) return sss_set_err(ctx, SSS_ERR_ARG, "r_cut must be <= box / 3");
    const int M = (int)std::min(mf, 1024.0);
    if (s->n == 0) return SSS_OK;
    if (s->n >= ((int64_t)1 << 31)) return sss_set_err(ctx, SSS_ERR_ARG, "too many particles");
    for (int c = 0; c < 3; ++c)
        if (!s->x[c] || !s->v[c] || !s->a[c]) return sss_set_err(ctx, SSS_ERR_ARG, "NULL particle array");
    SSS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    const long long n = s->n;
    const long long cells = (long long)M * M * M;
    int bits = 0;
    while ((1LL << bits) < cells) ++bits;
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off += (bytes + 255) & ~(size_t)255; return o; };
    const size_t o_k0 = take(8 * n), o_k1 = take(8 * n), o_v0 = take(4 * n), o_v1 = take(4 * n);
    const size_t o_src = take(32 * n);
    const size_t o_rs = take(8 * sss_dev::radix_scratch(n));
    const long long max_items = n / 32 + std::min<long long>(cells, n);
    const size_t o_items = take(8 * (size_t)max_items);
    // zero at the start, so next to one another: one memset for the four
    const size_t o_first = take(4 * cells), o_last = take(4 * cells), o_cnt = take(4 * (2 * PP_CLASSES + 1));
    const size_t o_acc = take(12 * n);
    void* scr = nullptr;
    int rc = sss_scratch(ctx, off, &scr);
    if (rc) return rc;
    char* B = (char*)scr;
    unsigned long long* k0 = (unsigned long long*)(B + o_k0);
    unsigned long long* k1 = (unsigned long long*)(B + o_k1);
    unsigned* v0 = (unsigned*)(B + o_v0);
    unsigned* v1 = (unsigned*)(B + o_v1);
    double4* src = (double4*)(B + o_src);
    int* first = (int*)(B + o_first);
    int* last = (int*)(B + o_last);
    int2* items = (int2*)(B + o_items);
    unsigned* counters = (unsigned*)(B + o_cnt);                  // items per class, cursors, work counter
    const Pm3Parts parts = pm3_parts(s);
    const double l = p->box / M;
    k_pp_keys<<<blocks_for(n, 256), 256, 0, st>>>(parts, M, 1.0 / l, k0, v0);
    SSS_LAUNCH_CHECK(ctx, "k_pp_keys");
    SSS_CUDA_TRY(ctx, sss_dev::radix_sort(k0, v0, k1, v1, n, (long long*)(B + o_rs), st, ctx->d_status, bits));
    k_pp_gather<<<blocks_for(n, 256), 256, 0, st>>>(parts, v0, src);
    SSS_LAUNCH_CHECK(ctx, "k_pp_gather");
    SSS_CUDA_TRY(ctx, cudaMemsetAsync(first, 0, off - o_first, st));
    k_pp_bounds<<<blocks_for(n, 256), 256, 0, st>>>(k0, n, first, last);
    SSS_LAUNCH_CHECK(ctx, "k_pp_bounds");
    int per_sm = 0;
    SSS_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pp_pairs, PP_WARPS * 32, 0));
    const unsigned ib = blocks_for(cells, 128);
    k_pp_items<true><<<ib, 128, 0, st>>>(first, last, M, cells, counters, counters + PP_CLASSES, items);
    SSS_LAUNCH_CHECK(ctx, "k_pp_items (count)");
    k_pp_items<false><<<ib, 128, 0, st>>>(first, last, M, cells, counters, counters + PP_CLASSES, items);
    SSS_LAUNCH_CHECK(ctx, "k_pp_items");
    PPArgs q;
    q.src = src;
    q.order = v0;
    q.first = first;
    q.last = last;
    q.M = M;
    q.l = l;
    q.box = p->box;
    q.G = G;
    q.alpha = (float)alpha;
    q.rc2 = (float)(r_cut * r_cut);
    q.eps2 = (float)(eps * eps);
    q.items = items;
    q.n_items = counters;
    q.next = counters + 2 * PP_CLASSES;
    q.acc = (float*)(B + o_acc);
    q.n = n;
    const unsigned grid = (unsigned)(ctx->num_sms * std::max(per_sm, 1));
    k_pp_pairs<<<grid, PP_WARPS * 32, 0, st>>>(q);
    SSS_LAUNCH_CHECK(ctx, "k_pp_pairs");
    Pm3Epi e{mode, hdt, dt, p->box, snap};
    k_pp_finish<<<blocks_for(n, 256), 256, 0, st>>>(q, parts, e);
    SSS_LAUNCH_CHECK(ctx, "k_pp_finish");
    return SSS_OK;
}
