// All-pairs Plummer self-gravity for sm_100a.
//
// Replaces the tiled force loop `beschleunigung` and the KDK step loop of
// `selfgrav_kernel` (reference backend/selfgrav_kernel.py:222-420).
//
// Work decomposition: a CTA owns a block of NT*R targets (R per thread, in
// registers) and one CHUNK of the source list. Source tiles are staged in
// shared memory by 1-D bulk async copies (cp.async.bulk + mbarrier, double
// buffered) and read back as broadcast loads. Chunks split the source sum so
// the grid has enough CTAs for an even load on 148 SMs; the chunk partials
// are added in ascending chunk order by the last CTA of each target block to
// arrive (arrival counted by one atomic per target block, no spinning), and
// that CTA runs the integrator epilogue: closing half kick, snapshot, next
// opening half kick and drift (the Yoshida / KDK sequence fused into the
// force kernel). Within a tile each target sums its sources in ascending
// index order, tiles in ascending order, as the reference does
// (selfgrav_kernel.py:235-256).
//
// Equal-mass tiles: when every source of a tile has the same Gm, the pair
// loop drops the mass multiply and the tile's sum is scaled by Gm once when
// it is folded into the accumulator (detected per tile, automatically).
//
// f64 path: every operation in f64; r^-3 from an f32 seed refined in f64.
// Mixed path: sources are pre-shifted per tile to the tile's bounding-box
// centre and rounded to f32; each target's offset to the centre is formed
// in f64 and rounded once per tile, so the f32 pair difference is a
// difference of small numbers. f32 pair terms are summed over sub-tiles of
// MIX_SUB sources and folded into f64 accumulators. The f32 arithmetic is
// issued as packed f32x2 instructions (two targets per instruction).

#include "allpairs.cuh"

#include <pthread.h>

namespace {

// f64 kernel: 2 targets per thread, 64 registers, 4 CTAs (32 warps) per SM
constexpr int F64_NT = 256;
constexpr int F64_R = 2;
constexpr int F64_TS = 512;     // sources per shared-memory tile (16 KiB)
constexpr int F64_MINB = 4;
constexpr int F64_UNROLL = 4;

// mixed kernel: 8 targets per thread (4 packed pairs), 2 CTAs per SM
constexpr int MIX_NT = 128;
constexpr int MIX_R = 8;
constexpr int MIX_TS = 512;     // sources per tile (32 B each, duplicated: 16 KiB)
constexpr int MIX_SUB = 128;    // f32 partial-sum length before the f64 fold
constexpr int MIX_MINB = 2;

constexpr int WAVES = 16;       // target number of CTA waves per evaluation

// warp-split kernels (use_split): 8 warps share 64 or 128 targets and split the
// CTA's sources.
constexpr int WS_W = 8;
constexpr int WS_NT = WS_W * 32;
constexpr int WS_TS = 512;      // sources per tile (mixed: the tile with one centre)
constexpr int WS_MAXCHUNKS = 16;
constexpr int WS_R_F64 = 2, WS_R_MIX = 4;
constexpr int WS_MINB_F64 = 4, WS_MINB_MIX = 2;

// lane kernels (use_lanes): a warp per target
constexpr int LN_NT = 256, LN_U = 4;

// Which form an evaluation takes. The limits are where the forms cross, over
// 1 .. 1,048,576 sources and 1 .. 1,000,000 targets (device us per evaluation
// among others).
//
// Lanes / warp-split: a warp alone walks n_src / 128 rounds, and from ~4,000
// targets on they queue for the SMs, so both counts are bounded:
//   mixed 2-D  300^2 2.5 / 5.5, 512 x 1,024 3.6 / 5.4, 1,024^2 5.7 / 5.8, 1 x 4,096 2.7 / 2.8, 1 x 16,384 5.3 / 2.8,
//              2,048 x 64 9.5 / 5.7, 65,536 x 1 225 / 36
//   f64 3-D    100 x 1,024 2.5 / 4.0, 512 x 4,096 6.8 / 8.4, 512 x 64 5.1 / 5.3, 1,024 x 64 8.8 / 5.7, 100 x 16,384 7.6 / 5.0
//
// Warp-split / general. By pairs where both counts are large:
//   mixed 3-D  10,007^2 57 / 88, 17,000^2 148 / 156, 20,000^2 199 / 207, 25,000^2 294 / 290, 40,000^2 748 / 671
//   f64 3-D    10,007^2 125 / 133, 17,000^2 316 / 326, 20,000^2 438 / 437, 30,000^2 960 / 927
// Few sources on many targets leave a CTA of 64 or 128 targets little but its fixed part, while the general form's time
// rises by the round of 148 CTAs of 1,024 (f64: 512) targets; us of both as fitted to the sweep (within 7 %):
//   mixed 2-D  1 x 65,536 5.0 / 6.1, 1 x 131,072 8.5 / 6.1, 100 x 131,072 12 / 11, 192 x 196,608 24 / 26 (two rounds),
//              500 x 300,000 67 / 61, 100 x 1,000,000 82 / 42, 512 x 262,144 56 / 57
//   f64 3-D    1 x 8,192 2.6 / 2.8, 1 x 65,536 6.1 / 2.9, 100 x 65,536 11.3 / 11.6, 100 x 1,000,000 130 / 111, 512 x 262,144 144 / 160
// Many sources on a few targets give it 16 chunks only, of sources the general form spreads over all SMs:
//   mixed 3-D  65,536 x 8 47 / 45, 131,072 x 64 91 / 82, 1,048,576 x 1 699 / 517, 131,072 x 200 92 / 94
//   f64 3-D    32,768 x 8 34 / 53, 65,536 x 64 64 / 62, 262,144 x 64 243 / 204, 262,144 x 300 244 / 262
constexpr double SPLIT_PAIRS_F64 = 3e8, SPLIT_PAIRS_MIX = 4.5e8;

constexpr bool use_lanes(bool mixed, int64_t n_src, int64_t n_tgt) {
    return (n_src <= 512 && n_tgt <= 4096) || (mixed && n_src <= 1024 && n_tgt <= 1024);
}

constexpr bool use_split(bool mixed, int dim, int64_t n_src, int64_t n_tgt) {
    const double n = (double)n_src, t = (double)n_tgt;
    if (n * t >= (mixed ? SPLIT_PAIRS_MIX : SPLIT_PAIRS_F64)) return false;
    if (n_src <= 512) {
        const double w = (double)((n_tgt + (mixed ? 151551 : 75775)) / (mixed ? 151552 : 75776));     // rounds
        const double general = mixed ? 4.8 + w * (1.1 + 0.049 * n) : 2.0 + 0.7 * w + n * (0.0615 * w + 0.006);
        const double split = mixed ? 2.0 + t * (5.0e-5 + 3.0e-7 * n) : 1.7 + t * ((dim == 3 ? 4.8e-5 : 3.7e-5) + 8.0e-7 * n);
        if (general < split) return false;
    }
    const int64_t few = !mixed || (dim == 3 && n_src >= 131072) ? 256 : 128;
    return !(n_tgt <= few && n_src >= (mixed && dim == 2 ? 98304 : 65536));
}

using sss_ap::Epi;
using sss_ap::epilogue;

struct ForceArgs {
    const double4* src;      // f64 path: sources
    const float4* srcf;      // mixed path: tile-shifted, duplicated f32 sources
    const double4* centers;  // mixed path: tile centres, .w = common Gm or NaN
    int64_t n_src;
    const double4* tgt;
    int64_t n_tgt;
    double eps2;
    int n_tiles;
    int n_chunks;
    int tiles_per_chunk;
    double4* part;           // [n_chunks][n_tgt] partial sums (n_chunks > 1)
    unsigned* counters;      // [n_target_blocks]
    int* status;
    Epi epi;
};

// Chunk partial -> (last arriving CTA) fixed-order sum -> epilogue.
template <int D, int R, int NT>
__device__ __forceinline__ void finish_block(const ForceArgs& a, int tb, int ch,
                                             const double (&ax)[R], const double (&ay)[R],
                                             const double (&az)[R]) {
    __shared__ unsigned s_last;
    const int tid = threadIdx.x;
    const int64_t tbase = (int64_t)tb * (NT * R);
    if (a.n_chunks == 1) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int64_t i = tbase + r * NT + tid;
            if (i < a.n_tgt) epilogue<D>(a.epi, i, ax[r], ay[r], az[r], a.tgt[i]);
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t i = tbase + r * NT + tid;
        if (i < a.n_tgt) {
            double2* q = reinterpret_cast<double2*>(a.part + (int64_t)ch * a.n_tgt + i);
            __stcg(q, make_double2(ax[r], ay[r]));
            __stcg(q + 1, make_double2(az[r], 0.0));
        }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const unsigned prev = atomicAdd(&a.counters[tb], 1u);
        s_last = (prev == (unsigned)(a.n_chunks - 1)) ? 1u : 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t i = tbase + r * NT + tid;
        if (i >= a.n_tgt) continue;
        double sx = 0.0, sy = 0.0, sz = 0.0;
        for (int c = 0; c < a.n_chunks; ++c) {
            const double2* q = reinterpret_cast<const double2*>(a.part + (int64_t)c * a.n_tgt + i);
            const double2 q0 = __ldcg(q), q1 = __ldcg(q + 1);
            sx += q0.x;
            sy += q0.y;
            sz += q1.x;
        }
        epilogue<D>(a.epi, i, sx, sy, sz, a.tgt[i]);
    }
    if (tid == 0) a.counters[tb] = 0u;  // ready for the next launch
}

// Wait (bounded) for copies still in flight after an abort, so the CTA does
// not exit while the async proxy writes its shared memory.
__device__ __noinline__ void drain_after_abort(uint64_t* bar, int issued, int consumed, int* status) {
    for (int k = consumed; k < issued; ++k) sss_mbar_wait_bounded(&bar[k & 1], (k >> 1) & 1, status);
}

// ------------------------------------------------------------------ f64

// r2^(-3/2), times gm unless UNIT (the equal-mass tile loop scales later):
// the series of sss_gm_rinv3 with the hardware's f64 seed. (One evaluation
// of 10,007 bodies: 126 us; 136 with an f32 seed whose argument and result
// were re-biased by integer operations. On the benchmark shape the f32 seed
// took 200 ms and CUDA's rsqrt(double) with three multiplies 246 ms.)
//
// GUARD: 0 for an r2 that overflows (distances from 1e154 on), NaN without. Only
// softenings below GUARD_EPS2, point masses, whose scenes may have any scale, take
// the guard: in every pair it took 10,007 bodies from 441 to 454 us a Yoshida step,
// and a second, guarded sum of the NaN targets alone cost as much (30,000 bodies
// 3-D: 924 -> 943 us an evaluation, by the registers of the pair loop). The
// lanes kernel, which latency bounds, always has it.
constexpr double GUARD_EPS2 = 0x1p-126;

template <bool UNIT, bool GUARD>
__device__ __forceinline__ double rinv3(double gm, double r2) {
    if (GUARD) return sss_gm_rinv3(UNIT ? 1.0 : gm, r2);
    double c;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(c) : "d"(r2));
    const double c2 = c * c;
    const double e = fma(-r2, c2, 1.0);
    const double g3 = UNIT ? c * c2 : (gm * c) * c2;
    const double p = fma(e, 1.875, 1.5);
    return fma(g3, e * p, g3);
}

template <int D, int R, bool UNIT, bool GUARD, int UNROLL>
__device__ __forceinline__ void tile_f64(const double4* __restrict__ s, int cnt, double eps2,
                                         const double (&px)[R], const double (&py)[R],
                                         const double (&pz)[R], double (&tx)[R], double (&ty)[R],
                                         double (&tz)[R]) {
#pragma unroll UNROLL
    for (int j = 0; j < cnt; ++j) {
        const double4 sj = s[j];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const double dx = sj.x - px[r];
            const double dy = sj.y - py[r];
            double r2;
            double dz = 0.0;
            if (D == 3) {
                dz = sj.z - pz[r];
                r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
            } else {
                r2 = fma(dx, dx, fma(dy, dy, eps2));
            }
            const double f = rinv3<UNIT, GUARD>(sj.w, r2);
            tx[r] = fma(f, dx, tx[r]);
            ty[r] = fma(f, dy, ty[r]);
            if (D == 3) tz[r] = fma(f, dz, tz[r]);
        }
    }
}

template <int D, int R, int NT, int TS, int MINB, int UNROLL, bool GUARD>
__global__ void __launch_bounds__(NT, MINB) k_force_f64(const ForceArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    double4* tiles = reinterpret_cast<double4*>(smem);
    __shared__ __align__(8) uint64_t bar[2];
    // chunk accumulators live in shared memory (touched once per tile), which
    // leaves the registers to the pair loop
    __shared__ double s_acc[3 * R][NT];

    const int S = a.n_chunks;
    const int tb = blockIdx.x / S;
    const int ch = blockIdx.x - tb * S;
    const int tid = threadIdx.x;
    const int64_t tbase = (int64_t)tb * (NT * R);

    double px[R], py[R], pz[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t i = tbase + r * NT + tid;
        const double4 p = (i < a.n_tgt) ? a.tgt[i] : make_double4(0.0, 0.0, 0.0, 0.0);
        px[r] = p.x; py[r] = p.y; pz[r] = p.z;
        s_acc[r][tid] = 0.0;
        s_acc[R + r][tid] = 0.0;
        s_acc[2 * R + r][tid] = 0.0;
    }

    const int t_begin = ch * a.tiles_per_chunk;
    const int t_end = min(t_begin + a.tiles_per_chunk, a.n_tiles);
    const int nt = t_end - t_begin;

    if (tid == 0) {
        sss_mbar_init(&bar[0], 1);
        sss_mbar_init(&bar[1], 1);
        sss_fence_mbar_init();
    }
    __syncthreads();

    int issued = 0;
    auto issue = [&](int k) {
        const int64_t j0 = (int64_t)(t_begin + k) * TS;
        const int cnt = (int)min((int64_t)TS, a.n_src - j0);
        const unsigned bytes = (unsigned)cnt * (unsigned)sizeof(double4);
        sss_mbar_arrive_expect_tx(&bar[k & 1], bytes);
        sss_bulk_g2s(tiles + (k & 1) * TS, a.src + j0, bytes, &bar[k & 1]);
    };
    if (tid == 0) {
        issue(0);
        issued = 1;
        if (nt > 1) { issue(1); issued = 2; }
    }

    const double eps2 = a.eps2;
    int k = 0;
    for (; k < nt; ++k) {
        const int64_t j0 = (int64_t)(t_begin + k) * TS;
        const int cnt = (int)min((int64_t)TS, a.n_src - j0);
        const bool waited = sss_mbar_wait_bounded(&bar[k & 1], (k >> 1) & 1, a.status);
        if (__syncthreads_or(!waited)) break;
        const double4* s = tiles + (k & 1) * TS;
        const double w0 = s[0].w;
        bool same = true;
        for (int j = tid; j < cnt; j += NT) same &= (s[j].w == w0);
        const bool uni = __syncthreads_and(same) != 0;
        double tx[R], ty[R], tz[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { tx[r] = 0.0; ty[r] = 0.0; tz[r] = 0.0; }
        if (uni) tile_f64<D, R, true, GUARD, UNROLL>(s, cnt, eps2, px, py, pz, tx, ty, tz);
        else tile_f64<D, R, false, GUARD, UNROLL>(s, cnt, eps2, px, py, pz, tx, ty, tz);
        const double wt = uni ? w0 : 1.0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            s_acc[r][tid] = fma(wt, tx[r], s_acc[r][tid]);
            s_acc[R + r][tid] = fma(wt, ty[r], s_acc[R + r][tid]);
            s_acc[2 * R + r][tid] = fma(wt, tz[r], s_acc[2 * R + r][tid]);
        }
        __syncthreads();
        if (tid == 0 && k + 2 < nt) { issue(k + 2); issued = k + 3; }
    }
    if (k < nt) {  // aborted on a timed-out wait
        if (tid == 0) drain_after_abort(bar, issued, k, a.status);
        return;
    }
    double ax[R], ay[R], az[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        ax[r] = s_acc[r][tid];
        ay[r] = s_acc[R + r][tid];
        az[r] = s_acc[2 * R + r][tid];
    }
    finish_block<D, R, NT>(a, tb, ch, ax, ay, az);
}

// ---------------------------------------------------------------- mixed

typedef unsigned long long f2x;   // two packed f32

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

// One CTA per tile of TS sources: bounding-box centre (f64), common Gm of
// the tile (NaN if the masses differ), and every source's f32 offset from
// the centre, duplicated {x,x,y,y},{z,z,Gm,Gm} for the packed loop
// (padding entries get Gm = 0).
template <int D, int TS>
__global__ void __launch_bounds__(256) k_prep_mixed(const double4* __restrict__ src, int64_t n_src,
                                                    float4* __restrict__ out,
                                                    double4* __restrict__ centers) {
    __shared__ double red[6][8];
    __shared__ int s_diff;
    const int tile = blockIdx.x;
    const int64_t j0 = (int64_t)tile * TS;
    if (threadIdx.x == 0) s_diff = 0;
    const double w0 = src[j0].w;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    bool diff = false;
    for (int j = threadIdx.x; j < TS; j += blockDim.x) {
        const int64_t g = j0 + j;
        if (g < n_src) {
            const double4 s = src[g];
            lo[0] = fmin(lo[0], s.x); hi[0] = fmax(hi[0], s.x);
            lo[1] = fmin(lo[1], s.y); hi[1] = fmax(hi[1], s.y);
            lo[2] = fmin(lo[2], s.z); hi[2] = fmax(hi[2], s.z);
            diff |= (s.w != w0);
        }
    }
    for (int c = 0; c < 3; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[c] = fmin(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
            hi[c] = fmax(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
        }
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (diff) s_diff = 1;
    if (l == 0) {
        for (int c = 0; c < 3; ++c) { red[c][w] = lo[c]; red[3 + c][w] = hi[c]; }
    }
    __syncthreads();
    double cen[3];
    for (int c = 0; c < 3; ++c) {
        double a = red[c][0], b = red[3 + c][0];
        for (int q = 1; q < (int)(blockDim.x >> 5); ++q) { a = fmin(a, red[c][q]); b = fmax(b, red[3 + c][q]); }
        cen[c] = (a <= b) ? 0.5 * (a + b) : 0.0;
    }
    if (D == 2) cen[2] = 0.0;
    if (threadIdx.x == 0)
        centers[tile] = make_double4(cen[0], cen[1], cen[2], s_diff ? __longlong_as_double(0x7ff8000000000000ll) : w0);
    for (int j = threadIdx.x; j < TS; j += blockDim.x) {
        const int64_t g = j0 + j;
        float x = 0.f, y = 0.f, z = 0.f, m = 0.f;
        if (g < n_src) {
            const double4 s = src[g];
            x = __double2float_rn(s.x - cen[0]);
            y = __double2float_rn(s.y - cen[1]);
            z = (D == 3) ? __double2float_rn(s.z - cen[2]) : 0.f;
            m = __double2float_rn(s.w);
        }
        out[2 * (j0 + j)] = make_float4(x, x, y, y);
        out[2 * (j0 + j) + 1] = make_float4(z, z, m, m);
    }
}

template <int D, int P, bool UNIT>
__device__ __forceinline__ void subtile_mixed(const ulonglong2* __restrict__ s, int js, int je, f2x eps2x,
                                              const f2x (&ox)[P], const f2x (&oy)[P], const f2x (&oz)[P],
                                              f2x (&fx)[P], f2x (&fy)[P], f2x (&fz)[P]) {
#pragma unroll 4
    for (int j = js; j < je; ++j) {
        const ulonglong2 xy = s[2 * j];
        const ulonglong2 zw = s[2 * j + 1];
#pragma unroll
        for (int q = 0; q < P; ++q) {
            const f2x dx = add2(xy.x, ox[q]);
            const f2x dy = add2(xy.y, oy[q]);
            f2x r2;
            f2x dz = 0ull;
            if (D == 3) {
                dz = add2(zw.x, oz[q]);
                r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, eps2x)));
            } else {
                r2 = fma2(dx, dx, fma2(dy, dy, eps2x));
            }
            float r0, r1;
            upk2(r2, r0, r1);
            const f2x inv = pk2(sss_rsqrt_approx_f32(r0), sss_rsqrt_approx_f32(r1));
            const f2x f = UNIT ? mul2(inv, mul2(inv, inv)) : mul2(mul2(zw.y, inv), mul2(inv, inv));
            fx[q] = fma2(f, dx, fx[q]);
            fy[q] = fma2(f, dy, fy[q]);
            if (D == 3) fz[q] = fma2(f, dz, fz[q]);
        }
    }
}

template <int D, int R, int NT, int TS, int SUB, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_force_mixed(const ForceArgs a) {
    static_assert(R % 2 == 0, "packed kernel needs an even target count");
    constexpr int P = R / 2;
    extern __shared__ __align__(128) unsigned char smem[];
    ulonglong2* tiles = reinterpret_cast<ulonglong2*>(smem);   // [2][TS][2]
    __shared__ __align__(8) uint64_t bar[2];

    const int S = a.n_chunks;
    const int tb = blockIdx.x / S;
    const int ch = blockIdx.x - tb * S;
    const int tid = threadIdx.x;
    const int64_t tbase = (int64_t)tb * (NT * R);

    double px[R], py[R], pz[R], ax[R], ay[R], az[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t i = tbase + r * NT + tid;
        const double4 p = (i < a.n_tgt) ? a.tgt[i] : make_double4(0.0, 0.0, 0.0, 0.0);
        px[r] = p.x; py[r] = p.y; pz[r] = p.z;
        ax[r] = 0.0; ay[r] = 0.0; az[r] = 0.0;
    }

    const int t_begin = ch * a.tiles_per_chunk;
    const int t_end = min(t_begin + a.tiles_per_chunk, a.n_tiles);
    const int nt = t_end - t_begin;

    if (tid == 0) {
        sss_mbar_init(&bar[0], 1);
        sss_mbar_init(&bar[1], 1);
        sss_fence_mbar_init();
    }
    __syncthreads();

    int issued = 0;
    constexpr unsigned kTileBytes = TS * 2 * sizeof(float4);
    const float4* srcf = a.srcf;
    auto issue = [&](int k) {
        sss_mbar_arrive_expect_tx(&bar[k & 1], kTileBytes);
        sss_bulk_g2s(tiles + (k & 1) * TS * 2, srcf + (int64_t)(t_begin + k) * TS * 2, kTileBytes, &bar[k & 1]);
    };
    if (tid == 0) {
        issue(0);
        issued = 1;
        if (nt > 1) { issue(1); issued = 2; }
    }

    const float eps2f = (float)a.eps2;
    const f2x eps2x = pk2(eps2f, eps2f);
    int k = 0;
    for (; k < nt; ++k) {
        const int tile = t_begin + k;
        const int64_t j0 = (int64_t)tile * TS;
        const int cnt = (int)min((int64_t)TS, a.n_src - j0);
        const double4 c = a.centers[tile];
        const bool uni = (c.w == c.w);   // the tile's common Gm, NaN if masses differ
        f2x ox[P], oy[P], oz[P];
#pragma unroll
        for (int q = 0; q < P; ++q) {
            ox[q] = pk2(__double2float_rn(c.x - px[2 * q]), __double2float_rn(c.x - px[2 * q + 1]));
            oy[q] = pk2(__double2float_rn(c.y - py[2 * q]), __double2float_rn(c.y - py[2 * q + 1]));
            oz[q] = (D == 3) ? pk2(__double2float_rn(c.z - pz[2 * q]), __double2float_rn(c.z - pz[2 * q + 1]))
                             : pk2(0.f, 0.f);
        }
        const bool waited = sss_mbar_wait_bounded(&bar[k & 1], (k >> 1) & 1, a.status);
        if (__syncthreads_or(!waited)) break;
        const ulonglong2* s = tiles + (k & 1) * TS * 2;
        const double wt = uni ? c.w : 1.0;
        for (int js = 0; js < cnt; js += SUB) {
            const int je = min(js + SUB, cnt);
            f2x fx[P], fy[P], fz[P];
#pragma unroll
            for (int q = 0; q < P; ++q) { fx[q] = 0ull; fy[q] = 0ull; fz[q] = 0ull; }
            if (uni) subtile_mixed<D, P, true>(s, js, je, eps2x, ox, oy, oz, fx, fy, fz);
            else subtile_mixed<D, P, false>(s, js, je, eps2x, ox, oy, oz, fx, fy, fz);
#pragma unroll
            for (int q = 0; q < P; ++q) {
                float l0, l1;
                upk2(fx[q], l0, l1);
                ax[2 * q] = fma(wt, (double)l0, ax[2 * q]);
                ax[2 * q + 1] = fma(wt, (double)l1, ax[2 * q + 1]);
                upk2(fy[q], l0, l1);
                ay[2 * q] = fma(wt, (double)l0, ay[2 * q]);
                ay[2 * q + 1] = fma(wt, (double)l1, ay[2 * q + 1]);
                if (D == 3) {
                    upk2(fz[q], l0, l1);
                    az[2 * q] = fma(wt, (double)l0, az[2 * q]);
                    az[2 * q + 1] = fma(wt, (double)l1, az[2 * q + 1]);
                }
            }
        }
        __syncthreads();
        if (tid == 0 && k + 2 < nt) { issue(k + 2); issued = k + 3; }
    }
    if (k < nt) {
        if (tid == 0) drain_after_abort(bar, issued, k, a.status);
        return;
    }
    finish_block<D, R, NT>(a, tb, ch, ax, ay, az);
}

// ----------------------------------------------- few pairs: split by warps
//
// With few bodies the kernels above leave the device idle: 3,000 targets are
// three blocks of 1,024, and cutting the sources finer only moves the time
// into the partial sums one CTA has to add. Here a CTA takes 32 R targets
// (every warp the same ones, R per lane) and its 8 warps a slice each of the
// CTA's sources, so a block of targets meets 8 sources at a time; the warps'
// sums are added through shared memory in slice order, the chunks' (at most 16)
// by the last CTA of the target block as above. Latency-bound below ~2,000
// bodies (an evaluation of 300 or 1,000 bodies: under 8.5 us a call, host
// included, against 23-55), FP32 / FP64 pipe above (3,000 sources on 23,000
// targets, 2-D mixed: 33 us against 45; 10,007 bodies, f64 3-D: 125 against 133).
// 128 registers for the mixed form, 64 for f64: 3,000^2 3-D mixed 12.3 us against
// 15.8 with 80; 3,000 x 23,000 3-D f64 89 against 103 with 80. The mixed form centres and
// rounds its tiles itself (bounding-box centre of at most 512 consecutive
// sources, as k_prep_mixed), which saves that kernel's launch.

// Block-wide bounding box of the tile's sources (f32 offsets v from the first
// one, `base`) and its centre; whether all Gm are equal.
template <int D>
__device__ __forceinline__ void ws_centre(const float (&v)[2][3], const bool (&ok)[2], bool same,
                                          const double4& base, double (&cen)[3], bool& uni) {
    __shared__ float s_box[6][WS_W];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float lo[3], hi[3];
#pragma unroll
    for (int c = 0; c < D; ++c) {
        lo[c] = fminf(ok[0] ? v[0][c] : 3e38f, ok[1] ? v[1][c] : 3e38f);
        hi[c] = fmaxf(ok[0] ? v[0][c] : -3e38f, ok[1] ? v[1][c] : -3e38f);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
            hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
        }
        if (lane == 0) { s_box[c][w] = lo[c]; s_box[3 + c][w] = hi[c]; }
    }
    uni = __syncthreads_and(same) != 0;
    cen[0] = base.x;
    cen[1] = base.y;
    cen[2] = D == 3 ? base.z : 0.0;
#pragma unroll
    for (int c = 0; c < D; ++c) {
        float l = s_box[c][0], h = s_box[3 + c][0];
#pragma unroll
        for (int q = 1; q < WS_W; ++q) { l = fminf(l, s_box[c][q]); h = fmaxf(h, s_box[3 + c][q]); }
        cen[c] += 0.5 * ((double)l + (double)h);
    }
}

// Sum over the warps (ascending slices) of acc[R][3], chunk partials, epilogue.
// red: [3][WS_W][32 R] doubles of shared memory, free to overwrite.
template <int D, int R>
__device__ __forceinline__ void ws_finish(const ForceArgs& a, int tb, int ch, double* red, const double (&ax)[R],
                                          const double (&ay)[R], const double (&az)[R]) {
    constexpr int TB = 32 * R;
    __shared__ unsigned s_last;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        red[(0 * WS_W + w) * TB + 32 * r + lane] = ax[r];
        red[(1 * WS_W + w) * TB + 32 * r + lane] = ay[r];
        if (D == 3) red[(2 * WS_W + w) * TB + 32 * r + lane] = az[r];
    }
    __syncthreads();
    const int64_t i = (int64_t)tb * TB + tid;
    const bool mine = tid < TB && i < a.n_tgt;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    if (mine) {
#pragma unroll
        for (int q = 0; q < WS_W; ++q) {
            sx += red[(0 * WS_W + q) * TB + tid];
            sy += red[(1 * WS_W + q) * TB + tid];
            if (D == 3) sz += red[(2 * WS_W + q) * TB + tid];
        }
    }
    if (a.n_chunks == 1) {
        if (mine) epilogue<D>(a.epi, i, sx, sy, sz, a.tgt[i]);
        return;
    }
    if (mine) {
        double2* q = reinterpret_cast<double2*>(a.part + (int64_t)ch * a.n_tgt + i);
        __stcg(q, make_double2(sx, sy));
        __stcg(q + 1, make_double2(sz, 0.0));
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const unsigned prev = atomicAdd(&a.counters[tb], 1u);
        s_last = (prev == (unsigned)(a.n_chunks - 1)) ? 1u : 0u;
        if (s_last) a.counters[tb] = 0u;   // ready for the next launch
    }
    __syncthreads();
    if (!s_last || !mine) return;
    __threadfence();
    double2 p0[WS_MAXCHUNKS], p1[WS_MAXCHUNKS];
#pragma unroll
    for (int c = 0; c < WS_MAXCHUNKS; ++c)
        if (c < a.n_chunks) {
            const double2* q = reinterpret_cast<const double2*>(a.part + (int64_t)c * a.n_tgt + i);
            p0[c] = __ldcg(q);
            p1[c] = __ldcg(q + 1);
        }
    sx = sy = sz = 0.0;
#pragma unroll
    for (int c = 0; c < WS_MAXCHUNKS; ++c)
        if (c < a.n_chunks) {
            sx += p0[c].x;
            sy += p0[c].y;
            sz += p1[c].x;
        }
    epilogue<D>(a.epi, i, sx, sy, sz, a.tgt[i]);
}

template <int D, int R, bool GUARD>
__global__ void __launch_bounds__(WS_NT, WS_MINB_F64) k_force_f64_ws(const ForceArgs a) {
    constexpr int TB = 32 * R;
    constexpr int RED = 3 * WS_W * TB * (int)sizeof(double), SRC = WS_TS * (int)sizeof(double4);
    __shared__ __align__(16) unsigned char smem[RED > SRC ? RED : SRC];
    double4* tile = reinterpret_cast<double4*>(smem);
    const int S = a.n_chunks, tb = blockIdx.x / S, ch = blockIdx.x - tb * S;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    double px[R], py[R], pz[R], ax[R], ay[R], az[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t i = (int64_t)tb * TB + 32 * r + lane;
        const double4 p = (i < a.n_tgt) ? a.tgt[i] : make_double4(0.0, 0.0, 0.0, 0.0);
        px[r] = p.x; py[r] = p.y; pz[r] = p.z;
        ax[r] = 0.0; ay[r] = 0.0; az[r] = 0.0;
    }
    const int64_t c0 = ch * a.n_src / S, c1 = (ch + 1) * a.n_src / S;
    for (int64_t j0 = c0; j0 < c1; j0 += WS_TS) {
        const int cnt = (int)min((int64_t)WS_TS, c1 - j0);
        const double w0 = a.src[j0].w;
        bool same = true;
        if (j0 > c0) __syncthreads();                       // the previous tile is consumed
        for (int j = tid; j < cnt; j += WS_NT) {
            const double4 v = a.src[j0 + j];
            tile[j] = v;
            same &= (v.w == w0);
        }
        const bool uni = __syncthreads_and(same) != 0;
        const int b = w * cnt / WS_W, e = (w + 1) * cnt / WS_W;
        double tx[R], ty[R], tz[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { tx[r] = 0.0; ty[r] = 0.0; tz[r] = 0.0; }
        if (uni) tile_f64<D, R, true, GUARD, F64_UNROLL>(tile + b, e - b, a.eps2, px, py, pz, tx, ty, tz);
        else tile_f64<D, R, false, GUARD, F64_UNROLL>(tile + b, e - b, a.eps2, px, py, pz, tx, ty, tz);
        const double wt = uni ? w0 : 1.0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            ax[r] = fma(wt, tx[r], ax[r]);
            ay[r] = fma(wt, ty[r], ay[r]);
            az[r] = fma(wt, tz[r], az[r]);
        }
    }
    __syncthreads();                                        // the last tile is consumed
    ws_finish<D, R>(a, tb, ch, reinterpret_cast<double*>(smem), ax, ay, az);
}

template <int D, int R>
__global__ void __launch_bounds__(WS_NT, WS_MINB_MIX) k_force_mixed_ws(const ForceArgs a) {
    static_assert(WS_TS == 2 * WS_NT, "two sources per thread and tile");
    constexpr int TB = 32 * R, P = R / 2;
    constexpr int RED = 3 * WS_W * TB * (int)sizeof(double), SRC = WS_TS * 2 * (int)sizeof(float4);
    __shared__ __align__(16) unsigned char smem[RED > SRC ? RED : SRC];
    const int S = a.n_chunks, tb = blockIdx.x / S, ch = blockIdx.x - tb * S;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    double px[R], py[R], pz[R], ax[R], ay[R], az[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t i = (int64_t)tb * TB + 32 * r + lane;
        const double4 p = (i < a.n_tgt) ? a.tgt[i] : make_double4(0.0, 0.0, 0.0, 0.0);
        px[r] = p.x; py[r] = p.y; pz[r] = p.z;
        ax[r] = 0.0; ay[r] = 0.0; az[r] = 0.0;
    }
    const float eps2f = (float)a.eps2;
    const f2x eps2x = pk2(eps2f, eps2f);
    const int64_t c0 = ch * a.n_src / S, c1 = (ch + 1) * a.n_src / S;
    for (int64_t j0 = c0; j0 < c1; j0 += WS_TS) {
        const int cnt = (int)min((int64_t)WS_TS, c1 - j0);
        const double4 base = a.src[j0];
        const double w0 = base.w;
        double4 v[2];
        float f[2][3];
        bool ok[2], same = true;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = tid + h * WS_NT;
            ok[h] = j < cnt;
            v[h] = ok[h] ? a.src[j0 + j] : make_double4(0.0, 0.0, 0.0, 0.0);
            f[h][0] = (float)(v[h].x - base.x);
            f[h][1] = (float)(v[h].y - base.y);
            f[h][2] = (float)(v[h].z - base.z);
            if (ok[h]) same &= (v[h].w == w0);
        }
        double cen[3];
        bool uni;
        ws_centre<D>(f, ok, same, base, cen, uni);               // (its barrier: the previous tile is consumed)
        float4* out = reinterpret_cast<float4*>(smem);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (ok[h]) {
                const int j = tid + h * WS_NT;
                const float x = __double2float_rn(v[h].x - cen[0]), y = __double2float_rn(v[h].y - cen[1]);
                const float z = (D == 3) ? __double2float_rn(v[h].z - cen[2]) : 0.f, m = __double2float_rn(v[h].w);
                out[2 * j] = make_float4(x, x, y, y);
                out[2 * j + 1] = make_float4(z, z, m, m);
            }
        f2x ox[P], oy[P], oz[P], fx[P], fy[P], fz[P];
#pragma unroll
        for (int q = 0; q < P; ++q) {
            ox[q] = pk2(__double2float_rn(cen[0] - px[2 * q]), __double2float_rn(cen[0] - px[2 * q + 1]));
            oy[q] = pk2(__double2float_rn(cen[1] - py[2 * q]), __double2float_rn(cen[1] - py[2 * q + 1]));
            oz[q] = (D == 3) ? pk2(__double2float_rn(cen[2] - pz[2 * q]), __double2float_rn(cen[2] - pz[2 * q + 1]))
                             : pk2(0.f, 0.f);
            fx[q] = 0ull; fy[q] = 0ull; fz[q] = 0ull;
        }
        __syncthreads();                                    // the tile is staged
        // a warp's slice is at most WS_TS / WS_W = 64 sources: one f32 partial sum (MIX_SUB = 128 above)
        const int b = w * cnt / WS_W, e = (w + 1) * cnt / WS_W;
        const ulonglong2* s = reinterpret_cast<const ulonglong2*>(smem);
        if (uni) subtile_mixed<D, P, true>(s, b, e, eps2x, ox, oy, oz, fx, fy, fz);
        else subtile_mixed<D, P, false>(s, b, e, eps2x, ox, oy, oz, fx, fy, fz);
        const double wt = uni ? w0 : 1.0;
#pragma unroll
        for (int q = 0; q < P; ++q) {
            float l0, l1;
            upk2(fx[q], l0, l1);
            ax[2 * q] = fma(wt, (double)l0, ax[2 * q]);
            ax[2 * q + 1] = fma(wt, (double)l1, ax[2 * q + 1]);
            upk2(fy[q], l0, l1);
            ay[2 * q] = fma(wt, (double)l0, ay[2 * q]);
            ay[2 * q + 1] = fma(wt, (double)l1, ay[2 * q + 1]);
            if (D == 3) {
                upk2(fz[q], l0, l1);
                az[2 * q] = fma(wt, (double)l0, az[2 * q]);
                az[2 * q + 1] = fma(wt, (double)l1, az[2 * q + 1]);
            }
        }
    }
    __syncthreads();                                        // the last tile is consumed
    ws_finish<D, R>(a, tb, ch, reinterpret_cast<double*>(smem), ax, ay, az);
}

// A warp per target, its lanes over the sources: the smallest evaluations. No
// tile, no centre, no partial sums between CTAs; a source's offset is formed
// in f64 and rounded to f32 (mixed), the f32 sums of LN_U sources a lane fold
// into f64, and the lanes meet in one butterfly. Sources of equal Gm are summed
// with weight one and Gm is applied in f64, as the tiles above do: rounded to
// f32 it would be one common factor of every force, up to 6e-8 off. Bound by
// latency (a launch, one load, n / 32 pairs, five shuffles).
template <int D, bool MIXED>
__global__ void __launch_bounds__(LN_NT) k_force_lanes(const ForceArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * (LN_NT / 32) + (threadIdx.x >> 5);
    if (i >= a.n_tgt) return;
    const double4 p = a.tgt[i];
    const float epsf = (float)a.eps2;
    const double w0 = MIXED ? a.src[0].w : 1.0;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int64_t j0 = lane; j0 < a.n_src; j0 += 32 * LN_U) {
        double4 v[LN_U];
        bool ok[LN_U];
#pragma unroll
        for (int u = 0; u < LN_U; ++u) {
            ok[u] = j0 + 32 * u < a.n_src;
            v[u] = ok[u] ? a.src[j0 + 32 * u] : make_double4(0.0, 0.0, 0.0, 0.0);
        }
        if (MIXED) {
            float fx = 0.f, fy = 0.f, fz = 0.f;
            bool uni = true;
#pragma unroll
            for (int u = 0; u < LN_U; ++u) uni &= !ok[u] || v[u].w == w0;
#pragma unroll
            for (int u = 0; u < LN_U; ++u) {
                const float dx = __double2float_rn(v[u].x - p.x), dy = __double2float_rn(v[u].y - p.y);
                const float dz = D == 3 ? __double2float_rn(v[u].z - p.z) : 0.f;
                const float r2 = D == 3 ? fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, epsf))) : fmaf(dx, dx, fmaf(dy, dy, epsf));
                const float inv = sss_rsqrt_approx_f32(ok[u] ? r2 : 1.0f);
                const float f = (ok[u] && uni ? 1.0f : __double2float_rn(v[u].w)) * ((inv * inv) * inv);  // (no source: 0)
                fx = fmaf(f, dx, fx);
                fy = fmaf(f, dy, fy);
                if (D == 3) fz = fmaf(f, dz, fz);
            }
            const double wt = uni ? w0 : 1.0;
            sx = fma(wt, (double)fx, sx);
            sy = fma(wt, (double)fy, sy);
            if (D == 3) sz = fma(wt, (double)fz, sz);
        } else {
#pragma unroll
            for (int u = 0; u < LN_U; ++u) {
                const double dx = v[u].x - p.x, dy = v[u].y - p.y, dz = D == 3 ? v[u].z - p.z : 0.0;
                const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, a.eps2)));
                const double f = rinv3<false, true>(v[u].w, ok[u] ? r2 : 1.0);
                sx = fma(f, dx, sx);
                sy = fma(f, dy, sy);
                if (D == 3) sz = fma(f, dz, sz);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
        if (D == 3) sz += __shfl_xor_sync(0xffffffffu, sz, o);
    }
    if (lane == 0) epilogue<D>(a.epi, i, sx, sy, sz, p);
}

// ------------------------------------------------------------- potential

// phi_t = -sum_s Gm_s / sqrt(|d|^2 + eps2), f64, one target per thread,
// sources through shared memory in ascending order (diagnostic path).
template <int D>
__global__ void __launch_bounds__(256) k_potential(const double4* __restrict__ src, int64_t n_src,
                                                   const double4* __restrict__ tgt, int64_t n_tgt,
                                                   double* __restrict__ phi, double eps2) {
    __shared__ double4 sh[256];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const double4 p = (i < n_tgt) ? tgt[i] : make_double4(0.0, 0.0, 0.0, 0.0);
    double acc = 0.0;
    for (int64_t j0 = 0; j0 < n_src; j0 += 256) {
        const int64_t g = j0 + threadIdx.x;
        sh[threadIdx.x] = (g < n_src) ? src[g] : make_double4(0.0, 0.0, 0.0, 0.0);
        __syncthreads();
        const int cnt = (int)min((int64_t)256, n_src - j0);
        for (int j = 0; j < cnt; ++j) {
            const double4 s = sh[j];
            const double dx = s.x - p.x, dy = s.y - p.y;
            double r2 = dx * dx + dy * dy + eps2;
            if (D == 3) { const double dz = s.z - p.z; r2 += dz * dz; }
            acc += s.w * rsqrt(r2);
        }
        __syncthreads();
    }
    if (i < n_tgt) phi[i] = -acc;
}

// -------------------------------------------------------------- integrate

// Opening half kick + drift of the first substep of a batch.
template <int D>
__global__ void k_open(const double4* __restrict__ pos, double4* __restrict__ pos_nxt,
                       double4* __restrict__ vel, const double4* __restrict__ acc, int64_t n,
                       double ko, double kd) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4 a = acc[i];
    double4 v = vel[i];
    const double4 p = pos[i];
    v.x += a.x * ko;
    v.y += a.y * ko;
    if (D == 3) v.z += a.z * ko;
    double4 q = p;
    q.x = p.x + v.x * kd;
    q.y = p.y + v.y * kd;
    if (D == 3) q.z = p.z + v.z * kd;
    vel[i] = v;
    pos_nxt[i] = q;
}

// ---------------------------------------------------------------- host side

struct Plan {
    int n_tblocks, n_tiles, n_chunks, tiles_per_chunk;
};

Plan make_plan(int64_t n_src, int64_t n_tgt, int targets_per_block, int ts, int slots) {
    Plan p;
    p.n_tblocks = (int)((n_tgt + targets_per_block - 1) / targets_per_block);
    p.n_tiles = (int)((n_src + ts - 1) / ts);
    const int64_t want = (int64_t)WAVES * slots;
    int64_t s = (want + p.n_tblocks - 1) / p.n_tblocks;
    if (s < 1) s = 1;
    if (s > p.n_tiles) s = p.n_tiles;
    p.tiles_per_chunk = (int)((p.n_tiles + s - 1) / s);
    p.n_chunks = (p.n_tiles + p.tiles_per_chunk - 1) / p.tiles_per_chunk;
    return p;
}

// Chunks per target block of a warp-split kernel: the split that takes the
// fewest rounds of CTAs times their length, a CTA's fixed part (launch,
// targets, sums over warps and chunks) counted as WS_FIXED sources; no chunk
// shorter than 8 sources a warp.
Plan make_plan_ws(int64_t n_src, int64_t n_tgt, int targets_per_block, int slots) {
    constexpr int64_t WS_FIXED = 96;
    Plan p;
    p.n_tblocks = (int)((n_tgt + targets_per_block - 1) / targets_per_block);
    p.n_tiles = p.tiles_per_chunk = 0;
    p.n_chunks = 1;
    int64_t best = -1;
    for (int64_t s = 1; s <= WS_MAXCHUNKS && (s == 1 || n_src / s >= 8 * WS_W); ++s) {
        const int64_t rounds = (p.n_tblocks * s + slots - 1) / slots;
        const int64_t cost = rounds * ((n_src + s - 1) / s + WS_FIXED + 4 * s);
        if (best < 0 || cost < best) {
            best = cost;
            p.n_chunks = (int)s;
        }
    }
    return p;
}

// The force kernel a launch uses and its launch shape.
struct KSel {
    void* fn;
    int nt, tpb, ts;
    size_t smem;       // dynamic shared memory
    int key;           // index of its cached occupancy (0 .. SSS_AP_KERNELS - 1)
    bool mixed;        // takes the tiles k_prep_mixed writes
    bool ws;           // warp-split (make_plan_ws)
    bool lanes;        // a warp per target (one chunk)
};

template <bool GUARD>
void* f64_kernel(int dim, bool ws) {
    if (ws) return dim == 3 ? (void*)k_force_f64_ws<3, WS_R_F64, GUARD> : (void*)k_force_f64_ws<2, WS_R_F64, GUARD>;
    return dim == 3 ? (void*)k_force_f64<3, F64_R, F64_NT, F64_TS, F64_MINB, F64_UNROLL, GUARD>
                    : (void*)k_force_f64<2, F64_R, F64_NT, F64_TS, F64_MINB, F64_UNROLL, GUARD>;
}

KSel select_kernel(int dim, int precision, int64_t n_src, int64_t n_tgt, double eps2) {
    KSel k;
    k.mixed = (precision == SSS_PREC_MIXED);
    k.lanes = use_lanes(k.mixed, n_src, n_tgt);
    k.ws = !k.lanes && use_split(k.mixed, dim, n_src, n_tgt);
    if (k.lanes) {
        if (k.mixed) k.fn = (dim == 3) ? (void*)k_force_lanes<3, true> : (void*)k_force_lanes<2, true>;
        else k.fn = (dim == 3) ? (void*)k_force_lanes<3, false> : (void*)k_force_lanes<2, false>;
        k.nt = LN_NT;
        k.tpb = LN_NT / 32;
        k.ts = 1;
        k.smem = 0;
        k.key = (k.mixed ? 12 : 10) + (dim == 3);
        k.mixed = false;
        return k;
    }
    const bool guard = eps2 < GUARD_EPS2;
    void* const f64 = guard ? f64_kernel<true>(dim, k.ws) : f64_kernel<false>(dim, k.ws);
    if (k.ws) {
        if (k.mixed)
            k.fn = (dim == 3) ? (void*)k_force_mixed_ws<3, WS_R_MIX> : (void*)k_force_mixed_ws<2, WS_R_MIX>;
        else
            k.fn = f64;
        k.nt = WS_NT;
        k.tpb = 32 * (k.mixed ? WS_R_MIX : WS_R_F64);
        k.ts = WS_TS;
        k.smem = 0;
        k.key = (k.mixed ? 8 : guard ? 16 : 4) + (dim == 3);      // (6 and 7: allpairs_tc.cu)
        k.mixed = false;
        return k;
    }
    if (k.mixed) {
        k.fn = (dim == 3) ? (void*)k_force_mixed<3, MIX_R, MIX_NT, MIX_TS, MIX_SUB, MIX_MINB>
                          : (void*)k_force_mixed<2, MIX_R, MIX_NT, MIX_TS, MIX_SUB, MIX_MINB>;
        k.nt = MIX_NT;
        k.tpb = MIX_NT * MIX_R;
        k.ts = MIX_TS;
        k.smem = 2 * (size_t)MIX_TS * 2 * sizeof(float4);
        k.key = 2 + (dim == 3);
        return k;
    }
    k.fn = f64;
    k.nt = F64_NT;
    k.tpb = F64_NT * F64_R;
    k.ts = F64_TS;
    k.smem = 2 * (size_t)F64_TS * sizeof(double4);
    k.key = (guard ? 14 : 0) + (dim == 3);
    return k;
}

Plan plan_of(const KSel& ks, int64_t n_src, int64_t n_tgt, int slots) {
    if (ks.lanes) return Plan{(int)((n_tgt + ks.tpb - 1) / ks.tpb), 0, 1, 0};
    return ks.ws ? make_plan_ws(n_src, n_tgt, ks.tpb, slots) : make_plan(n_src, n_tgt, ks.tpb, ks.ts, slots);
}

// Bytes of mixed-precision tile copies and tile centres for n_tiles tiles.
size_t mixed_tile_bytes(int n_tiles) { return (size_t)n_tiles * MIX_TS * 2 * sizeof(float4); }
size_t mixed_centre_bytes(int n_tiles) { return ((size_t)n_tiles * sizeof(double4) + 255) & ~(size_t)255; }

cudaError_t launch_prep(int dim, const double4* src, int64_t n_src, int n_tiles, float4* tiles,
                        double4* centres, cudaStream_t s) {
    if (dim == 3) k_prep_mixed<3, MIX_TS><<<n_tiles, 256, 0, s>>>(src, n_src, tiles, centres);
    else k_prep_mixed<2, MIX_TS><<<n_tiles, 256, 0, s>>>(src, n_src, tiles, centres);
    return cudaGetLastError();
}

// CTAs per SM of a force kernel (sets its shared-memory attribute first).
cudaError_t query_occupancy(const KSel& k, int* per_sm) {
    cudaError_t e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k.fn, k.nt, k.smem);
    *per_sm = n < 1 ? 1 : n;
    return e;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

int force_eval(sss_ctx* ctx, int dim, int precision, const double4* src, int64_t n_src,
               const double4* tgt, int64_t n_tgt, double eps2, const Epi& epi, cudaStream_t stream) {
    if (n_tgt <= 0) return SSS_OK;
    if (n_src <= 0) return sss_set_err(ctx, SSS_ERR_ARG, "all-pairs: n_src must be >= 1");
    if (n_src > ((int64_t)1 << 40) || n_tgt > ((int64_t)1 << 40))
        return sss_set_err(ctx, SSS_ERR_ARG, "all-pairs: size out of range");
    if (precision == SSS_PREC_MIXED_TC)
        return sss_ap::force_eval_tc(ctx, dim, src, n_src, tgt, n_tgt, eps2, epi, stream);
    const KSel ks = select_kernel(dim, precision, n_src, n_tgt, eps2);
    if (ctx->occ[ks.key] == 0) {
        int per_sm = 0;
        SSS_CUDA_TRY(ctx, query_occupancy(ks, &per_sm));
        ctx->occ[ks.key] = per_sm;
    }
    const int slots = ctx->occ[ks.key] * ctx->num_sms;
    const Plan pl = plan_of(ks, n_src, n_tgt, slots);

    ForceArgs a;
    memset(&a, 0, sizeof(a));
    a.src = src;
    a.n_src = n_src;
    a.tgt = tgt;
    a.n_tgt = n_tgt;
    a.eps2 = eps2;
    a.status = ctx->d_status;
    a.epi = epi;
    a.n_tiles = pl.n_tiles;
    a.n_chunks = pl.n_chunks;
    a.tiles_per_chunk = pl.tiles_per_chunk;

    // scratch: [mixed tiles][centres][partials]
    const size_t bytes_tiles = ks.mixed ? mixed_tile_bytes(pl.n_tiles) : 0;
    const size_t bytes_cent = ks.mixed ? mixed_centre_bytes(pl.n_tiles) : 0;
    const size_t bytes_part = pl.n_chunks > 1 ? (size_t)pl.n_chunks * (size_t)n_tgt * sizeof(double4) : 0;
    void* scr = nullptr;
    const size_t total = bytes_tiles + bytes_cent + bytes_part;
    if (total > 0) {
        int rc = sss_scratch(ctx, total, &scr);
        if (rc) return rc;
    }
    if (ks.mixed) {
        a.srcf = (const float4*)scr;
        a.centers = (const double4*)((char*)scr + bytes_tiles);
    }
    if (pl.n_chunks > 1) {
        a.part = (double4*)((char*)scr + bytes_tiles + bytes_cent);
        int rc = sss_counters(ctx, (size_t)pl.n_tblocks, &a.counters);
        if (rc) return rc;
    }
    if (ks.mixed) {
        cudaError_t e = launch_prep(dim, src, n_src, pl.n_tiles, (float4*)a.srcf, (double4*)a.centers, stream);
        if (e != cudaSuccess) return sss_cuda_err(ctx, e, "k_prep_mixed launch");
    }
    const unsigned grid = (unsigned)pl.n_tblocks * (unsigned)pl.n_chunks;
    void* args[] = {&a};
    SSS_CUDA_TRY(ctx, cudaLaunchKernel(ks.fn, dim3(grid), dim3(ks.nt), args, ks.smem, stream));
    return SSS_OK;
}

int check_common(sss_ctx* ctx, int dim, int precision) {
    if (!ctx) return SSS_ERR_ARG;
    if (dim != 2 && dim != 3) return sss_set_err(ctx, SSS_ERR_ARG, "dim must be 2 or 3 (got %d)", dim);
    if (precision != SSS_PREC_F64 && precision != SSS_PREC_MIXED && precision != SSS_PREC_MIXED_TC)
        return sss_set_err(ctx, SSS_ERR_ARG,
                           "precision must be SSS_PREC_F64, SSS_PREC_MIXED or SSS_PREC_MIXED_TC (got %d)", precision);
    if (cudaSetDevice(ctx->device) != cudaSuccess) return sss_set_err(ctx, SSS_ERR_CUDA, "cudaSetDevice failed");
    return SSS_OK;
}

}  // namespace

// ------------------------------------------------------------------ C ABI

extern "C" int sss_allpairs_accel(sss_ctx* ctx, int dim, int precision, const double* src4, int64_t n_src,
                                  const double* tgt4, int64_t n_tgt, double* acc4, double eps2,
                                  void* stream) {
    int rc = check_common(ctx, dim, precision);
    if (rc) return rc;
    if (n_tgt < 0 || n_src < 0) return sss_set_err(ctx, SSS_ERR_ARG, "negative size");
    if (n_tgt == 0) return SSS_OK;
    if (!src4 || !tgt4 || !acc4) return sss_set_err(ctx, SSS_ERR_ARG, "NULL pointer");
    if (!aligned16(src4) || !aligned16(tgt4) || !aligned16(acc4))
        return sss_set_err(ctx, SSS_ERR_ARG, "pointers must be 16-byte aligned");
    if (!(eps2 >= 0.0)) return sss_set_err(ctx, SSS_ERR_ARG, "eps2 must be >= 0");
    Epi e;
    memset(&e, 0, sizeof(e));
    e.mode = 0;
    e.acc = (double4*)acc4;
    return force_eval(ctx, dim, precision, (const double4*)src4, n_src, (const double4*)tgt4, n_tgt, eps2, e,
                      (cudaStream_t)stream);
}

extern "C" int sss_allpairs_potential(sss_ctx* ctx, int dim, const double* src4, int64_t n_src,
                                      const double* tgt4, int64_t n_tgt, double* phi, double eps2,
                                      void* stream) {
    int rc = check_common(ctx, dim, SSS_PREC_F64);
    if (rc) return rc;
    if (n_tgt < 0 || n_src < 0) return sss_set_err(ctx, SSS_ERR_ARG, "negative size");
    if (n_tgt == 0) return SSS_OK;
    if (!src4 || !tgt4 || !phi) return sss_set_err(ctx, SSS_ERR_ARG, "NULL pointer");
    const unsigned grid = (unsigned)((n_tgt + 255) / 256);
    if (dim == 3)
        k_potential<3><<<grid, 256, 0, (cudaStream_t)stream>>>((const double4*)src4, n_src, (const double4*)tgt4,
                                                                n_tgt, phi, eps2);
    else
        k_potential<2><<<grid, 256, 0, (cudaStream_t)stream>>>((const double4*)src4, n_src, (const double4*)tgt4,
                                                                n_tgt, phi, eps2);
    SSS_LAUNCH_CHECK(ctx, "k_potential launch");
    return SSS_OK;
}

static int check_state(sss_ctx* ctx, const sss_selfgrav_state* st) {
    if (!st) return sss_set_err(ctx, SSS_ERR_ARG, "NULL state");
    int rc = check_common(ctx, st->dim, st->precision);
    if (rc) return rc;
    if (st->n_src < 1) return sss_set_err(ctx, SSS_ERR_ARG, "state needs at least one massive body");
    if (st->n_tracer < 0) return sss_set_err(ctx, SSS_ERR_ARG, "negative tracer count");
    if (st->cur != 0 && st->cur != 1) return sss_set_err(ctx, SSS_ERR_ARG, "cur must be 0 or 1");
    if (!st->pos4[0] || !st->pos4[1] || !st->vel4 || !st->acc4) return sss_set_err(ctx, SSS_ERR_ARG, "NULL buffer");
    if (!aligned16(st->pos4[0]) || !aligned16(st->pos4[1]) || !aligned16(st->vel4) || !aligned16(st->acc4))
        return sss_set_err(ctx, SSS_ERR_ARG, "buffers must be 16-byte aligned");
    if (!(st->eps2 > 0.0)) return sss_set_err(ctx, SSS_ERR_ARG, "softening must be positive");
    return SSS_OK;
}

extern "C" int sss_selfgrav_init_accel(sss_ctx* ctx, sss_selfgrav_state* st, void* stream) {
    int rc = check_state(ctx, st);
    if (rc) return rc;
    const int64_t n_all = st->n_src + st->n_tracer;
    const double4* pos = (const double4*)st->pos4[st->cur];
    Epi e;
    memset(&e, 0, sizeof(e));
    e.mode = 0;
    e.acc = (double4*)st->acc4;
    return force_eval(ctx, st->dim, st->precision, pos, st->n_src, pos, n_all, st->eps2, e, (cudaStream_t)stream);
}

extern "C" int sss_selfgrav_step_batch(sss_ctx* ctx, sss_selfgrav_state* st, int integrator, double dt,
                                       int steps, float* snap, void* stream) {
    int rc = check_state(ctx, st);
    if (rc) return rc;
    if (steps < 1) return sss_set_err(ctx, SSS_ERR_ARG, "steps must be >= 1 (got %d)", steps);
    if (integrator != SSS_INT_KDK && integrator != SSS_INT_YOSHIDA4)
        return sss_set_err(ctx, SSS_ERR_ARG, "unknown integrator %d", integrator);
    if (!(dt == dt)) return sss_set_err(ctx, SSS_ERR_ARG, "dt is NaN");
    cudaStream_t s = (cudaStream_t)stream;
    const int D = st->dim;
    const int64_t n_all = st->n_src + st->n_tracer;
    const int64_t row = 2 * (int64_t)D * st->n_src + (int64_t)D * st->n_tracer;

    // substep weights (Yoshida 1990 fourth-order triple-jump composition)
    double w[3];
    int nsub;
    if (integrator == SSS_INT_KDK) {
        nsub = 1;
        w[0] = 1.0;
    } else {
        const double cbrt2 = cbrt(2.0);
        nsub = 3;
        w[0] = 1.0 / (2.0 - cbrt2);
        w[1] = -cbrt2 / (2.0 - cbrt2);
        w[2] = w[0];
    }

    // opening half kick + drift of the first substep
    {
        const double4* p = (const double4*)st->pos4[st->cur];
        double4* q = (double4*)st->pos4[1 - st->cur];
        const unsigned grid = (unsigned)((n_all + 255) / 256);
        if (D == 3)
            k_open<3><<<grid, 256, 0, s>>>(p, q, (double4*)st->vel4, (const double4*)st->acc4, n_all,
                                          0.5 * w[0] * dt, w[0] * dt);
        else
            k_open<2><<<grid, 256, 0, s>>>(p, q, (double4*)st->vel4, (const double4*)st->acc4, n_all,
                                          0.5 * w[0] * dt, w[0] * dt);
        SSS_LAUNCH_CHECK(ctx, "k_open launch");
        st->cur = 1 - st->cur;
    }
    for (int step = 0; step < steps; ++step) {
        for (int k = 0; k < nsub; ++k) {
            Epi e;
            memset(&e, 0, sizeof(e));
            e.mode = 1;
            e.last = (step == steps - 1 && k == nsub - 1) ? 1 : 0;
            e.acc = (double4*)st->acc4;
            e.vel = (double4*)st->vel4;
            e.pos_nxt = (double4*)st->pos4[1 - st->cur];
            e.snap = (snap && k == nsub - 1) ? snap + (int64_t)step * row : nullptr;
            e.kc = 0.5 * w[k] * dt;
            const int kn = (k + 1) % nsub;
            e.ko = 0.5 * w[kn] * dt;
            e.kd = w[kn] * dt;
            e.n_src = st->n_src;
            e.n_tr = st->n_tracer;
            const double4* pos = (const double4*)st->pos4[st->cur];
            rc = force_eval(ctx, D, st->precision, pos, st->n_src, pos, n_all, st->eps2, e, s);
            if (rc) return rc;
            st->cur = 1 - st->cur;
        }
    }
    return SSS_OK;
}

// ------------------------------------------------ no-allocation variant
//
// sss_allpairs_accel_noalloc: the all-pairs force of sss_allpairs_accel for
// callers that must not allocate device memory (see include/sss.h). Its
// scratch (status word, chunk-arrival counters, mixed-precision tiles and
// chunk partial sums) lives in the file-scope array below, which every GPU
// that loads libsss holds until the process exits. Host code reaches the
// array only through the device address cudaGetSymbolAddress returns; the
// symbol itself names a host-side stand-in.

#define SSS_NOALLOC_STATUS_BYTES 256u
#define SSS_NOALLOC_COUNTERS 16384u

static __device__ __align__(256) unsigned char g_sss_noalloc_scratch[SSS_NOALLOC_SCRATCH_BYTES];

// The stated mixed-precision source limit must be exactly what the scratch
// layout holds: whole tiles plus their 256-byte-rounded centres.
constexpr size_t noalloc_fixed_bytes(size_t n_src) {
    return ((n_src + MIX_TS - 1) / MIX_TS) * MIX_TS * 2 * sizeof(float4) +
           ((((n_src + MIX_TS - 1) / MIX_TS) * sizeof(double4) + 255) & ~(size_t)255);
}
constexpr size_t kNoAllocAvail =
    (size_t)SSS_NOALLOC_SCRATCH_BYTES - SSS_NOALLOC_STATUS_BYTES - SSS_NOALLOC_COUNTERS * sizeof(unsigned);
static_assert(noalloc_fixed_bytes(SSS_NOALLOC_MAX_MIXED_SOURCES) <= kNoAllocAvail &&
                  noalloc_fixed_bytes(SSS_NOALLOC_MAX_MIXED_SOURCES + 1) > kNoAllocAvail,
              "SSS_NOALLOC_MAX_MIXED_SOURCES does not match the no-allocation scratch layout");

namespace {

struct NoAllocDevice {
    int ready;
    unsigned char* base;  // device address of g_sss_noalloc_scratch on this device
    int num_sms;
    int occ[SSS_AP_KERNELS];   // CTAs per SM of the force kernels (KSel::key)
};

constexpr int kNoAllocMaxDevices = 64;
NoAllocDevice g_noalloc_dev[kNoAllocMaxDevices];
pthread_mutex_t g_noalloc_mu = PTHREAD_MUTEX_INITIALIZER;

int noalloc_err(char* buf, size_t len, int code, const char* fmt, ...) {
    if (buf && len) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, len, fmt, ap);
        va_end(ap);
    }
    return code;
}

// Once per device, with that device current: resolve the scratch array's
// device address and the launch parameters of the force kernels.
int noalloc_setup(int device, NoAllocDevice** out, char* eb, size_t el) {
    pthread_mutex_lock(&g_noalloc_mu);
    NoAllocDevice* d = &g_noalloc_dev[device];
    int rc = SSS_OK;
    if (!d->ready) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_sss_noalloc_scratch);
        if (e != cudaSuccess) {
            rc = noalloc_err(eb, el, SSS_ERR_CUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        } else if (((uintptr_t)p & 255u) != 0) {
            rc = noalloc_err(eb, el, SSS_ERR_CUDA, "static scratch is not 256-byte aligned");
        } else {
            d->base = (unsigned char*)p;
            e = cudaDeviceGetAttribute(&d->num_sms, cudaDevAttrMultiProcessorCount, device);
            // one size for each kind of kernel, each with and without the guard
            const int64_t probe_n[3] = {1, 16384, (int64_t)1 << 20};
            static_assert(use_lanes(true, 1, 1) && use_lanes(false, 1, 1) && !use_lanes(true, 16384, 16384) &&
                          use_split(true, 3, 16384, 16384) && use_split(false, 3, 16384, 16384) &&
                          !use_split(true, 3, 1 << 20, 1 << 20) && !use_split(false, 3, 1 << 20, 1 << 20), "probe sizes");
            for (int prec = 0; prec < 2 && e == cudaSuccess; ++prec)
                for (int dim = 2; dim <= 3 && e == cudaSuccess; ++dim)
                    for (int q = 0; q < 6 && e == cudaSuccess; ++q) {
                        const KSel ks = select_kernel(dim, prec, probe_n[q / 2], probe_n[q / 2], q % 2 ? 1.0 : 0.0);
                        e = query_occupancy(ks, &d->occ[ks.key]);
                    }
            if (e != cudaSuccess)
                rc = noalloc_err(eb, el, SSS_ERR_CUDA, "no-alloc setup: %s", cudaGetErrorString(e));
            else
                d->ready = 1;
        }
    }
    pthread_mutex_unlock(&g_noalloc_mu);
    *out = d;
    return rc;
}

}  // namespace

extern "C" int sss_allpairs_accel_noalloc(int device, int dim, int precision, const double* src4, int64_t n_src,
                                          const double* tgt4, int64_t n_tgt, double* acc4, double eps2,
                                          int* d_status, void* stream, char* errbuf, size_t errbuf_len) {
    char* eb = errbuf;
    const size_t el = errbuf_len;
    if (dim != 2 && dim != 3) return noalloc_err(eb, el, SSS_ERR_ARG, "dim must be 2 or 3 (got %d)", dim);
    if (precision != SSS_PREC_F64 && precision != SSS_PREC_MIXED)
        return noalloc_err(eb, el, SSS_ERR_ARG, "unknown precision %d", precision);
    if (n_src < 0 || n_tgt < 0) return noalloc_err(eb, el, SSS_ERR_ARG, "negative size");
    if (n_tgt == 0) return SSS_OK;
    if (n_src < 1) return noalloc_err(eb, el, SSS_ERR_ARG, "n_src must be >= 1");
    if (n_src > ((int64_t)1 << 40) || n_tgt > ((int64_t)1 << 40))
        return noalloc_err(eb, el, SSS_ERR_ARG, "size out of range");
    if (!src4 || !tgt4 || !acc4) return noalloc_err(eb, el, SSS_ERR_ARG, "NULL pointer");
    if (!aligned16(src4) || !aligned16(tgt4) || !aligned16(acc4) || ((uintptr_t)d_status & 3u))
        return noalloc_err(eb, el, SSS_ERR_ARG, "pointers must be 16-byte aligned (status 4-byte)");
    if (!(eps2 >= 0.0)) return noalloc_err(eb, el, SSS_ERR_ARG, "eps2 must be >= 0");
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || device < 0 || device >= n_dev || device >= kNoAllocMaxDevices)
        return noalloc_err(eb, el, SSS_ERR_ARG, "bad device %d", device);
    if (cudaSetDevice(device) != cudaSuccess) return noalloc_err(eb, el, SSS_ERR_CUDA, "cudaSetDevice failed");
    NoAllocDevice* d = nullptr;
    int rc = noalloc_setup(device, &d, eb, el);
    if (rc) return rc;

    const KSel ks = select_kernel(dim, precision, n_src, n_tgt, eps2);
    const int slots = d->occ[ks.key] * d->num_sms;
    Plan pl = plan_of(ks, n_src, n_tgt, slots);

    // scratch layout: [status 256 B][counters 64 KiB][tiles][centres][partials]
    const size_t data_off = SSS_NOALLOC_STATUS_BYTES + SSS_NOALLOC_COUNTERS * sizeof(unsigned);
    const size_t avail = (size_t)SSS_NOALLOC_SCRATCH_BYTES - data_off;
    const size_t bytes_tiles = ks.mixed ? mixed_tile_bytes(pl.n_tiles) : 0;
    const size_t bytes_cent = ks.mixed ? mixed_centre_bytes(pl.n_tiles) : 0;
    const size_t fixed = bytes_tiles + bytes_cent;
    // (the mixed limit holds for every mixed call, whichever kernel takes it)
    if (fixed > avail || (precision == SSS_PREC_MIXED && n_src > SSS_NOALLOC_MAX_MIXED_SOURCES))
        return noalloc_err(eb, el, SSS_ERR_CAPACITY,
                           "n_src = %lld needs %zu bytes of mixed-precision tiles; the no-allocation "
                           "scratch holds %zu (at most %d sources)", (long long)n_src, fixed, avail,
                           SSS_NOALLOC_MAX_MIXED_SOURCES);
    // narrow the source split until its partial sums fit (1 chunk needs none)
    if (pl.n_chunks > 1) {
        const size_t per_chunk = (size_t)n_tgt * sizeof(double4);
        size_t s_fit = (avail - fixed) / per_chunk;
        if (pl.n_tblocks > (int)SSS_NOALLOC_COUNTERS) s_fit = 1;
        if (s_fit < (size_t)pl.n_chunks) {
            if (ks.ws) {
                pl.n_chunks = s_fit < 1 ? 1 : (int)s_fit;
            } else if (s_fit <= 1) {
                pl.tiles_per_chunk = pl.n_tiles;
                pl.n_chunks = 1;
            } else {
                pl.tiles_per_chunk = (int)((pl.n_tiles + s_fit - 1) / s_fit);
                pl.n_chunks = (pl.n_tiles + pl.tiles_per_chunk - 1) / pl.tiles_per_chunk;
            }
        }
    }
    unsigned char* base = d->base;
    cudaStream_t s = (cudaStream_t)stream;
    int* status = d_status ? d_status : (int*)base;
    unsigned* counters = (unsigned*)(base + SSS_NOALLOC_STATUS_BYTES);
    unsigned char* data = base + data_off;

    ForceArgs a;
    memset(&a, 0, sizeof(a));
    a.src = (const double4*)src4;
    a.n_src = n_src;
    a.tgt = (const double4*)tgt4;
    a.n_tgt = n_tgt;
    a.eps2 = eps2;
    a.n_tiles = pl.n_tiles;
    a.n_chunks = pl.n_chunks;
    a.tiles_per_chunk = pl.tiles_per_chunk;
    a.status = status;
    a.epi.mode = 0;
    a.epi.acc = (double4*)acc4;
    if (ks.mixed) {
        a.srcf = (const float4*)data;
        a.centers = (const double4*)(data + bytes_tiles);
    }
    if (pl.n_chunks > 1) {
        a.part = (double4*)(data + fixed);
        a.counters = counters;
    }

    // the array keeps the previous call's contents: zero what must start at 0
    cudaError_t e = cudaSuccess;
    if (!d_status) e = cudaMemsetAsync(status, 0, sizeof(int), s);
    if (e == cudaSuccess && pl.n_chunks > 1)
        e = cudaMemsetAsync(counters, 0, (size_t)pl.n_tblocks * sizeof(unsigned), s);
    if (e != cudaSuccess) return noalloc_err(eb, el, SSS_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
    if (ks.mixed) {
        e = launch_prep(dim, a.src, n_src, pl.n_tiles, (float4*)a.srcf, (double4*)a.centers, s);
        if (e != cudaSuccess) return noalloc_err(eb, el, SSS_ERR_CUDA, "k_prep_mixed: %s", cudaGetErrorString(e));
    }
    const unsigned grid = (unsigned)pl.n_tblocks * (unsigned)pl.n_chunks;
    void* args[] = {&a};
    e = cudaLaunchKernel(ks.fn, dim3(grid), dim3(ks.nt), args, ks.smem, s);
    if (e != cudaSuccess) return noalloc_err(eb, el, SSS_ERR_CUDA, "force kernel: %s", cudaGetErrorString(e));
    return SSS_OK;
}
