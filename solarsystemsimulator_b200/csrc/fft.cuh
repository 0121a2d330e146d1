// Block-level complex FFTs for the particle meshes (pm.cu in f64, pm3d.cu in
// f32): one or several transforms of the same length held by a CTA, so that
// the passes around a transform (zero padding, the Green's function, packing
// of real rows) happen while the data is in registers.
//
// Stockham stages of radix 16, 8, 5, 4, 3, 2 over shared memory: every thread
// holds up to FFT_E = 16 complex values (one radix-16 butterfly, two of radix
// 8, ...), a stage reads its inputs, the CTA synchronises, and the outputs go
// back to the same buffer. The first stage reads through a functor and the
// last one writes through a functor, so a transform of length 4096 crosses
// shared memory twice. Twiddles come from per-stage tables, [t - 1][k] with k
// contiguous, rounded once from long double. The length is a template
// parameter: with a runtime length and one code path for all radices the
// compiler spilled (4.7 KB of stack), with a fixed one every address but the
// thread's own is an immediate.
#pragma once

#include "sss_internal.cuh"

#include <cmath>
#include <cstdlib>

constexpr int FFT_E = 16;              // complex values per thread

// Stage s of length n = 2^a 3^b 5^c: its radix (1: no such stage). Powers of
// two come first: the strided writes of the first stages then fall on the
// padded layout.
constexpr int fft_radix(int n, int s) {
    int a = 0;
    while (n % 2 == 0) { n /= 2; ++a; }
    while (a > 0) {
        const int q = a == 5 ? 3 : a >= 4 ? 4 : a;     // 32 = 8 * 4
        if (s-- == 0) return 1 << q;
        a -= q;
    }
    while (n % 5 == 0) { n /= 5; if (s-- == 0) return 5; }
    while (n % 3 == 0) { n /= 3; if (s-- == 0) return 3; }
    return 1;
}
constexpr int fft_span(int n, int s) {                 // product of the radices before stage s
    int q = 1;
    for (int k = 0; k < s; ++k) q *= fft_radix(n, k);
    return q;
}
constexpr int fft_stages(int n) {
    int s = 0;
    while (fft_radix(n, s) > 1) ++s;
    return s;
}
constexpr int fft_off(int n, int s) {                  // stage s's twiddles in the table
    int q = 0;
    for (int k = 1; k < s; ++k) q += (fft_radix(n, k) - 1) * fft_span(n, k);
    return q;
}
// Threads that `batch` transforms of length n need.
constexpr int fft_threads(int n, int batch) {
    int nt = 0;
    for (int s = 0; s < fft_stages(n); ++s) {
        const int r = fft_radix(n, s), per = FFT_E / r;
        const int need = (n / r * batch + per - 1) / per;
        nt = need > nt ? need : nt;
    }
    return (nt + 31) / 32 * 32;
}

// Twiddle table of length n in device memory (freed by the owner, also after an
// error). Complete on return: a pageable copy may return before its data has
// arrived, and the transforms run on streams that do not wait for the default one.
template <class C>
cudaError_t fft_table(int n, C** out) {
    *out = nullptr;
    const int size = fft_off(n, fft_stages(n));
    C* tw = (C*)malloc((size_t)size * sizeof(C));
    if (!tw) return cudaErrorMemoryAllocation;
    const long double pi = 3.14159265358979323846264338327950288L;
    int q = 0;
    for (int s = 1; s < fft_stages(n); ++s) {
        const int r = fft_radix(n, s), span = fft_span(n, s);
        for (int t = 1; t < r; ++t)
            for (int k = 0; k < span; ++k, ++q) {
                const long double a = -2.0L * pi * (long double)(t * k) / (long double)(span * r);
                tw[q].x = (decltype(tw[q].x))cosl(a);
                tw[q].y = (decltype(tw[q].y))sinl(a);
            }
    }
    cudaError_t e = cudaMalloc(out, (size_t)size * sizeof(C));
    if (e == cudaSuccess) e = cudaMemcpy(*out, tw, (size_t)size * sizeof(C), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
    free(tw);
    return e;
}

namespace fft {

template <class C> __device__ __forceinline__ C add(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <class C> __device__ __forceinline__ C sub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <class C> __device__ __forceinline__ C mul(C a, C b) {
    C r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
// a * conj(b)
template <class C> __device__ __forceinline__ C mulc(C a, C b) {
    C r;
    r.x = a.x * b.x + a.y * b.y;
    r.y = a.y * b.x - a.x * b.y;
    return r;
}
// a * (c - i s) forward, a * (c + i s) inverse
template <int DIR, class C, class R> __device__ __forceinline__ C rot(C a, R c, R s) {
    C r;
    if (DIR < 0) { r.x = a.x * c + a.y * s; r.y = a.y * c - a.x * s; }
    else { r.x = a.x * c - a.y * s; r.y = a.y * c + a.x * s; }
    return r;
}
// a * (-i) forward, a * (+i) inverse
template <int DIR, class C> __device__ __forceinline__ C quarter(C a) {
    C r;
    if (DIR < 0) { r.x = a.y; r.y = -a.x; }
    else { r.x = -a.y; r.y = a.x; }
    return r;
}

template <int DIR, class C> __device__ __forceinline__ void dft2(C& a, C& b) {
    const C s = add(a, b);
    b = sub(a, b);
    a = s;
}
template <int DIR, class C> __device__ __forceinline__ void dft4(C& a, C& b, C& c, C& d) {
    const C s0 = add(a, c), s1 = sub(a, c), s2 = add(b, d), s3 = quarter<DIR>(sub(b, d));
    a = add(s0, s2);
    b = add(s1, s3);
    c = sub(s0, s2);
    d = sub(s1, s3);
}

// In-place DFT of R values, natural order in and out.
template <int R, int DIR, class C> __device__ __forceinline__ void dft(C* v) {
    using T = decltype(v[0].x);
    if constexpr (R == 2) {
        dft2<DIR>(v[0], v[1]);
    } else if constexpr (R == 3) {
        const T h = (T)0.86602540378443864676372317075293618;
        const C s = add(v[1], v[2]), d = quarter<DIR>(sub(v[1], v[2]));
        C m;
        m.x = v[0].x - (T)0.5 * s.x;
        m.y = v[0].y - (T)0.5 * s.y;
        v[0] = add(v[0], s);
        v[1].x = m.x + h * d.x; v[1].y = m.y + h * d.y;
        v[2].x = m.x - h * d.x; v[2].y = m.y - h * d.y;
    } else if constexpr (R == 4) {
        dft4<DIR>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 5) {
        const T c1 = (T)0.30901699437494742410229341718281906, c2 = (T)-0.80901699437494742410229341718281906;
        const T s1 = (T)0.95105651629515357211643933337938214, s2 = (T)0.58778525229247312916870595463907277;
        const C p1 = add(v[1], v[4]), p2 = add(v[2], v[3]);
        const C m1 = quarter<DIR>(sub(v[1], v[4])), m2 = quarter<DIR>(sub(v[2], v[3]));
        C a, b, e, f;
        a.x = v[0].x + c1 * p1.x + c2 * p2.x; a.y = v[0].y + c1 * p1.y + c2 * p2.y;
        b.x = v[0].x + c2 * p1.x + c1 * p2.x; b.y = v[0].y + c2 * p1.y + c1 * p2.y;
        e.x = s1 * m1.x + s2 * m2.x; e.y = s1 * m1.y + s2 * m2.y;
        f.x = s2 * m1.x - s1 * m2.x; f.y = s2 * m1.y - s1 * m2.y;
        v[0] = add(v[0], add(p1, p2));
        v[1] = add(a, e);
        v[2] = add(b, f);
        v[3] = sub(b, f);
        v[4] = sub(a, e);
    } else if constexpr (R == 8) {
        const T q = (T)0.70710678118654752440084436210484904;
        C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft4<DIR>(e[0], e[1], e[2], e[3]);
        dft4<DIR>(o[0], o[1], o[2], o[3]);
        o[1] = rot<DIR>(o[1], q, q);
        o[2] = quarter<DIR>(o[2]);
        o[3] = rot<DIR>(o[3], -q, q);
#pragma unroll
        for (int k = 0; k < 4; ++k) { v[k] = add(e[k], o[k]); v[k + 4] = sub(e[k], o[k]); }
    } else {
        static_assert(R == 16, "radix");
        const T q = (T)0.70710678118654752440084436210484904;
        const T c = (T)0.92387953251128675612818318939678829, s = (T)0.38268343236508977172845998403039887;
        // X[k1 + 4 k2] = sum_b W16^(b k1) W4^(b k2) sum_a x[4 a + b] W4^(a k1)
        C y[4][4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            y[b][0] = v[b]; y[b][1] = v[4 + b]; y[b][2] = v[8 + b]; y[b][3] = v[12 + b];
            dft4<DIR>(y[b][0], y[b][1], y[b][2], y[b][3]);
        }
        y[1][1] = rot<DIR>(y[1][1], c, s);
        y[1][2] = rot<DIR>(y[1][2], q, q);
        y[1][3] = rot<DIR>(y[1][3], s, c);
        y[2][1] = rot<DIR>(y[2][1], q, q);
        y[2][2] = quarter<DIR>(y[2][2]);
        y[2][3] = rot<DIR>(y[2][3], -q, q);
        y[3][1] = rot<DIR>(y[3][1], s, c);
        y[3][2] = rot<DIR>(y[3][2], -q, q);
        y[3][3] = rot<DIR>(y[3][3], -c, -s);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            dft4<DIR>(y[0][k], y[1][k], y[2][k], y[3][k]);
            v[k] = y[0][k]; v[k + 4] = y[1][k]; v[k + 8] = y[2][k]; v[k + 12] = y[3][k];
        }
    }
}

// How a CTA's transforms lie in shared memory and on its threads: work item w
// of a stage with NB butterflies per transform is butterfly j of transform c.
struct One {                           // one transform
    static constexpr int batch = 1;
    template <int NB> __device__ __forceinline__ static void split(int w, int& j, int& c) { j = w; c = 0; }
    __device__ __forceinline__ static int at(int i, int) { return i + (i >> 4); }
};
template <int COUNT>
struct Inner {                         // COUNT transforms, the transform index fastest
    static constexpr int batch = COUNT;
    template <int NB> __device__ __forceinline__ static void split(int w, int& j, int& c) { j = w / COUNT; c = w % COUNT; }
    __device__ __forceinline__ static int at(int i, int c) { return i * COUNT + c; }
};
template <int COUNT, int STRIDE>
struct Outer {                         // COUNT transforms one after another, STRIDE values apart
    static constexpr int batch = COUNT;
    template <int NB> __device__ __forceinline__ static void split(int w, int& j, int& c) { c = w / NB; j = w % NB; }
    __device__ __forceinline__ static int at(int i, int c) { return c * STRIDE + i + (i >> 4); }
};

// Stage S of length N: `get(i, c, hi)` reads input i of transform c, `put(i, c,
// v, hi)` writes output i; hi = (i >= N / 2), a constant of the unrolled code in
// the first and the last stage where the radix is even. INPLACE: the inputs are
// in the buffer that the outputs go to.
template <int N, int S, int DIR, class Map, bool INPLACE, class C, class Get, class Put>
__device__ __forceinline__ void stage(const C* __restrict__ tw, Get get, Put put) {
    constexpr int R = fft_radix(N, S), B = FFT_E / R, NB = N / R, SPAN = fft_span(N, S);
    constexpr int ITEMS = NB * Map::batch, NT = fft_threads(N, Map::batch);
    // opaque to the compiler: it would otherwise keep the addresses of all stages in registers
    // across the loops around them
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    C v[B * R];
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const int w = tid + b * NT;
        if (b * NT >= ITEMS || ((b + 1) * NT > ITEMS && w >= ITEMS)) continue;
        int j, c;
        Map::template split<NB>(w, j, c);
#pragma unroll
        for (int t = 0; t < R; ++t) v[b * R + t] = get(j + t * NB, c, S == 0 && R % 2 == 0 ? 2 * t >= R : 2 * (j + t * NB) >= N);
    }
    if (INPLACE) __syncthreads();
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const int w = tid + b * NT;
        if (b * NT >= ITEMS || ((b + 1) * NT > ITEMS && w >= ITEMS)) continue;
        int j, c;
        Map::template split<NB>(w, j, c);
        const int k = j % SPAN;
        if (S > 0) {
            // f64: the powers 1, 2, 4, 8 of the butterfly's twiddle from the table, the others as
            // their products (at most three factors): 15 loads of radix 16 were more L1
            // traffic than the exchange itself. f32: all from the table, as exact as it is
            const C* q = tw + fft_off(N, S) + k;
            C f[R];
#pragma unroll
            for (int t = 1; t < R; ++t) {
                const int top = t >= 8 ? 8 : t >= 4 ? 4 : t >= 2 ? 2 : 1;
                f[t] = t == top || sizeof(C) == 8 ? __ldg(q + (t - 1) * SPAN) : mul(f[top], f[t - top]);
                v[b * R + t] = DIR < 0 ? mul(v[b * R + t], f[t]) : mulc(v[b * R + t], f[t]);
            }
        }
        dft<R, DIR>(v + b * R);
        const int o = (j - k) * R + k;
#pragma unroll
        for (int t = 0; t < R; ++t)
            put(o + t * SPAN, c, v[b * R + t], SPAN * R == N && R % 2 == 0 ? 2 * t >= R : 2 * (o + t * SPAN) >= N);
    }
}

template <int N, int S, int DIR, class Map, class C, class Put>
__device__ __forceinline__ void stages(const C* __restrict__ tw, C* sm, Put put) {
    auto rd = [&](int i, int c, bool) { return sm[Map::at(i, c)]; };
    if constexpr (S + 1 == fft_stages(N)) {
        stage<N, S, DIR, Map, true>(tw, rd, put);
    } else {
        stage<N, S, DIR, Map, true>(tw, rd, [&](int i, int c, C v, bool) { sm[Map::at(i, c)] = v; });
        __syncthreads();
        stages<N, S + 1, DIR, Map>(tw, sm, put);
    }
}

// The transforms of length N (at least two stages) of one CTA of
// fft_threads(N, Map::batch) threads: DIR -1 forward, +1 inverse (unscaled).
// `sm` holds Map::at() of every element; earlier reads of it by other threads
// must lie before a __syncthreads() of the caller. Outputs that `put` writes
// to `sm` are safe: all inputs of the last stage have been read. INPLACE: `get`
// reads `sm` too.
template <int N, int DIR, class Map, bool INPLACE = false, class C, class Get, class Put>
__device__ __forceinline__ void run(const C* __restrict__ tw, C* sm, Get get, Put put) {
    static_assert(fft_stages(N) >= 2, "one stage only");
    stage<N, 0, DIR, Map, INPLACE>(tw, get, [&](int i, int c, C v, bool) { sm[Map::at(i, c)] = v; });
    __syncthreads();
    stages<N, 1, DIR, Map>(tw, sm, put);
}

}  // namespace fft
