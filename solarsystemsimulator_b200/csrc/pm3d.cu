// 3-D periodic particle mesh for sm_100a: the reference's PM cycle
// (TODO.md:225-253: deposit, Poisson solve in Fourier space, interpolation
// with the deposit's stencil; 2-D code pm_kernel.py:63-154) on an n^3 f32
// mesh in a periodic box.
//
//   deposit  : CIC, positions f64, weights f32, warp-aggregated atomics:
//              lanes of a warp whose particles share a cell add their
//              weights in registers first and one lane issues the atomics.
//   solve    : real transform, Green's function -4 pi G / k^2 (divided by the
//              CIC window W(k)^deconv, 2: deposit and gather, and filtered by
//              exp(-k^2 r_split^2)), spectral gradient a_d = -i k_d phi with
//              the 1/n^3 of the inverse transform, three inverse transforms.
//              Mesh sides 2^a and 3 2^a from 32 to 512 take five passes over
//              the block transforms of fft.cuh: z forward (two rows as one
//              complex transform), y forward, x forward + Green's function +
//              x inverse, y inverse, z inverse. The gradient's factor along an
//              axis is applied when that axis is transformed back, so the x
//              pass writes two spectra (phi and i k_x phi) and only the y pass
//              makes three of them: 18 mesh passes of memory where R2C, the
//              spectrum kernel and a batched C2R moved 36. Other sides: cuFFT
//              for the transforms around k_spectrum3.
//   gather   : trilinear (CIC) interpolation of the three f32 meshes into
//              f64 accelerations, fused with the KDK epilogue.
//
// HBM per step at 1,048,576 particles on 256^3: deposit reads 24 B per
// particle and makes 8 atomic f32 updates, the gather reads 24 B per particle plus 24 f32 mesh values
// (L2-resident for a 64 MiB mesh) and writes the state.

#include "pm3d.cuh"
#include "fft.cuh"

#include <algorithm>

namespace {

unsigned blocks_for(long long n, int nt) { return (unsigned)((n + nt - 1) / nt); }

int cufft_err(sss_ctx* ctx, cufftResult r, const char* what) {
    return sss_set_err(ctx, SSS_ERR_CUDA, "%s: cuFFT error %d", what, (int)r);
}

constexpr unsigned FULL = 0xffffffffu;

// Sum of v over the lanes in `peers` (this lane's group, lane order); all 32
// lanes must call it with their own group and the warp's largest group
// size `most`.
__device__ __forceinline__ float group_sum(unsigned peers, unsigned most, float v) {
    const int lane = threadIdx.x & 31;
    float sum = 0.0f;
    unsigned rest = peers;
    for (unsigned k = 0; k < most; ++k) {
        const int src = rest ? __ffs(rest) - 1 : lane;
        const float o = __shfl_sync(FULL, v, src);
        if (rest) {
            sum += o;
            rest &= rest - 1;
        }
    }
    return sum;
}

// Warp-aggregated CIC deposit. Lanes whose particles lie in the same cell
// share all 8 corner nodes: one __match_any_sync on the cell finds them, the
// group's weights are added in registers (lane order) and its lowest lane
// issues one atomic per corner. Particles of different cells that share a
// node still add separately (atomics keep that correct).
__global__ void __launch_bounds__(256) k_deposit3(const Pm3Parts s, int n, double inv_h, double inv_h3,
                                                  float* __restrict__ rho) {
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    for (long long base = w0 * 32; base < s.n; base += warps * 32) {
        const long long p = base + lane;
        const bool ok = p < s.n;
        int i[3] = {0, 0, 0};
        double t[3] = {0.0, 0.0, 0.0};
        double mass = 0.0;
        if (ok) {
            for (int c = 0; c < 3; ++c) pm3_cell(s.x[c][p], inv_h, n, i[c], t[c]);
            mass = (s.m ? s.m[p] : s.mass_const) * inv_h3;
        }
        const int cell = ok ? (i[0] * n + i[1]) * n + i[2] : -1;
        const unsigned peers = __match_any_sync(FULL, cell);
        const bool leader = ok && (__ffs(peers) - 1) == lane;
        const unsigned most = __reduce_max_sync(FULL, (unsigned)__popc(peers));
        const int j[3] = {i[0] + 1 == n ? 0 : i[0] + 1, i[1] + 1 == n ? 0 : i[1] + 1, i[2] + 1 == n ? 0 : i[2] + 1};
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int dx = c >> 2, dy = (c >> 1) & 1, dz = c & 1;
            const double w = (dx ? t[0] : 1.0 - t[0]) * (dy ? t[1] : 1.0 - t[1]) * (dz ? t[2] : 1.0 - t[2]);
            float v = (float)(mass * w);
            if (most > 1) v = group_sum(peers, most, v);
            if (leader) {
                const int key = ((dx ? j[0] : i[0]) * n + (dy ? j[1] : i[1])) * n + (dz ? j[2] : i[2]);
                atomicAdd(rho + key, v);
            }
        }
    }
}

// Per-axis tables of the spectrum kernel, index i of a full axis (frequency
// f = i for i < n/2, i - n otherwise): kd = k_i (0 on the Nyquist index:
// the derivative of that mode is dropped so the spectra stay Hermitian),
// k2 = k_i^2, fac = sinc(pi f / n)^(-2 deconv) * exp(-k_i^2 rs2), then kd as
// the sum of two f32. The
// Green's function factorises: W(k)^-deconv e^{-k^2 rs2} = fac_x fac_y fac_z.
// The half axis of the real transform (iz <= n/2) reads the same tables.
__global__ void k_spectrum_tables(int n, double box, int deconv, double rs2, double* __restrict__ tab) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int f = i < n / 2 ? i : i - n;
    const double k = 2.0 * 3.14159265358979323846 / box * f;
    double fac = 1.0;
    if (f != 0) {
        const double a = (double)f / (double)n;
        const double sinc = sinpi(a) / (3.14159265358979323846 * a);
        const double s2 = sinc * sinc;
        for (int q = 0; q < deconv; ++q) fac /= s2;
    }
    if (rs2 > 0.0) fac *= exp(-k * k * rs2);
    const double kd = (i == n / 2) ? 0.0 : k;
    tab[i] = kd;
    reinterpret_cast<float2*>(tab + 3 * n)[i] = make_float2((float)kd, (float)(kd - (double)(float)kd));
    tab[n + i] = k * k;
    tab[2 * n + i] = fac;
}

// Acceleration spectra from the density spectrum (half-complex layout,
// index (ix, iy, iz), iz in [0, n/2]); grid (z blocks, n, n):
// a_d = -i k_d phi, phi = -4 pi G rho_k fac / k^2  ->  a_d = i k_d c rho_k
// with c = 4 pi G fac / (k^2 n^3) (the inverse transform's 1/n^3 folded in).
__global__ void __launch_bounds__(128) k_spectrum3(const float2* __restrict__ rk, int n, double cscale,
                                                   const double* __restrict__ tab, float2* __restrict__ ak) {
    const int nh = n / 2 + 1;
    const int iz = blockIdx.x * blockDim.x + threadIdx.x;
    if (iz >= nh) return;
    const int iy = blockIdx.y, ix = blockIdx.z;
    const long long m = (long long)n * n * nh;
    const long long t = ((long long)ix * n + iy) * nh + iz;
    float2 out[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if (ix != 0 || iy != 0 || iz != 0) {
        const double* kd = tab;
        const double* k2t = tab + n;
        const double* fac = tab + 2 * n;
        const double k2 = k2t[ix] + k2t[iy] + k2t[iz];
        const double c = cscale * (fac[ix] * fac[iy] * fac[iz]) / k2;
        const float2 r = rk[t];
        const double kk[3] = {kd[ix], kd[iy], kd[iz]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double f = kk[d] * c;
            out[d] = make_float2((float)(-f * (double)r.y), (float)(f * (double)r.x));
        }
    }
    ak[t] = out[0];
    ak[m + t] = out[1];
    ak[2 * m + t] = out[2];
}

// ------------------------------------------------------- solve, own FFTs

// Values per row of the half spectra: n / 2 + 1 rounded up to a 32-byte sector (rows of 1032 bytes
// shared sectors between CTAs).
__host__ __device__ constexpr int pitch_of(int n) { return (n / 2 + 4) / 4 * 4; }

// The transforms along y or x of one half-complex mesh, 16 to a CTA: 16
// neighbouring z of one plane (128-byte rows), the nh % 16 last z of several
// planes together (nh = n / 2 + 1: one z a plane would leave 15 idle).
template <int N>
struct Tile16 {
    static constexpr int NH = N / 2 + 1, PITCH = pitch_of(N), FULL_T = NH / 16, REST = NH % 16, TILES = N * FULL_T + N * REST / 16;
    static_assert(N % 16 == 0, "mesh side");
    using Map = fft::Inner<16>;
    static constexpr int NT = fft_threads(N, 16);
    static constexpr size_t SMEM = (size_t)N * 16 * sizeof(float2);
    int plane, iz;
    __device__ __forceinline__ Tile16() {
        const int b = blockIdx.x, c = threadIdx.x & 15;
        if (b < N * FULL_T) {
            plane = b / (FULL_T > 0 ? FULL_T : 1);
            iz = (b - plane * FULL_T) * 16 + c;
        } else {
            const int u = (b - N * FULL_T) * 16 + c;
            plane = u / (REST > 0 ? REST : 1);
            iz = FULL_T * 16 + u - plane * REST;
        }
    }
};

// 16 pairs of rows along z
template <int N>
struct Rows16 {
    static constexpr int NH = N / 2 + 1, PITCH = pitch_of(N), STRIDE = N + N / 16, TILES = N * N / 32;
    using Map = fft::Outer<16, STRIDE>;
    static constexpr int NT = fft_threads(N, 16);
    static constexpr size_t SMEM = (size_t)16 * STRIDE * sizeof(float2);
};

template <int N>
__global__ void __launch_bounds__(Rows16<N>::NT, 1024 / Rows16<N>::NT)
k_z_fwd(const float2* __restrict__ tw, const float* __restrict__ rho, float2* __restrict__ rk) {
    using R = Rows16<N>;
    using Map = typename R::Map;
    extern __shared__ float2 smf[];
    const long long row0 = (long long)blockIdx.x * 32;
    const float* src = rho + row0 * N;
    fft::run<N, -1, Map>(tw, smf,
                         [&](int i, int c, bool) { return make_float2(__ldg(src + 2 * c * N + i), __ldg(src + (2 * c + 1) * N + i)); },
                         [&](int i, int c, float2 z, bool) { smf[Map::at(i, c)] = z; });
    __syncthreads();
    float2* dst = rk + row0 * R::PITCH;
    for (int q = threadIdx.x; q < 16 * R::NH; q += R::NT) {
        const int c = q / R::NH, k = q - c * R::NH;
        const float2 z = smf[Map::at(k, c)], w = smf[Map::at(k == 0 ? 0 : N - k, c)];
        dst[(2 * c) * R::PITCH + k] = make_float2(0.5f * (z.x + w.x), 0.5f * (z.y - w.y));
        dst[(2 * c + 1) * R::PITCH + k] = make_float2(0.5f * (z.y + w.y), 0.5f * (w.x - z.x));
    }
}

template <int N>
__global__ void __launch_bounds__(Tile16<N>::NT, 1024 / Tile16<N>::NT) k_y_fwd(const float2* __restrict__ tw, float2* rk) {
    using T = Tile16<N>;
    extern __shared__ float2 smf[];
    const T t;
    float2* p = rk + (long long)t.plane * N * T::PITCH + t.iz;
    fft::run<N, -1, typename T::Map>(tw, smf, [&](int i, int, bool) { return p[i * T::PITCH]; },
                                     [&](int i, int, float2 z, bool) { p[i * T::PITCH] = z; });
}

// k (f64) z rounded once, as the products of k_spectrum3, from k = hi + lo in two
// f32: hi z = p + e exactly, so p + (e + lo z) is within 2^-46 of k z before its
// rounding (Dekker, "A floating-point technique for extending the available
// precision", 1971). A 256^3 solve takes 331 us; 360 in f64 with its conversions,
// 335 with k rounded to f32 (512^3: 3,020, 3,268, 2,992).
__device__ __forceinline__ float times_k(float2 k, float z) {
    const float p = __fmul_rn(k.x, z);
    return __fadd_rn(p, __fmaf_rn(k.y, z, __fmaf_rn(k.x, z, -p)));
}
__device__ __forceinline__ float2 times_ik(float2 k, float2 z) {
    return make_float2(-times_k(k, z.y), times_k(k, z.x));
}
__device__ __forceinline__ const float2* split_k(const double* tab, int n) {
    return reinterpret_cast<const float2*>(tab + 3 * n);
}

// a_x = i k_x c rho_k and phi' = c rho_k (c as in k_spectrum3), both inverse
// transformed along x; plane = iy.
template <int N>
__global__ void __launch_bounds__(Tile16<N>::NT, 1024 / Tile16<N>::NT)
k_x_solve(const float2* __restrict__ tw, const float2* __restrict__ rk, double cscale, const double* __restrict__ tab,
          float2* __restrict__ ax, float2* __restrict__ phi) {
    using T = Tile16<N>;
    using Map = typename T::Map;
    extern __shared__ float2 smf[];
    float2* sp = smf + N * 16;
    const T t;
    const long long o = (long long)t.plane * T::PITCH + t.iz;
    constexpr int ST = N * T::PITCH;
    const double k2yz = tab[N + t.plane] + tab[N + t.iz];
    const double cyz = cscale * (tab[2 * N + t.plane] * tab[2 * N + t.iz]);
    const bool mean = t.plane == 0 && t.iz == 0;
    fft::run<N, -1, Map>(tw, smf, [&](int i, int, bool) { return __ldg(rk + o + i * ST); },
                         [&](int i, int c, float2 r, bool) {
                             float2 a = make_float2(0.f, 0.f), b = a;
                             if (!mean || i != 0) {
                                 const double q = cyz * __ldg(tab + 2 * N + i) * sss_recip_f64(k2yz + __ldg(tab + N + i));
                                 const double f = __ldg(tab + i) * q;
                                 a = make_float2((float)(-f * (double)r.y), (float)(f * (double)r.x));
                                 b = make_float2((float)(q * (double)r.x), (float)(q * (double)r.y));
                             }
                             smf[Map::at(i, c)] = a;
                             sp[Map::at(i, c)] = b;
                         });
    __syncthreads();
#pragma unroll 1
    for (int d = 0; d < 2; ++d) {
        float2* buf = d ? sp : smf;
        float2* out = (d ? phi : ax) + o;
        fft::run<N, 1, Map, true>(tw, buf, [&](int i, int c, bool) { return buf[Map::at(i, c)]; },
                                  [&](int i, int, float2 z, bool) { out[i * ST] = z; });
    }
}

// Along y, component blockIdx.y of a_x (in place), phi -> a_y = i k_y phi (the
// density spectrum's buffer, free by now) and phi itself for the third one (its
// k_z comes with the z pass); plane = ix. The three are blocks of their own: one
// block after another on the same tile, a 64^3 pass took 9 us.
template <int N>
__global__ void __launch_bounds__(Tile16<N>::NT, 1024 / Tile16<N>::NT)
k_y_inv(const float2* __restrict__ tw, const double* __restrict__ tab, float2* ax, const float2* __restrict__ phi,
        float2* __restrict__ ay, float2* __restrict__ third) {
    using T = Tile16<N>;
    using Map = typename T::Map;
    extern __shared__ float2 smf[];
    const T t;
    const long long o = (long long)t.plane * N * T::PITCH + t.iz;
    const int d = blockIdx.y;
    const float2* in = (d == 0 ? ax : phi) + o;
    float2* out = (d == 0 ? ax : d == 1 ? ay : third) + o;
    fft::run<N, 1, Map>(tw, smf,
                        [&](int i, int, bool) {
                            const float2 z = in[i * T::PITCH];
                            return d == 1 ? times_ik(__ldg(split_k(tab, N) + i), z) : z;
                        },
                        [&](int i, int, float2 z, bool) { out[i * T::PITCH] = z; });
}

// Half spectra along z of two rows -> the rows: one complex transform of
// a + i b. blockIdx.y = component; the third one takes its i k_z here.
template <int N>
__global__ void __launch_bounds__(Rows16<N>::NT, 1024 / Rows16<N>::NT)
k_z_inv(const float2* __restrict__ tw, const double* __restrict__ tab, const float2* __restrict__ ax,
        const float2* __restrict__ ay, const float2* __restrict__ az, float* __restrict__ acc) {
    using R = Rows16<N>;
    using Map = typename R::Map;
    extern __shared__ float2 smf[];
    const int d = blockIdx.y;
    const long long row0 = (long long)blockIdx.x * 32;
    const float2* src = (d == 0 ? ax : d == 1 ? ay : az) + row0 * R::PITCH;
#pragma unroll 4
    for (int q = threadIdx.x; q < 16 * R::NH; q += R::NT) {
        const int c = q / R::NH, k = q - c * R::NH;
        float2 a = __ldg(src + (2 * c) * R::PITCH + k), b = __ldg(src + (2 * c + 1) * R::PITCH + k);
        if (d == 2) {
            const float2 kz = __ldg(split_k(tab, N) + k);
            a = times_ik(kz, a);
            b = times_ik(kz, b);
        }
        if (k == 0 || k == N / 2) { a.y = 0.f; b.y = 0.f; }      // real modes
        smf[Map::at(k, c)] = make_float2(a.x - b.y, a.y + b.x);
        if (k > 0 && k < N / 2) smf[Map::at(N - k, c)] = make_float2(a.x + b.y, b.x - a.y);
    }
    __syncthreads();
    float* dst = acc + ((long long)d * N * N + row0) * N;
    fft::run<N, 1, Map, true>(tw, smf, [&](int i, int c, bool) { return smf[Map::at(i, c)]; },
                              [&](int i, int c, float2 z, bool) {
                                  dst[2 * c * N + i] = z.x;
                                  dst[(2 * c + 1) * N + i] = z.y;
                              });
}

template <int N>
cudaError_t solve_of(sss_pm3* p, double cscale, bool setup, cudaStream_t st) {
    using T = Tile16<N>;
    using R = Rows16<N>;
    if (setup) {
        const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
        cudaError_t e = cudaFuncSetAttribute((const void*)k_z_fwd<N>, attr, (int)R::SMEM);
        e = e ? e : cudaFuncSetAttribute((const void*)k_y_fwd<N>, attr, (int)T::SMEM);
        e = e ? e : cudaFuncSetAttribute((const void*)k_x_solve<N>, attr, (int)(2 * T::SMEM));
        e = e ? e : cudaFuncSetAttribute((const void*)k_y_inv<N>, attr, (int)T::SMEM);
        e = e ? e : cudaFuncSetAttribute((const void*)k_z_inv<N>, attr, (int)R::SMEM);
        return e ? e : fft_table(N, &p->tw);
    }
    const size_t m = (size_t)N * N * T::PITCH;
    k_z_fwd<N><<<R::TILES, R::NT, R::SMEM, st>>>(p->tw, p->rho, p->rk);
    k_y_fwd<N><<<T::TILES, T::NT, T::SMEM, st>>>(p->tw, p->rk);
    k_x_solve<N><<<T::TILES, T::NT, 2 * T::SMEM, st>>>(p->tw, p->rk, cscale, p->tab, p->ak, p->ak + m);
    k_y_inv<N><<<dim3(T::TILES, 3), T::NT, T::SMEM, st>>>(p->tw, p->tab, p->ak, p->ak + m, p->rk, p->ak + 2 * m);
    k_z_inv<N><<<dim3(R::TILES, 3), R::NT, R::SMEM, st>>>(p->tw, p->tab, p->ak, p->rk, p->ak + 2 * m, p->acc);
    return cudaGetLastError();
}

// Mesh sides with own transforms: 2^a and 3 2^a from 32 (one stage less than
// two below) to 512 (512 threads and 128 KB for 16 columns twice above).
bool own_solve(sss_pm3* p, double cscale, bool setup, cudaStream_t st, cudaError_t* e) {
    switch (p->n) {
#define CASE(q) case q: *e = solve_of<q>(p, cscale, setup, st); return true
        CASE(32); CASE(48); CASE(64); CASE(96); CASE(128); CASE(192); CASE(256); CASE(384); CASE(512);
#undef CASE
        default: return false;
    }
}

__global__ void __launch_bounds__(256) k_gather3(const Pm3Parts s, int n, double inv_h,
                                                 const float* __restrict__ acc, const Pm3Epi e) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.n) return;
    int i[3];
    double t[3];
    for (int c = 0; c < 3; ++c) pm3_cell(s.x[c][p], inv_h, n, i[c], t[c]);
    const int j[3] = {i[0] + 1 == n ? 0 : i[0] + 1, i[1] + 1 == n ? 0 : i[1] + 1, i[2] + 1 == n ? 0 : i[2] + 1};
    const long long n3 = (long long)n * n * n;
    double a[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int dx = c >> 2, dy = (c >> 1) & 1, dz = c & 1;
        const double w = (dx ? t[0] : 1.0 - t[0]) * (dy ? t[1] : 1.0 - t[1]) * (dz ? t[2] : 1.0 - t[2]);
        const long long q = ((long long)(dx ? j[0] : i[0]) * n + (dy ? j[1] : i[1])) * n + (dz ? j[2] : i[2]);
        a[0] += w * (double)__ldg(acc + q);
        a[1] += w * (double)__ldg(acc + n3 + q);
        a[2] += w * (double)__ldg(acc + 2 * n3 + q);
    }
    pm3_epilogue(s, e, p, a[0], a[1], a[2]);
}

__global__ void __launch_bounds__(256) k_kick_drift3(const Pm3Parts s, double hdt, double dt, double box) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= s.n) return;
    for (int c = 0; c < 3; ++c) {
        const double v = s.v[c][p] + s.a[c][p] * hdt;
        s.v[c][p] = v;
        s.x[c][p] = pm3_wrap(s.x[c][p] + v * dt, box);
    }
}

void pm3_free(sss_pm3* p) {
    if (p->fwd) cufftDestroy(p->fwd);
    if (p->inv3) cufftDestroy(p->inv3);
    cudaFree(p->rho);
    cudaFree(p->lrho);
    cudaFree(p->rk);
    cudaFree(p->ak);
    cudaFree(p->acc);
    cudaFree(p->tab);
    cudaFree(p->tw);
    free(p);
}

int check_parts(sss_ctx* ctx, const sss_pm3_particles* s) {
    if (!s) return sss_set_err(ctx, SSS_ERR_ARG, "NULL particle state");
    if (s->n < 0) return sss_set_err(ctx, SSS_ERR_ARG, "negative particle count");
    if (s->n == 0) return SSS_OK;
    for (int c = 0; c < 3; ++c)
        if (!s->x[c] || !s->v[c] || !s->a[c]) return sss_set_err(ctx, SSS_ERR_ARG, "NULL particle array");
    return SSS_OK;
}

}  // namespace

extern "C" int sss_pm3_create(sss_ctx* ctx, int mesh_n, double box, sss_pm3** out) {
    if (!ctx || !out) return SSS_ERR_ARG;
    *out = nullptr;
    if (mesh_n < 8 || mesh_n > 1024 || (mesh_n & 1))
        return sss_set_err(ctx, SSS_ERR_ARG, "mesh_n must be even and in [8, 1024]");
    if (!(box > 0.0)) return sss_set_err(ctx, SSS_ERR_ARG, "box must be > 0");
    SSS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    sss_pm3* p = (sss_pm3*)calloc(1, sizeof(sss_pm3));
    p->ctx = ctx;
    p->n = mesh_n;
    p->box = box;
    const size_t n3 = (size_t)mesh_n * mesh_n * mesh_n;
    const size_t m = (size_t)mesh_n * mesh_n * (mesh_n / 2 + 1), mp = (size_t)mesh_n * mesh_n * pitch_of(mesh_n);
    cudaError_t e = cudaSuccess;
    e = e ? e : cudaMalloc(&p->rho, n3 * sizeof(float));
    e = e ? e : cudaMalloc(&p->lrho, n3 * sizeof(float));
    e = e ? e : cudaMalloc(&p->rk, mp * sizeof(float2));
    e = e ? e : cudaMalloc(&p->ak, 3 * mp * sizeof(float2));
    e = e ? e : cudaMalloc(&p->acc, 3 * n3 * sizeof(float));
    e = e ? e : cudaMalloc(&p->tab, 4 * (size_t)mesh_n * sizeof(double));
    p->tab_deconv = -1;
    if (e != cudaSuccess) {
        pm3_free(p);
        return sss_cuda_err(ctx, e, "cudaMalloc (pm3)");
    }
    p->own = own_solve(p, 0.0, true, nullptr, &e);
    if (e != cudaSuccess) {
        pm3_free(p);
        return sss_cuda_err(ctx, e, "transforms (pm3)");
    }
    if (p->own) {
        *out = p;
        return SSS_OK;
    }
    cufftResult r = cufftPlan3d(&p->fwd, mesh_n, mesh_n, mesh_n, CUFFT_R2C);
    if (r == CUFFT_SUCCESS) {
        int dims[3] = {mesh_n, mesh_n, mesh_n};
        r = cufftPlanMany(&p->inv3, 3, dims, nullptr, 1, (int)m, nullptr, 1, (int)n3, CUFFT_C2R, 3);
    }
    if (r != CUFFT_SUCCESS) {
        pm3_free(p);
        return cufft_err(ctx, r, "cufftPlan (pm3)");
    }
    *out = p;
    return SSS_OK;
}

extern "C" void sss_pm3_destroy(sss_pm3* p) {
    if (!p) return;
    cudaSetDevice(p->ctx->device);
    cudaDeviceSynchronize();
    pm3_free(p);
}

extern "C" int sss_pm3_meshes(sss_pm3* p, float** rho, float** accel) {
    if (!p) return SSS_ERR_ARG;
    if (rho) *rho = p->rho;
    if (accel) *accel = p->acc;
    return SSS_OK;
}

extern "C" int sss_pm3_density(sss_pm3* p, const sss_pm3_particles* s, void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    int rc = check_parts(ctx, s);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const long long n3 = (long long)p->n * p->n * p->n;
    SSS_CUDA_TRY(ctx, cudaMemsetAsync(p->rho, 0, (size_t)n3 * sizeof(float), st));
    if (s->n == 0) return SSS_OK;
    const double inv_h = p->n / p->box;
    const double h = p->box / p->n;
    const int blocks = (int)std::min<long long>((s->n + 255) / 256, (long long)ctx->num_sms * 8);
    k_deposit3<<<blocks, 256, 0, st>>>(pm3_parts(s), p->n, inv_h, 1.0 / (h * h * h), p->rho);
    SSS_LAUNCH_CHECK(ctx, "k_deposit3");
    return SSS_OK;
}

extern "C" int sss_pm3_solve(sss_pm3* p, double G, int deconv, double r_split, void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    if (deconv < 0 || deconv > 4) return sss_set_err(ctx, SSS_ERR_ARG, "deconv must be in [0, 4]");
    if (!(r_split >= 0.0)) return sss_set_err(ctx, SSS_ERR_ARG, "r_split must be >= 0");
    cudaStream_t st = (cudaStream_t)stream;
    const double rs2 = r_split * r_split;
    if (p->tab_deconv != deconv || p->tab_rs2 != rs2) {
        k_spectrum_tables<<<blocks_for(p->n, 128), 128, 0, st>>>(p->n, p->box, deconv, rs2, p->tab);
        SSS_LAUNCH_CHECK(ctx, "k_spectrum_tables");
        p->tab_deconv = deconv;
        p->tab_rs2 = rs2;
    }
    const int nh = p->n / 2 + 1;
    const double cscale = 4.0 * 3.14159265358979323846 * G / ((double)p->n * p->n * p->n);
    if (p->own) {
        cudaError_t e = cudaSuccess;
        own_solve(p, cscale, false, st, &e);
        if (e != cudaSuccess) return sss_cuda_err(ctx, e, "own transforms (pm3)");
        return SSS_OK;
    }
    cufftSetStream(p->fwd, st);
    cufftSetStream(p->inv3, st);
    cufftResult r = cufftExecR2C(p->fwd, p->rho, (cufftComplex*)p->rk);
    if (r != CUFFT_SUCCESS) return cufft_err(ctx, r, "cufftExecR2C");
    k_spectrum3<<<dim3((nh + 127) / 128, p->n, p->n), 128, 0, st>>>(p->rk, p->n, cscale, p->tab, p->ak);
    SSS_LAUNCH_CHECK(ctx, "k_spectrum3");
    r = cufftExecC2R(p->inv3, (cufftComplex*)p->ak, p->acc);
    if (r != CUFFT_SUCCESS) return cufft_err(ctx, r, "cufftExecC2R");
    return SSS_OK;
}

extern "C" int sss_pm3_gather(sss_pm3* p, const sss_pm3_particles* s, int mode, double hdt, double dt,
                              float* snap, void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    int rc = check_parts(ctx, s);
    if (rc) return rc;
    if (mode < SSS_PM3_FORCE || mode > SSS_PM3_KICK_DRIFT) return sss_set_err(ctx, SSS_ERR_ARG, "bad mode");
    if (s->n == 0) return SSS_OK;
    Pm3Epi e{mode, hdt, dt, p->box, snap};
    k_gather3<<<blocks_for(s->n, 256), 256, 0, (cudaStream_t)stream>>>(pm3_parts(s), p->n, p->n / p->box, p->acc,
                                                                      e);
    SSS_LAUNCH_CHECK(ctx, "k_gather3");
    return SSS_OK;
}

extern "C" int sss_pm3_kick_drift(sss_pm3* p, const sss_pm3_particles* s, double hdt, double dt, void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    int rc = check_parts(ctx, s);
    if (rc) return rc;
    if (s->n == 0) return SSS_OK;
    k_kick_drift3<<<blocks_for(s->n, 256), 256, 0, (cudaStream_t)stream>>>(pm3_parts(s), hdt, dt, p->box);
    SSS_LAUNCH_CHECK(ctx, "k_kick_drift3");
    return SSS_OK;
}
