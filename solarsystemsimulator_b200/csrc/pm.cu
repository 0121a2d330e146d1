// Particle-mesh forces for sm_100a: replaces the 2-D isolated PM of the
// reference (backend/pm_kernel.py:34-293). Deposit, kernel build, the
// convolution, gather and the KDK integration are kernels of this file.
//
// 2-D isolated (Hockney-James): masses are deposited by cloud-in-cell, the
// zero-padded 2N x 2N density is transformed, multiplied by the transforms of
// the softened force kernels K_x, K_y (with the inverse transform's 1/(2N)^2
// folded in), transformed back and read bilinearly with the deposit's
// stencil. f64 throughout, as the reference.
//
// The convolution (2N = 2^a, 3 2^a, 1000, 2000 or 4000 up to 8192) is three kernels
// over the block transforms of fft.cuh:
//   k_rows_fwd : two real rows a, b as one complex transform a + i b; only
//                the N rows and the N columns that hold mass are read
//   k_cols     : one column: forward, times each kernel spectrum, inverse,
//                only the N rows of the crop written
//   k_rows_inv : the two force components of a row as one complex transform
//                f_x + i f_y, stored as pairs that the gather reads whole
// K(d; h, eps) = G / h^2 K(d / h; 1, eps / h), and offsets of +-N never meet
// two grid points, so the spectra are those of the unit kernel with those
// offsets zeroed: purely imaginary, odd along the force's axis and even along
// the other, one (N + 1)^2 table of reals (kept with its transpose) that a
// plan remakes only when eps / h changes, not with every new h.
// Other sizes go through cuFFT with the kernels of the current h.

#include "fft.cuh"

#include <cufft.h>

namespace {

// ------------------------------------------------------------ 2-D kernels

// K(d) = -G d / (|d|^2 + eps2)^(3/2) on the padded grid, offsets wrapped so
// that index m maps to m (m < N) or m - 2N (pm_kernel.py:42-59).
__global__ void k_force_kernels_2d(int n, double h, double eps2, double G, double* __restrict__ kx,
                                   double* __restrict__ ky) {
    const int np = 2 * n;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)np * np) return;
    const int i = (int)(t / np), j = (int)(t % np);
    const double oi = (double)(i < n ? i : i - np), oj = (double)(j < n ? j : j - np);
    const double dx = __dmul_rn(oi, h), dy = __dmul_rn(oj, h);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), eps2);
    const double inv_r3 = __ddiv_rn(1.0, __dmul_rn(r2, sqrt(r2)));
    kx[t] = __dmul_rn(__dmul_rn(-G, dx), inv_r3);
    ky[t] = __dmul_rn(__dmul_rn(-G, dy), inv_r3);
}

// Grid geometry of a step in device memory (pm_kernel.py:110-124), with the
// cell size the force kernels stand for (remade when h moves by more than
// 1e-6 of it, :216-221) and the factor of the unit kernel's spectrum.
struct Geo {
    double x0, y0, h, kernel_h, scale;
};

// CIC corner index/weights of the reference (pm_kernel.py:63-90): cell
// clipped to [0, N-2], fractional offsets from the clipped cell.
__device__ __forceinline__ void cic2(double gx, double gy, double x0, double y0, double h, int n, int& i,
                                     int& j, double& tx, double& ty) {
    const double fx = __ddiv_rn(__dsub_rn(gx, x0), h);
    const double fy = __ddiv_rn(__dsub_rn(gy, y0), h);
    i = (int)floor(fx);
    j = (int)floor(fy);
    i = min(max(i, 0), n - 2);
    j = min(max(j, 0), n - 2);
    tx = __dsub_rn(fx, (double)i);
    ty = __dsub_rn(fy, (double)j);
}

// deposit into the grid of row stride s (2N where the padded array is transformed whole)
__global__ void k_cic_deposit_2d(const double* __restrict__ gx, const double* __restrict__ gy,
                                 const double* __restrict__ gm, long long np_, int n, long long s, double x0,
                                 double y0, double h, double* __restrict__ rho_pad,
                                 const Geo* __restrict__ g) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np_) return;
    if (g) { x0 = g->x0; y0 = g->y0; h = g->h; }
    int i, j;
    double tx, ty;
    cic2(gx[p], gy[p], x0, y0, h, n, i, j, tx, ty);
    const double m = gm[p];
    const double ux = __dsub_rn(1.0, tx), uy = __dsub_rn(1.0, ty);
    atomicAdd(&rho_pad[(long long)i * s + j], __dmul_rn(__dmul_rn(m, ux), uy));
    atomicAdd(&rho_pad[(long long)(i + 1) * s + j], __dmul_rn(__dmul_rn(m, tx), uy));
    atomicAdd(&rho_pad[(long long)i * s + (j + 1)], __dmul_rn(__dmul_rn(m, ux), ty));
    atomicAdd(&rho_pad[(long long)(i + 1) * s + (j + 1)], __dmul_rn(__dmul_rn(m, tx), ty));
}

// F_x = rho_k * FK_x * scale, F_y = rho_k * FK_y * scale (complex, numpy order)
__global__ void k_spectrum_mul_2d(const double2* __restrict__ fr, const double2* __restrict__ fkx,
                                  const double2* __restrict__ fky, long long m, double scale,
                                  double2* __restrict__ outx, double2* __restrict__ outy) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m) return;
    const double2 a = fr[t], bx = fkx[t], by = fky[t];
    double2 cx, cy;
    cx.x = __dmul_rn(__dsub_rn(__dmul_rn(a.x, bx.x), __dmul_rn(a.y, bx.y)), scale);
    cx.y = __dmul_rn(__dadd_rn(__dmul_rn(a.x, bx.y), __dmul_rn(a.y, bx.x)), scale);
    cy.x = __dmul_rn(__dsub_rn(__dmul_rn(a.x, by.x), __dmul_rn(a.y, by.y)), scale);
    cy.y = __dmul_rn(__dadd_rn(__dmul_rn(a.x, by.y), __dmul_rn(a.y, by.x)), scale);
    outx[t] = cx;
    outy[t] = cy;
}

// bilinear read of the [0:N, 0:N] crop of the 2N x 2N fields (pm_kernel.py:93-107)
__global__ void k_cic_gather_2d(const double* __restrict__ px, const double* __restrict__ py, long long np_,
                                int n, double x0, double y0, double h, const double* __restrict__ fx_pad,
                                const double* __restrict__ fy_pad, double* __restrict__ ax,
                                double* __restrict__ ay) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np_) return;
    int i, j;
    double tx, ty;
    cic2(px[p], py[p], x0, y0, h, n, i, j, tx, ty);
    const double ux = __dsub_rn(1.0, tx), uy = __dsub_rn(1.0, ty);
    const long long s = 2LL * n;
    const long long c00 = (long long)i * s + j, c10 = c00 + s, c01 = c00 + 1, c11 = c10 + 1;
    // f[..] * (1 - tx) * (1 - ty) + ... evaluated left to right, as the reference
    const double* F[2] = {fx_pad, fy_pad};
    double out[2];
    for (int q = 0; q < 2; ++q) {
        const double* f = F[q];
        const double t00 = __dmul_rn(__dmul_rn(f[c00], ux), uy);
        const double t10 = __dmul_rn(__dmul_rn(f[c10], tx), uy);
        const double t01 = __dmul_rn(__dmul_rn(f[c01], ux), ty);
        const double t11 = __dmul_rn(__dmul_rn(f[c11], tx), ty);
        out[q] = __dadd_rn(__dadd_rn(__dadd_rn(t00, t10), t01), t11);
    }
    ax[p] = out[0];
    ay[p] = out[1];
}

// the same read of the N x N field of pairs (f_x, f_y)
__device__ __forceinline__ double2 gather_pair(double px, double py, int n, double x0, double y0, double h,
                                               const double2* __restrict__ f) {
    int i, j;
    double tx, ty;
    cic2(px, py, x0, y0, h, n, i, j, tx, ty);
    const double ux = __dsub_rn(1.0, tx), uy = __dsub_rn(1.0, ty);
    const long long c00 = (long long)i * n + j;
    const double2 f00 = f[c00], f10 = f[c00 + n], f01 = f[c00 + 1], f11 = f[c00 + n + 1];
    double2 a;
    a.x = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(f00.x, ux), uy), __dmul_rn(__dmul_rn(f10.x, tx), uy)),
                              __dmul_rn(__dmul_rn(f01.x, ux), ty)), __dmul_rn(__dmul_rn(f11.x, tx), ty));
    a.y = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(f00.y, ux), uy), __dmul_rn(__dmul_rn(f10.y, tx), uy)),
                              __dmul_rn(__dmul_rn(f01.y, ux), ty)), __dmul_rn(__dmul_rn(f11.y, tx), ty));
    return a;
}

__global__ void k_cic_gather_pairs_2d(const double* __restrict__ px, const double* __restrict__ py, long long np_,
                                      int n, double x0, double y0, double h, const double2* __restrict__ f,
                                      double* __restrict__ ax, double* __restrict__ ay) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np_) return;
    const double2 a = gather_pair(px[p], py[p], n, x0, y0, h, f);
    ax[p] = a.x;
    ay[p] = a.y;
}

__global__ void k_split_pairs_2d(const double2* __restrict__ f, long long m, double* __restrict__ ax,
                                 double* __restrict__ ay) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m) return;
    ax[t] = f[t].x;
    ay[t] = f[t].y;
}

// ---------------------------------------------------- convolution, own FFTs

// K_x of unit cell size and G = 1, zero at the offsets +-N
__global__ void k_unit_kernel_2d(int n, double e2, double* __restrict__ kx) {
    const int np = 2 * n;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)np * np) return;
    const int i = (int)(t / np), j = (int)(t % np);
    if (i == n || j == n) { kx[t] = 0.0; return; }
    const double dx = (double)(i < n ? i : i - np), dy = (double)(j < n ? j : j - np);
    const double r2 = dx * dx + dy * dy + e2;
    kx[t] = -dx / (r2 * sqrt(r2));
}

// U[a][b] = Im of the spectrum at (a, b), a, b <= N, and its transpose V
__global__ void __launch_bounds__(256) k_kernel_tables_2d(const double2* __restrict__ fk, int n,
                                                          double* __restrict__ u, double* __restrict__ v) {
    __shared__ double tile[32][33];
    const int m = n + 1, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        const int a = blockIdx.y * 32 + r, b = blockIdx.x * 32 + tx;
        double q = 0.0;
        if (a < m && b < m) {
            q = (a == 0 || a == n) ? 0.0 : fk[(long long)a * m + b].y;      // odd in a
            u[(long long)a * m + b] = q;
        }
        tile[r][tx] = q;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int b = blockIdx.x * 32 + r, a = blockIdx.y * 32 + tx;
        if (a < m && b < m) v[(long long)b * m + a] = tile[tx][r];
    }
}

// One 32-byte access per lane for scattered pairs of complex values (half the
// L1 passes of two 16-byte ones).
__device__ __forceinline__ void st_pair(double2* p, double2 a, double2 b) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" :: "l"(p), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y) : "memory");
}
__device__ __forceinline__ void ld_pair(const double2* p, double2& a, double2& b) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(p));
}

// Rows 2p and 2p + 1 of the density -> their spectra, out[k][row], k <= N
// (two neighbouring rows: 32-byte sectors of the transposed output).
template <int L>
__global__ void __launch_bounds__(fft_threads(L, 1), 512 / fft_threads(L, 1))
k_rows_fwd(const double2* __restrict__ tw, const double* __restrict__ rho, double2* __restrict__ out) {
    constexpr int n = L / 2;
    static_assert(n % 2 == 0, "pairs of rows");
    extern __shared__ double2 sm2[];
    using Map = fft::One;
    for (int p = blockIdx.x; p < n / 2; p += gridDim.x) {
        const double* ra = rho + (long long)(2 * p) * n;
        __syncthreads();
        fft::run<L, -1, Map>(tw, sm2,
                     [&](int i, int, bool hi) {
                         double2 z = make_double2(0.0, 0.0);
                         if (!hi) z = make_double2(__ldg(ra + i), __ldg(ra + n + i));
                         return z;
                     },
                     [&](int i, int, double2 z, bool) { sm2[Map::at(i, 0)] = z; });
        __syncthreads();
        for (int k = threadIdx.x; k <= n; k += blockDim.x) {
            const double2 z = sm2[Map::at(k, 0)], w = sm2[Map::at(k == 0 ? 0 : L - k, 0)];
            st_pair(out + (long long)k * n + 2 * p, make_double2(0.5 * (z.x + w.x), 0.5 * (z.y - w.y)),
                    make_double2(0.5 * (z.y + w.y), 0.5 * (w.x - z.x)));
        }
    }
}

// Column kj of the density's row spectra -> the N crop rows of the two force
// spectra' columns, out[kj][row] = (F_x, F_y). The column's spectrum waits in
// `slot` (this CTA's L columns of scratch, L2 resident) for the second kernel.
template <int L>
__global__ void __launch_bounds__(fft_threads(L, 1), 512 / fft_threads(L, 1))
k_cols(const double2* __restrict__ tw, const double2* __restrict__ in, const double* __restrict__ u,
       const double* __restrict__ v, double scale, const Geo* __restrict__ geo, double2* slots,
       double2* __restrict__ out) {
    constexpr int n = L / 2;
    if (geo) scale = geo->scale;
    extern __shared__ double2 sm2[];
    using Map = fft::One;
    double2* slot = slots + (long long)blockIdx.x * L;
    for (int kj = blockIdx.x; kj <= n; kj += gridDim.x) {
        const double2* col = in + (long long)kj * n;
        double2* o = out + (long long)kj * n * 2;
        __syncthreads();
        fft::run<L, -1, Map>(tw, sm2,
                     [&](int i, int, bool hi) { return hi ? make_double2(0.0, 0.0) : __ldg(col + i); },
                     [&](int i, int, double2 z, bool) { slot[i] = z; });
        __syncthreads();
        // F_x: odd in the column index, F_y = its mirror image: even
#pragma unroll 1
        for (int d = 0; d < 2; ++d) {
            const double* q = (d ? u : v) + (long long)kj * (n + 1);
            const double up = d ? scale : -scale;
            fft::run<L, 1, Map>(tw, sm2,
                                [&](int i, int, bool hi) {
                                    const double2 a = slot[i];
                                    const double g = hi ? up * __ldg(q + (L - i)) : scale * __ldg(q + i);
                                    return make_double2(-a.y * g, a.x * g);
                                },
                                [&](int i, int, double2 z, bool hi) { if (!hi) o[2 * i + d] = z; });
            __syncthreads();
        }
    }
}

// Row i: f_x + i f_y from the half spectra of its two real components.
template <int L>
__global__ void __launch_bounds__(fft_threads(L, 1), 512 / fft_threads(L, 1))
k_rows_inv(const double2* __restrict__ tw, const double2* __restrict__ in, double2* __restrict__ field) {
    constexpr int n = L / 2;
    extern __shared__ double2 sm2[];
    using Map = fft::One;
    for (int row = blockIdx.x; row < n; row += gridDim.x) {
        __syncthreads();
#pragma unroll 4
        for (int k = threadIdx.x; k <= n; k += fft_threads(L, 1)) {
            double2 a, b;
            ld_pair(in + ((long long)k * n + row) * 2, a, b);
            if (k == 0 || k == n) { a.y = 0.0; b.y = 0.0; }     // real rows
            sm2[Map::at(k, 0)] = make_double2(a.x - b.y, a.y + b.x);
            if (k > 0 && k < n) sm2[Map::at(L - k, 0)] = make_double2(a.x + b.y, b.x - a.y);
        }
        __syncthreads();
        fft::run<L, 1, Map, true>(tw, sm2, [&](int i, int, bool) { return sm2[Map::at(i, 0)]; },
                                  [&](int i, int, double2 z, bool hi) { if (!hi) field[(long long)row * n + i] = z; });
    }
}

struct Convolve2d {
    void (*rows_fwd)(const double2*, const double*, double2*);
    void (*cols)(const double2*, const double2*, const double*, const double*, double, const Geo*, double2*,
                 double2*);
    void (*rows_inv)(const double2*, const double2*, double2*);
    int threads;
};

template <int L>
Convolve2d convolve_of() {
    return {k_rows_fwd<L>, k_cols<L>, k_rows_inv<L>, fft_threads(L, 1)};
}

// Padded lengths 2N with kernels: 2^a and 3 2^a from 64 to 8192, and 1000, 2000
// and 4000, the decimal grids of 500, 1,000 and 2,000 points. Every length is
// three kernels of its own, so only sizes that simulations ask for have them;
// any other grid (640, 1,200, ...) convolves through cuFFT as well. 8192 is the
// longest: 139 KB of shared memory and 512 threads of 128 registers. 8000 (a grid
// of 4,000) is none: its radix-5 stages, three butterflies a thread, need 544
// threads. A step on a 2048 grid: 343 us; through cuFFT, kernels remade for its
// h, 1,083.
bool convolve_for(int L, Convolve2d* c) {
    switch (L) {
#define CASE(n) case n: *c = convolve_of<n>(); return true
        CASE(64); CASE(96); CASE(128); CASE(192); CASE(256); CASE(384); CASE(512); CASE(768); CASE(1000);
        CASE(1024); CASE(1536); CASE(2000); CASE(2048); CASE(3072); CASE(4000); CASE(4096); CASE(6144); CASE(8192);
#undef CASE
        default: return false;
    }
}

// bilinear read of one caller-held N x N field with row stride ld (_cic_gather, pm_kernel.py:93-107)
__global__ void k_cic_gather_field_2d(const double* __restrict__ px, const double* __restrict__ py, long long np_,
                                      int n, long long ld, double x0, double y0, double h,
                                      const double* __restrict__ f, double* __restrict__ out) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np_) return;
    int i, j;
    double tx, ty;
    cic2(px[p], py[p], x0, y0, h, n, i, j, tx, ty);
    const double ux = __dsub_rn(1.0, tx), uy = __dsub_rn(1.0, ty);
    const long long c00 = (long long)i * ld + j, c10 = c00 + ld, c01 = c00 + 1, c11 = c10 + 1;
    const double t00 = __dmul_rn(__dmul_rn(f[c00], ux), uy);
    const double t10 = __dmul_rn(__dmul_rn(f[c10], tx), uy);
    const double t01 = __dmul_rn(__dmul_rn(f[c01], ux), ty);
    const double t11 = __dmul_rn(__dmul_rn(f[c11], tx), ty);
    out[p] = __dadd_rn(__dadd_rn(__dadd_rn(t00, t10), t01), t11);
}

// A block's min and max of x and y into its four values of part (warps of
// 32 threads, at most 8).
__device__ __forceinline__ void block_bbox(double a, double b, double c, double d, double* __restrict__ part) {
    __shared__ double s[4][8];
    for (int o = 16; o > 0; o >>= 1) {
        a = fmin(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
        c = fmin(c, __shfl_xor_sync(0xffffffffu, c, o));
        d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) { s[0][w] = a; s[1][w] = b; s[2][w] = c; s[3][w] = d; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
            a = fmin(a, s[0][k]); b = fmax(b, s[1][k]); c = fmin(c, s[2][k]); d = fmax(d, s[3][k]);
        }
        part[4 * blockIdx.x + 0] = a;
        part[4 * blockIdx.x + 1] = b;
        part[4 * blockIdx.x + 2] = c;
        part[4 * blockIdx.x + 3] = d;
    }
}

// min/max of x and y: out[0..3] = xmin, xmax, ymin, ymax (two-pass: blocks -> final)
__global__ void k_bbox_2d(const double* __restrict__ x, const double* __restrict__ y, long long n,
                          double* __restrict__ part) {
    double a = 1e308, b = -1e308, c = 1e308, d = -1e308;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        a = fmin(a, x[i]); b = fmax(b, x[i]);
        c = fmin(c, y[i]); d = fmax(d, y[i]);
    }
    block_bbox(a, b, c, d, part);
}

__global__ void k_bbox_final(const double* __restrict__ part, int nb, double* __restrict__ out) {
    double a = 1e308, b = -1e308, c = 1e308, d = -1e308;
    for (int k = threadIdx.x; k < nb; k += 32) {
        a = fmin(a, part[4 * k]); b = fmax(b, part[4 * k + 1]);
        c = fmin(c, part[4 * k + 2]); d = fmax(d, part[4 * k + 3]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        a = fmin(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
        c = fmin(c, __shfl_xor_sync(0xffffffffu, c, o));
        d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
    }
    if (threadIdx.x != 0) return;
    out[0] = a; out[1] = b; out[2] = c; out[3] = d;
}

// KDK pieces (pm_kernel.py:264-273): v += hdt*a; x += dt*v  /  v += hdt*a
__global__ void k_kick_drift_2d(double* __restrict__ x, double* __restrict__ y, double* __restrict__ vx,
                                double* __restrict__ vy, const double* __restrict__ ax,
                                const double* __restrict__ ay, long long n, double hdt, double dt, int drift) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double nvx = __dadd_rn(vx[i], __dmul_rn(hdt, ax[i]));
    const double nvy = __dadd_rn(vy[i], __dmul_rn(hdt, ay[i]));
    vx[i] = nvx;
    vy[i] = nvy;
    if (drift) {
        x[i] = __dadd_rn(x[i], __dmul_rn(dt, nvx));
        y[i] = __dadd_rn(y[i], __dmul_rn(dt, nvy));
    }
}

__global__ void k_snap_2d(const double* __restrict__ a, long long n, float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)a[i];
}

// The step's geometry from the blocks' boxes (grid_fuer, pm_kernel.py:110-124;
// its operations and their rounding): one block, the step stays on the device.
__global__ void __launch_bounds__(256) k_geo_2d(const double* __restrict__ part, int nb, double cells, double margin,
                                                double G, double np2, Geo* __restrict__ geo) {
    __shared__ double box[4];
    double a = 1e308, b = -1e308, c = 1e308, d = -1e308;
    for (int k = threadIdx.x; k < nb; k += blockDim.x) {
        a = fmin(a, part[4 * k]); b = fmax(b, part[4 * k + 1]);
        c = fmin(c, part[4 * k + 2]); d = fmax(d, part[4 * k + 3]);
    }
    block_bbox(a, b, c, d, box);
    if (threadIdx.x != 0) return;
    const double span = fmax(fmax(__dsub_rn(box[1], box[0]), __dsub_rn(box[3], box[2])), 1e-30);
    const double h = __ddiv_rn(span, cells);
    geo->x0 = __dsub_rn(box[0], __dmul_rn(margin, h));
    geo->y0 = __dsub_rn(box[2], __dmul_rn(margin, h));
    geo->h = h;
    double kh = geo->kernel_h;
    if (!(kh > 0.0) || fabs(__dsub_rn(h, kh)) > __dmul_rn(1e-6, h)) kh = h;
    geo->kernel_h = kh;
    geo->scale = G / (kh * kh) / np2;
}

// Masses (first n) and tracers of a step.
struct Bodies2d {
    double *x[2], *y[2], *vx[2], *vy[2], *ax[2], *ay[2];    // masses, tracers
    long long n, t;
};

// One pass over the bodies between two fields: with f the acceleration from
// the field, the closing half kick and the snapshot row; with open the next
// step's opening half kick and drift and the box of the moved masses. (As
// separate launches around a host that read the box back, these took 100 us
// of a step, against 290 of the transforms on a 2048 grid.)
__global__ void __launch_bounds__(256) k_move_2d(const Bodies2d b, int grid_n, const Geo* __restrict__ geo,
                                                 const double2* __restrict__ f, int open, double hdt, double dt,
                                                 float* __restrict__ row, double* __restrict__ part) {
    double lo[2] = {1e308, 1e308}, hi[2] = {-1e308, -1e308};
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < b.n + b.t;
         q += (long long)gridDim.x * blockDim.x) {
        const int k = q < b.n ? 0 : 1;
        const long long i = k ? q - b.n : q;
        double x = b.x[k][i], y = b.y[k][i], vx = b.vx[k][i], vy = b.vy[k][i];
        double2 a;
        if (f) {
            a = gather_pair(x, y, grid_n, geo->x0, geo->y0, geo->h, f);
            b.ax[k][i] = a.x;
            b.ay[k][i] = a.y;
            vx = __dadd_rn(vx, __dmul_rn(hdt, a.x));
            vy = __dadd_rn(vy, __dmul_rn(hdt, a.y));
            float* r = row + (k ? 4 * b.n : 0);
            const long long m = k ? b.t : b.n;
            r[i] = (float)x;
            r[m + i] = (float)y;
            if (!k) {
                r[2 * m + i] = (float)vx;
                r[3 * m + i] = (float)vy;
            }
        } else {
            a = make_double2(b.ax[k][i], b.ay[k][i]);
        }
        if (open) {
            vx = __dadd_rn(vx, __dmul_rn(hdt, a.x));
            vy = __dadd_rn(vy, __dmul_rn(hdt, a.y));
            x = __dadd_rn(x, __dmul_rn(dt, vx));
            y = __dadd_rn(y, __dmul_rn(dt, vy));
            b.x[k][i] = x;
            b.y[k][i] = y;
            if (!k) {
                lo[0] = fmin(lo[0], x); hi[0] = fmax(hi[0], x);
                lo[1] = fmin(lo[1], y); hi[1] = fmax(hi[1], y);
            }
        }
        b.vx[k][i] = vx;
        b.vy[k][i] = vy;
    }
    if (open) block_bbox(lo[0], hi[0], lo[1], hi[1], part);
}

unsigned blocks_for(long long n, int nt) { return (unsigned)((n + nt - 1) / nt); }

int cufft_err(sss_ctx* ctx, cufftResult r, const char* what) {
    return sss_set_err(ctx, SSS_ERR_CUDA, "%s: cuFFT error %d", what, (int)r);
}

}  // namespace

// ------------------------------------------------------------------ C ABI

struct sss_pm2d {
    sss_ctx* ctx;
    int n;                 // grid_n
    bool own;              // the convolution by the kernels of this file
    long long ld;          // row stride of the deposit: N (own) or 2N
    Convolve2d conv;
    int grid[3];           // CTAs of k_rows_fwd, k_cols, k_rows_inv
    double2* tw;           // twiddles of length 2N
    size_t smem;
    double* u;             // (N+1)^2 kernel spectrum and its transpose
    double* v;
    double e2_unit;        // (eps / h)^2 they were made for (-1: none yet)
    double scale;          // G / h^2 / (2N)^2 of the last build
    double2* t1;           // (N+1, N) row spectra of the density
    double2* t2;           // (N+1, N, 2) columns of the force spectra
    double2* slots;        // k_cols: 2N values per CTA
    double2* pairs;        // (N, N) field (f_x, f_y)
    cufftHandle fwd, inv;  // D2Z / Z2D on (2N, 2N); inv only without own
    double* rho;           // deposit
    double* kx;            // real work (2N x 2N): the force kernels
    double* ky;
    double2* fkx;          // (2N, N+1) spectra of the force kernels
    double2* fky;
    double2* fr;           // spectrum of the density
    double2* sx;           // product spectra
    double2* sy;
    double* fieldx;        // (2N x 2N) real fields
    double* fieldy;
    double* bb_part;       // bbox partials
    Geo* geo;              // own: the current step's geometry (sss_pm2d_step_batch)
};

static int pm2d_free(sss_pm2d* p) {
    if (!p) return SSS_OK;
    if (p->fwd) cufftDestroy(p->fwd);
    if (p->inv) cufftDestroy(p->inv);
    if (p->own) {
        cudaFree(p->rho); cudaFree(p->u); cudaFree(p->v); cudaFree(p->t1); cudaFree(p->t2); cudaFree(p->slots);
        cudaFree(p->pairs); cudaFree(p->tw); cudaFree(p->geo);
    }
    cudaFree(p->kx); cudaFree(p->ky); cudaFree(p->fkx); cudaFree(p->fky); cudaFree(p->fr);
    cudaFree(p->sx); cudaFree(p->sy); cudaFree(p->fieldx); cudaFree(p->fieldy);
    cudaFree(p->bb_part);
    free(p);
    return SSS_OK;
}

static cudaError_t pm2d_own_setup(sss_pm2d* p) {
    const int L = 2 * p->n;
    const void* fn[3] = {(const void*)p->conv.rows_fwd, (const void*)p->conv.cols, (const void*)p->conv.rows_inv};
    const int items[3] = {p->n / 2, p->n + 1, p->n};
    const size_t n = (size_t)p->n, m = n + 1;
    p->smem = (size_t)(L + L / 16 + 1) * sizeof(double2);
    cudaError_t e = fft_table(L, &p->tw);
    for (int k = 0; k < 3; ++k) {
        int per_sm = 0;
        e = e ? e : cudaFuncSetAttribute(fn[k], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem);
        e = e ? e : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn[k], p->conv.threads, p->smem);
        const long long cap = (long long)(per_sm > 0 ? per_sm : 1) * p->ctx->num_sms;
        p->grid[k] = (int)(items[k] < cap ? items[k] : cap);
    }
    e = e ? e : cudaMalloc(&p->rho, n * n * sizeof(double));
    e = e ? e : cudaMalloc(&p->u, m * m * sizeof(double));
    e = e ? e : cudaMalloc(&p->v, m * m * sizeof(double));
    e = e ? e : cudaMalloc(&p->t1, m * n * sizeof(double2));
    e = e ? e : cudaMalloc(&p->t2, 2 * m * n * sizeof(double2));
    e = e ? e : cudaMalloc(&p->slots, (size_t)p->grid[1] * L * sizeof(double2));
    e = e ? e : cudaMalloc(&p->pairs, n * n * sizeof(double2));
    e = e ? e : cudaMalloc(&p->kx, 4 * n * n * sizeof(double));
    e = e ? e : cudaMalloc(&p->geo, sizeof(Geo));
    return e;
}

extern "C" int sss_pm2d_create(sss_ctx* ctx, int grid_n, sss_pm2d** out) {
    if (!ctx || !out) return SSS_ERR_ARG;
    *out = nullptr;
    if (grid_n < 4 || grid_n > 16384) return sss_set_err(ctx, SSS_ERR_ARG, "grid_n must be in [4, 16384]");
    SSS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    sss_pm2d* p = (sss_pm2d*)calloc(1, sizeof(sss_pm2d));
    p->ctx = ctx;
    p->n = grid_n;
    p->e2_unit = -1.0;
    p->own = convolve_for(2 * grid_n, &p->conv);
    p->ld = p->own ? grid_n : 2LL * grid_n;
    const long long np = 2LL * grid_n;
    const size_t real_b = (size_t)np * np * sizeof(double);
    const size_t cplx_b = (size_t)np * (grid_n + 1) * sizeof(double2);
    cudaError_t e = cudaSuccess;
    if (p->own) {
        e = pm2d_own_setup(p);
    } else {
        e = e ? e : cudaMalloc(&p->kx, real_b);
        e = e ? e : cudaMalloc(&p->ky, real_b);
        e = e ? e : cudaMalloc(&p->fkx, cplx_b);
        e = e ? e : cudaMalloc(&p->fky, cplx_b);
        e = e ? e : cudaMalloc(&p->fr, cplx_b);
        e = e ? e : cudaMalloc(&p->sx, cplx_b);
        e = e ? e : cudaMalloc(&p->sy, cplx_b);
        e = e ? e : cudaMalloc(&p->fieldx, real_b);
        e = e ? e : cudaMalloc(&p->fieldy, real_b);
        p->rho = p->kx;
    }
    e = e ? e : cudaMalloc(&p->bb_part, 4 * 1024 * sizeof(double));
    if (e != cudaSuccess) {
        pm2d_free(p);
        return sss_cuda_err(ctx, e, "cudaMalloc (pm2d)");
    }
    cufftResult r = cufftPlan2d(&p->fwd, (int)np, (int)np, CUFFT_D2Z);
    if (r == CUFFT_SUCCESS && !p->own) r = cufftPlan2d(&p->inv, (int)np, (int)np, CUFFT_Z2D);
    if (r != CUFFT_SUCCESS) {
        pm2d_free(p);
        return cufft_err(ctx, r, "cufftPlan2d");
    }
    *out = p;
    return SSS_OK;
}

extern "C" void sss_pm2d_destroy(sss_pm2d* p) {
    if (!p) return;
    cudaSetDevice(p->ctx->device);
    cudaDeviceSynchronize();
    pm2d_free(p);
}

// Bounding box of (x, y) into bbox4 (device, xmin xmax ymin ymax).
extern "C" int sss_pm2d_bbox(sss_pm2d* p, const double* x, const double* y, int64_t n, double* bbox4,
                             void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    if (n < 1 || !x || !y || !bbox4) return sss_set_err(ctx, SSS_ERR_ARG, "bbox: empty or NULL input");
    cudaStream_t s = (cudaStream_t)stream;
    int nb = (int)((n + 255) / 256);
    if (nb > 1024) nb = 1024;
    k_bbox_2d<<<nb, 256, 0, s>>>(x, y, n, p->bb_part);
    k_bbox_final<<<1, 32, 0, s>>>(p->bb_part, nb, bbox4);
    SSS_LAUNCH_CHECK(ctx, "k_bbox");
    return SSS_OK;
}

// The unit kernel's spectrum for the softening e2 = (eps / h)^2. eps^2 / h^2
// of a softening tied to h differs from step to step by a few roundings:
// within 1e-15 it is the same kernel.
static int pm2d_unit_spectrum(sss_pm2d* p, double e2, cudaStream_t s) {
    sss_ctx* ctx = p->ctx;
    if (fabs(e2 - p->e2_unit) <= 1e-15 * e2) return SSS_OK;
    const long long np = 2LL * p->n;
    p->e2_unit = -1.0;
    k_unit_kernel_2d<<<blocks_for(np * np, 256), 256, 0, s>>>(p->n, e2, p->kx);
    SSS_LAUNCH_CHECK(ctx, "k_unit_kernel_2d");
    cufftSetStream(p->fwd, s);
    // the spectrum (2N x (N + 1)) fits t2 exactly
    cufftResult r = cufftExecD2Z(p->fwd, p->kx, (cufftDoubleComplex*)p->t2);
    if (r != CUFFT_SUCCESS) return cufft_err(ctx, r, "cufftExecD2Z (kernel)");
    const unsigned tiles = (unsigned)(p->n / 32 + 1);
    k_kernel_tables_2d<<<dim3(tiles, tiles), 256, 0, s>>>(p->t2, p->n, p->u, p->v);
    SSS_LAUNCH_CHECK(ctx, "k_kernel_tables_2d");
    p->e2_unit = e2;
    return SSS_OK;
}

// FFTs of the softened force kernels for cell size h (pm_kernel.py:34-60);
// kept inside the plan object until the next call.
extern "C" int sss_pm2d_build_kernels(sss_pm2d* p, double h, double eps2, double G, void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    if (!(h > 0.0)) return sss_set_err(ctx, SSS_ERR_ARG, "h must be > 0");
    cudaStream_t s = (cudaStream_t)stream;
    const long long np = 2LL * p->n;
    if (p->own) {
        p->scale = G / (h * h) / (double)(np * np);
        return pm2d_unit_spectrum(p, eps2 / (h * h), s);
    }
    k_force_kernels_2d<<<blocks_for(np * np, 256), 256, 0, s>>>(p->n, h, eps2, G, p->kx, p->ky);
    SSS_LAUNCH_CHECK(ctx, "k_force_kernels_2d");
    cufftSetStream(p->fwd, s);
    cufftResult r = cufftExecD2Z(p->fwd, p->kx, (cufftDoubleComplex*)p->fkx);
    if (r == CUFFT_SUCCESS) r = cufftExecD2Z(p->fwd, p->ky, (cufftDoubleComplex*)p->fky);
    if (r != CUFFT_SUCCESS) return cufft_err(ctx, r, "cufftExecD2Z (kernels)");
    return SSS_OK;
}

// Field on the grid from the masses (pm_kernel.py:127-147): deposit into the
// padded grid, D2Z, multiply by the kernel spectra, 2x Z2D. The fields stay
// in the plan object (fieldx/fieldy, 2N x 2N, the [0:N, 0:N] crop valid).
extern "C" int sss_pm2d_field(sss_pm2d* p, const double* gx, const double* gy, const double* gm, int64_t n,
                              double x0, double y0, double h, void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    if (n < 0 || (n > 0 && (!gx || !gy || !gm))) return sss_set_err(ctx, SSS_ERR_ARG, "field: bad input");
    cudaStream_t s = (cudaStream_t)stream;
    const long long np = 2LL * p->n;
    SSS_CUDA_TRY(ctx, cudaMemsetAsync(p->rho, 0, (size_t)p->ld * p->ld * sizeof(double), s));
    if (n > 0) {
        k_cic_deposit_2d<<<blocks_for(n, 256), 256, 0, s>>>(gx, gy, gm, n, p->n, p->ld, x0, y0, h, p->rho,
                                                            nullptr);
        SSS_LAUNCH_CHECK(ctx, "k_cic_deposit_2d");
    }
    if (p->own) {
        p->conv.rows_fwd<<<p->grid[0], p->conv.threads, p->smem, s>>>(p->tw, p->rho, p->t1);
        SSS_LAUNCH_CHECK(ctx, "k_rows_fwd");
        p->conv.cols<<<p->grid[1], p->conv.threads, p->smem, s>>>(p->tw, p->t1, p->u, p->v, p->scale, nullptr, p->slots,
                                                                       p->t2);
        SSS_LAUNCH_CHECK(ctx, "k_cols");
        p->conv.rows_inv<<<p->grid[2], p->conv.threads, p->smem, s>>>(p->tw, p->t2, p->pairs);
        SSS_LAUNCH_CHECK(ctx, "k_rows_inv");
        return SSS_OK;
    }
    cufftSetStream(p->fwd, s);
    cufftSetStream(p->inv, s);
    cufftResult r = cufftExecD2Z(p->fwd, p->rho, (cufftDoubleComplex*)p->fr);
    if (r != CUFFT_SUCCESS) return cufft_err(ctx, r, "cufftExecD2Z (density)");
    const long long m = np * (p->n + 1);
    k_spectrum_mul_2d<<<blocks_for(m, 256), 256, 0, s>>>(p->fr, p->fkx, p->fky, m, 1.0 / (double)(np * np), p->sx,
                                                         p->sy);
    SSS_LAUNCH_CHECK(ctx, "k_spectrum_mul_2d");
    r = cufftExecZ2D(p->inv, (cufftDoubleComplex*)p->sx, p->fieldx);
    if (r == CUFFT_SUCCESS) r = cufftExecZ2D(p->inv, (cufftDoubleComplex*)p->sy, p->fieldy);
    if (r != CUFFT_SUCCESS) return cufft_err(ctx, r, "cufftExecZ2D");
    return SSS_OK;
}

// Accelerations at (px, py) from the last field (pm_kernel.py:150-154).
extern "C" int sss_pm2d_gather(sss_pm2d* p, const double* px, const double* py, int64_t n, double x0, double y0,
                               double h, double* ax, double* ay, void* stream) {
    if (!p) return SSS_ERR_ARG;
    if (n <= 0) return SSS_OK;
    if (!px || !py || !ax || !ay) return sss_set_err(p->ctx, SSS_ERR_ARG, "gather: NULL");
    if (p->own)
        k_cic_gather_pairs_2d<<<blocks_for(n, 128), 128, 0, (cudaStream_t)stream>>>(px, py, n, p->n, x0, y0, h,
                                                                                   p->pairs, ax, ay);
    else
        k_cic_gather_2d<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(px, py, n, p->n, x0, y0, h, p->fieldx,
                                                                             p->fieldy, ax, ay);
    SSS_LAUNCH_CHECK(p->ctx, "k_cic_gather_2d");
    return SSS_OK;
}

// One field read at (px, py) with the deposit's stencil (_cic_gather, pm_kernel.py:93-107).
extern "C" int sss_pm2d_gather_field(sss_ctx* ctx, const double* field, int grid_n, int64_t ld, const double* px,
                                     const double* py, int64_t n, double x0, double y0, double h, double* out,
                                     void* stream) {
    if (!ctx) return SSS_ERR_ARG;
    if (grid_n < 2 || ld < grid_n || n < 0) return sss_set_err(ctx, SSS_ERR_ARG, "gather_field: bad sizes");
    if (n == 0) return SSS_OK;
    if (!field || !px || !py || !out) return sss_set_err(ctx, SSS_ERR_ARG, "gather_field: NULL");
    k_cic_gather_field_2d<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(px, py, n, grid_n, ld, x0, y0, h,
                                                                               field, out);
    SSS_LAUNCH_CHECK(ctx, "k_cic_gather_field_2d");
    return SSS_OK;
}

// The [0:N, 0:N] crops of the last field into ax, ay (device, N*N each).
extern "C" int sss_pm2d_fields(sss_pm2d* p, double* ax, double* ay, void* stream) {
    if (!p || !ax || !ay) return SSS_ERR_ARG;
    const size_t n = (size_t)p->n;
    cudaStream_t s = (cudaStream_t)stream;
    if (p->own) {
        k_split_pairs_2d<<<blocks_for((long long)(n * n), 256), 256, 0, s>>>(p->pairs, (long long)(n * n), ax, ay);
        SSS_LAUNCH_CHECK(p->ctx, "k_split_pairs_2d");
        return SSS_OK;
    }
    SSS_CUDA_TRY(p->ctx, cudaMemcpy2DAsync(ax, n * sizeof(double), p->fieldx, 2 * n * sizeof(double),
                                           n * sizeof(double), n, cudaMemcpyDeviceToDevice, s));
    SSS_CUDA_TRY(p->ctx, cudaMemcpy2DAsync(ay, n * sizeof(double), p->fieldy, 2 * n * sizeof(double),
                                           n * sizeof(double), n, cudaMemcpyDeviceToDevice, s));
    return SSS_OK;
}

// Density grid (N x N crop of the padded deposit) into rho (device, N*N).
extern "C" int sss_pm2d_density(sss_pm2d* p, double* rho, void* stream) {
    if (!p || !rho) return SSS_ERR_ARG;
    const size_t n = (size_t)p->n;
    SSS_CUDA_TRY(p->ctx, cudaMemcpy2DAsync(rho, n * sizeof(double), p->rho, p->ld * sizeof(double),
                                           n * sizeof(double), n, cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
    return SSS_OK;
}

// KDK piece: v += hdt a; if drift: x += dt v.
extern "C" int sss_pm2d_kick_drift(sss_pm2d* p, double* x, double* y, double* vx, double* vy, const double* ax,
                                   const double* ay, int64_t n, double hdt, double dt, int drift, void* stream) {
    if (!p) return SSS_ERR_ARG;
    if (n <= 0) return SSS_OK;
    k_kick_drift_2d<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(x, y, vx, vy, ax, ay, n, hdt, dt, drift);
    SSS_LAUNCH_CHECK(p->ctx, "k_kick_drift_2d");
    return SSS_OK;
}

// f32 copy of an f64 array (snapshot rows).
extern "C" int sss_pm2d_to_f32(sss_pm2d* p, const double* a, int64_t n, float* out, void* stream) {
    if (!p) return SSS_ERR_ARG;
    if (n <= 0) return SSS_OK;
    k_snap_2d<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(a, n, out);
    SSS_LAUNCH_CHECK(p->ctx, "k_snap_2d");
    return SSS_OK;
}

// Steps of NBodyPM.step_batch (pm_kernel.py:246-280) with a softening tied to
// the cell size, for the grids that convolve with the kernels of this file:
// the geometry of every step stays on the device. *kernel_h (host, in and
// out; <= 0: none yet) is the cell size the force kernels stand for.
extern "C" int sss_pm2d_step_batch(sss_pm2d* p, const sss_pm2d_bodies* st, double dt, int steps, double soft_cells,
                                   double margin_cells, double G, double* kernel_h, float* snap, void* stream) {
    if (!p) return SSS_ERR_ARG;
    sss_ctx* ctx = p->ctx;
    if (!p->own) return sss_set_err(ctx, SSS_ERR_ARG, "step_batch: this grid size steps by its parts");
    if (!st || !kernel_h || !snap || steps < 1 || st->n < 1 || st->t < 0)
        return sss_set_err(ctx, SSS_ERR_ARG, "step_batch: bad input");
    Bodies2d b;
    for (int k = 0; k < 2; ++k) {
        b.x[k] = st->x[k]; b.y[k] = st->y[k]; b.vx[k] = st->vx[k]; b.vy[k] = st->vy[k];
        b.ax[k] = st->ax[k]; b.ay[k] = st->ay[k];
        if ((k == 0 || st->t > 0) && (!b.x[k] || !b.y[k] || !b.vx[k] || !b.vy[k] || !b.ax[k] || !b.ay[k]))
            return sss_set_err(ctx, SSS_ERR_ARG, "step_batch: NULL array");
    }
    if (!st->m) return sss_set_err(ctx, SSS_ERR_ARG, "step_batch: NULL masses");
    b.n = st->n;
    b.t = st->t;
    SSS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = (cudaStream_t)stream;
    int rc = pm2d_unit_spectrum(p, soft_cells * soft_cells, s);
    if (rc) return rc;
    const double np = 2.0 * p->n, hdt = 0.5 * dt;
    const long long row = 4 * b.n + 2 * b.t;
    const unsigned want = blocks_for(b.n + b.t, 256), nb = want < 1024 ? want : 1024;
    SSS_CUDA_TRY(ctx, cudaMemcpyAsync(&p->geo->kernel_h, kernel_h, sizeof(double), cudaMemcpyHostToDevice, s));
    k_move_2d<<<nb, 256, 0, s>>>(b, p->n, p->geo, nullptr, 1, hdt, dt, nullptr, p->bb_part);
    for (int k = 0; k < steps; ++k) {
        k_geo_2d<<<1, 256, 0, s>>>(p->bb_part, (int)nb, p->n - 2.0 * margin_cells, margin_cells, G, np * np, p->geo);
        SSS_CUDA_TRY(ctx, cudaMemsetAsync(p->rho, 0, (size_t)p->n * p->n * sizeof(double), s));
        k_cic_deposit_2d<<<blocks_for(b.n, 256), 256, 0, s>>>(b.x[0], b.y[0], st->m, b.n, p->n, p->n, 0.0, 0.0, 1.0,
                                                             p->rho, p->geo);
        p->conv.rows_fwd<<<p->grid[0], p->conv.threads, p->smem, s>>>(p->tw, p->rho, p->t1);
        p->conv.cols<<<p->grid[1], p->conv.threads, p->smem, s>>>(p->tw, p->t1, p->u, p->v, 0.0, p->geo, p->slots,
                                                                 p->t2);
        p->conv.rows_inv<<<p->grid[2], p->conv.threads, p->smem, s>>>(p->tw, p->t2, p->pairs);
        k_move_2d<<<nb, 256, 0, s>>>(b, p->n, p->geo, p->pairs, k + 1 < steps, hdt, dt, snap + k * row, p->bb_part);
        SSS_LAUNCH_CHECK(ctx, "pm2d step");
    }
    Geo g;
    SSS_CUDA_TRY(ctx, cudaMemcpyAsync(&g, p->geo, sizeof(Geo), cudaMemcpyDeviceToHost, s));
    SSS_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    *kernel_h = g.kernel_h;
    p->scale = g.scale;
    return SSS_OK;
}

extern "C" int sss_pm2d_steps_natively(sss_pm2d* p) { return p && p->own ? 1 : 0; }
