// Internal helpers shared by the libsss translation units: the context,
// error plumbing, and the sm_100a primitives (mbarrier, bulk async copy,
// bounded waits) the kernels are built from.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>
#include <string.h>

#include "../../include/sss.h"

#define SSS_AP_KERNELS 18   // all-pairs force kernels by dimension, precision, size and softening

struct sss_ctx {
    int device;
    int num_sms;
    char err[512];
    // scratch owned by the context (grown on demand, freed by sss_destroy)
    void* scratch;
    size_t scratch_bytes;
    // device status word written by bounded waits (SSS_ERR_TIMEOUT ...)
    int* d_status;
    // chunk-arrival counters of the all-pairs kernels (kept zero between
    // launches: the last chunk of a target block resets its counter)
    unsigned* d_counters;
    size_t n_counters;
    // cached CTAs-per-SM of the all-pairs kernels (0 = not yet queried)
    int occ[SSS_AP_KERNELS];
    // the broadphase pipeline as an instantiated graph (broadphase.cu)
    struct sss_bp_graph* bp_graph;
};

void sss_bp_graph_free(struct sss_bp_graph* g);

int sss_set_err(sss_ctx* ctx, int code, const char* fmt, ...);
int sss_cuda_err(sss_ctx* ctx, cudaError_t e, const char* what);
// Ensure ctx->scratch holds at least `bytes` (256-byte aligned).
int sss_scratch(sss_ctx* ctx, size_t bytes, void** out);
int sss_counters(sss_ctx* ctx, size_t n, unsigned** out);
// Bounded-wait self-tests (a wait that nothing completes; sss_selftest_wait).
int sss_frame_barrier_selftest(sss_ctx* ctx, double limit_s, cudaStream_t s);
int sss_stream_barrier_selftest(sss_ctx* ctx, double limit_s, cudaStream_t s);

#define SSS_CUDA_TRY(ctx, call)                                   \
    do {                                                          \
        cudaError_t e__ = (call);                                 \
        if (e__ != cudaSuccess) return sss_cuda_err(ctx, e__, #call); \
    } while (0)

#define SSS_LAUNCH_CHECK(ctx, what)                               \
    do {                                                          \
        cudaError_t e__ = cudaGetLastError();                     \
        if (e__ != cudaSuccess) return sss_cuda_err(ctx, e__, what); \
    } while (0)

// ------------------------------------------------------------ device side

// Wall-clock limit of every spin on an mbarrier or flag (nanoseconds). A
// legitimate wait here is microseconds; the limit only turns a would-be hang
// into an SSS_ERR_TIMEOUT status.
#define SSS_WAIT_LIMIT_NS 2000000000ull

__device__ __forceinline__ uint64_t sss_globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned sss_smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void sss_mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(sss_smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void sss_mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;"
                 :: "r"(sss_smem_addr(bar)), "r"(count) : "memory");
}

// Make mbarrier initialisation visible to the async (bulk-copy) proxy.
__device__ __forceinline__ void sss_fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void sss_mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(sss_smem_addr(bar)), "r"(bytes) : "memory");
}

// 1-D bulk copy global -> shared, completion counted on `bar` (bytes must be
// a multiple of 16, both addresses 16-byte aligned).
__device__ __forceinline__ void sss_bulk_g2s(void* dst, const void* src, unsigned bytes,
                                             uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        :: "r"(sss_smem_addr(dst)), "l"(src), "r"(bytes), "r"(sss_smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ bool sss_mbar_try_wait(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(sss_smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}

// Bounded wait for phase `parity` of `bar`. Returns false (and records
// SSS_ERR_TIMEOUT in *status) if the phase did not complete within limit_ns.
__device__ __forceinline__ bool sss_mbar_wait_bounded(uint64_t* bar, unsigned parity,
                                                      int* status, uint64_t limit_ns = SSS_WAIT_LIMIT_NS) {
    if (sss_mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = sss_globaltimer();
    while (!sss_mbar_try_wait(bar, parity)) {
        if (sss_globaltimer() - t0 > limit_ns) {
            atomicExch(status, SSS_ERR_TIMEOUT);
            return false;
        }
    }
    return true;
}

// ------------------------------------------------------------- f64 kernels

__device__ __forceinline__ float sss_rsqrt_approx_f32(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Gm * r2^(-3/2) in f64 from the hardware's approximate reciprocal square root.
//
// Method (Householder-type series refinement of 1/sqrt, e.g. Householder,
// "The Numerical Treatment of a Single Nonlinear Equation", 1970): with a
// seed c ~ r2^(-1/2) and e = 1 - r2*c^2, the exact value is
//   r2^(-3/2) = c^3 (1 - e)^(-3/2) = c^3 (1 + 3/2 e + 15/8 e^2 + 35/16 e^3 + ...).
// The seed is rsqrt.approx.ftz.f64 (a coarse value over the full f64 range,
// no conversion of r2 or of the seed). Measured over 128 binades: |e| <
// 1.9e-6, so the cubic remainder is < 1.5e-17 and the series is cut after
// e^2; the result is within 2.3e-16 (rms 7.2e-17), against 5.5e-16 (1.6e-16)
// of the cube of CUDA's rsqrt and 2.7e-16 (8.1e-17) of 1 / (r2 sqrt(r2)), at
// 74 clocks of latency against 88 and 168 and 1.7 and 3.6 times their rate.
// 0 for r2 = +inf.
__device__ __forceinline__ double sss_gm_rinv3(double gm, double r2) {
    double c;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(c) : "d"(r2));
    const double c2 = c * c;
    double e = fma(-r2, c2, 1.0);
    // r2 = +inf: -inf * 0 is NaN, whose low word alone is a number near 0
    e = __hiloint2double(__double2hiint(c) == 0 ? 0 : __double2hiint(e), __double2loint(e));
    const double p = fma(e, 1.875, 1.5);
    const double g3 = (gm * c) * c2;
    return fma(g3, e * p, g3);
}

// 1 / d for a normal d > 0: the hardware's coarse reciprocal and two Newton
// steps r (2 - d r); within 2^-53 of it (tests/test_device_math_gpu.py). No branch,
// so the 16 modes of a thread of the 3-D mesh's x pass overlap; with a division
// each (its slow path a branch) the 64^3 pass took 14 us.
__device__ __forceinline__ double sss_recip_f64(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = fma(r, fma(-d, r, 1.0), r);
    return fma(r, fma(-d, r, 1.0), r);
}

// f32 hypot, correctly rounded as the C library's hypotf (which NumPy calls for float32
// hypot): the squares of f32 values are exact in f64, their sum is rounded once, the square
// root once, then the result to f32.
__device__ __forceinline__ float sss_hypot_f32(float x, float y) {
    if (isinf(x) || isinf(y)) return __int_as_float(0x7F800000);
    const double xd = x, yd = y;
    return __double2float_rn(__dsqrt_rn(__dadd_rn(__dmul_rn(xd, xd), __dmul_rn(yd, yd))));
}
