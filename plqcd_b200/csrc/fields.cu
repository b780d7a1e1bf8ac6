// fields.cu -- layout conversion and generation of device fields.
//
// API layout (include/su3.h): a spinor field is V spinors of 12 interleaved
// complex doubles in even/odd site order; a gauge field is 4V su3 links,
// link (i, mu) at u[4*i + mu] (lib/dirac.c:155, 262). The kernels here move
// between that array-of-structures layout and the structure-of-arrays
// layouts the hopping kernels read (include/plqcd_b200.h), in any storage
// precision, and generate random fields from a counter-based generator.
#include <cuda_runtime.h>

#include "device_fields.cuh"
#include "internal.h"
#include "philox.h"

namespace plqcd {
namespace dev {

constexpr int kBlock = 256;

inline unsigned nblocks(long n) { return (unsigned)((n + kBlock - 1) / kBlock); }

template <typename R>
__device__ __forceinline__ void to_real(const cx<double> in[12], cx<R> out[12]) {
#pragma unroll
    for (int k = 0; k < 12; k++) out[k] = {(R)in[k].re, (R)in[k].im};
}

// ---- API-layout staging ---------------------------------------------------------
// A site is contiguous in the API layout (12 complexes of a spinor, 36 of
// its four links) and spread over planes on the device. The import and
// export kernels move the API side through shared memory: consecutive
// threads copy consecutive 16-byte complexes, so both sides are whole
// 512-byte transactions per warp. A site takes an odd number of 16-byte
// slots there (13, 37), so that the 8 lanes of a 128-byte phase, one site
// each, fall on distinct banks. The bound is DRAM. At 24^3x48 in FP64 the
// export, which stored 16 bytes per 192-byte stride and thread, went from
// 34.5 us to 25.6 us per parity (5.0 TB/s), the import stayed at
// 22.7 us, the links went from 129 to 119 us (6.4 TB/s); both parities and
// the links together from 268 to 214 us.
constexpr int kSpinorSites = 128;  // sites (and threads) of a block
constexpr int kLinkSites = 32;     // sites of a block of 128 threads, one link each

// complexes of the n sites at `src` -> slots of `per + 1` at `st` (commit and wait included)
template <int PER, int SITES>
__device__ __forceinline__ void stage_sites(double2 *st, const double2 *__restrict__ src, int n) {
    const uint32_t s0 = smem_addr(st);
#pragma unroll
    for (int i = threadIdx.x; i < PER * SITES; i += 128)
        if (i < PER * n) cp_async16_cg(s0 + (uint32_t)(i + i / PER) * 16u, src + i);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
}

// ---- spinors ------------------------------------------------------------------
template <int PREC>
__global__ void __launch_bounds__(kSpinorSites) k_spinor_import(const double2 *__restrict__ aos, long Vh, int parity,
                                                                void *dst, long first, long count) {
    __shared__ double2 st[kSpinorSites * 13];
    const long b0 = (long)blockIdx.x * kSpinorSites;  // first site of the block, from `first`
    const int n = (int)min((long)kSpinorSites, count - b0);
    stage_sites<12, kSpinorSites>(st, aos + (parity * Vh + first + b0) * 12, n);
    if ((int)threadIdx.x >= n) return;
    cx<double> s[12];
#pragma unroll
    for (int k = 0; k < 12; k++) {
        double2 v = st[threadIdx.x * 13 + k];
        s[k] = {v.x, v.y};
    }
    using R = typename SpinorIO<PREC>::real;
    cx<R> r[12];
    to_real(s, r);
    SpinorIO<PREC>::store(dst, Vh, first + b0 + threadIdx.x, r);
}

template <int PREC>
__global__ void __launch_bounds__(kSpinorSites) k_spinor_export(const void *src, long Vh, int parity,
                                                                double2 *__restrict__ aos, long first, long count) {
    __shared__ double2 st[kSpinorSites * 13];
    const long b0 = (long)blockIdx.x * kSpinorSites;
    const int n = (int)min((long)kSpinorSites, count - b0);
    if ((int)threadIdx.x < n) {
        using R = typename SpinorIO<PREC>::real;
        cx<R> r[12];
        SpinorIO<PREC>::load(src, Vh, first + b0 + threadIdx.x, r);
#pragma unroll
        for (int k = 0; k < 12; k++) st[threadIdx.x * 13 + k] = make_double2((double)r[k].re, (double)r[k].im);
    }
    __syncthreads();
    double2 *p = aos + (parity * Vh + first + b0) * 12;
#pragma unroll
    for (int i = threadIdx.x; i < 12 * kSpinorSites; i += kSpinorSites)
        if (i < 12 * n) st_cs(p + i, st[i + i / 12]);
}

// split real / imaginary planes: component k of staged site h at re[12*h+k]
template <int PREC>
__global__ void k_spinor_import_split(const double *__restrict__ re, const double *__restrict__ im, long Vh,
                                      void *dst) {
    long h = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    using R = typename SpinorIO<PREC>::real;
    cx<R> r[12];
#pragma unroll
    for (int k = 0; k < 12; k++) r[k] = {(R)re[12 * h + k], (R)im[12 * h + k]};
    SpinorIO<PREC>::store(dst, Vh, h, r);
}

template <int PREC>
__global__ void k_spinor_export_split(const void *src, long Vh, double *__restrict__ re, double *__restrict__ im) {
    long h = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    using R = typename SpinorIO<PREC>::real;
    cx<R> r[12];
    SpinorIO<PREC>::load(src, Vh, h, r);
#pragma unroll
    for (int k = 0; k < 12; k++) {
        re[12 * h + k] = (double)r[k].re;
        im[12 * h + k] = (double)r[k].im;
    }
}

template <int DP, int SP>
__global__ void k_spinor_convert(void *dst, const void *src, long Vh) {
    long h = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    using RS = typename SpinorIO<SP>::real;
    using RD = typename SpinorIO<DP>::real;
    cx<RS> s[12];
    SpinorIO<SP>::load(src, Vh, h, s);
    cx<RD> d[12];
#pragma unroll
    for (int k = 0; k < 12; k++) d[k] = {(RD)s[k].re, (RD)s[k].im};
    SpinorIO<DP>::store(dst, Vh, h, d);
}

template <int PREC>
__global__ void k_spinor_gaussian(void *dst, long Vh, int parity, uint64_t seed) {
    long h = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= Vh) return;
    const uint64_t site = (uint64_t)parity * Vh + h;
    cx<double> s[12];
#pragma unroll
    for (int k = 0; k < 12; k++) {
        double2 g = philox_gaussian_pair(seed, site, kTagSpinor, (uint32_t)k);
        s[k] = {g.x, g.y};
    }
    using R = typename SpinorIO<PREC>::real;
    cx<R> r[12];
    to_real(s, r);
    SpinorIO<PREC>::store(dst, Vh, h, r);
}

// ---- gauge --------------------------------------------------------------------
// the four links of the sites [first, first + n) (even/odd index over both
// parities); `aos` points at the first one. Warp mu of a block stores the
// direction-mu links of 32 consecutive sites (a block may span the parities)
template <int PREC, int RECON>
__global__ void __launch_bounds__(4 * kLinkSites) k_gauge_import(const double2 *__restrict__ aos, long first, long n,
                                                                 long Vh, void *dst) {
    __shared__ double2 st[kLinkSites * 37];
    const long b0 = (long)blockIdx.x * kLinkSites;
    const int nb = (int)min((long)kLinkSites, n - b0);
    stage_sites<36, kLinkSites>(st, aos + b0 * 36, nb);
    const int mu = threadIdx.x / kLinkSites, j = threadIdx.x % kLinkSites;
    if (j >= nb) return;
    const long i = first + b0 + j;
    const int par = i >= Vh;
    cx<double> U[9];
#pragma unroll
    for (int e = 0; e < 9; e++) {
        double2 v = st[j * 37 + mu * 9 + e];
        U[e] = {v.x, v.y};
    }
    LinkIO<PREC, RECON>::store(dst, Vh, par, mu, i - par * Vh, U);
}

// links from split planes: element e of staged link k at re[9*k+e]
template <int PREC, int RECON>
__global__ void k_gauge_import_split(const double *__restrict__ re, const double *__restrict__ im, long first,
                                     long n, long Vh, void *dst) {
    long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    long l = first + k;
    long i = l >> 2;
    int mu = (int)(l & 3);
    int par = i >= Vh;
    long h = i - par * Vh;
    cx<double> U[9];
#pragma unroll
    for (int e = 0; e < 9; e++) U[e] = {re[9 * k + e], im[9 * k + e]};
    LinkIO<PREC, RECON>::store(dst, Vh, par, mu, h, U);
}

template <int PREC, int RECON>
__global__ void k_gauge_export(const void *src, long Vh, double2 *__restrict__ aos) {
    long l = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= 8 * Vh) return;
    long i = l >> 2;
    int mu = (int)(l & 3);
    int par = i >= Vh;
    long h = i - par * Vh;
    using R = typename LinkIO<PREC, RECON>::real;
    cx<R> U[9];
    LinkIO<PREC, RECON>::load(src, Vh, par, mu, h, U);
    double2 *p = aos + l * 9;
#pragma unroll
    for (int e = 0; e < 9; e++) p[e] = make_double2((double)U[e].re, (double)U[e].im);
}

// Random SU(3): Gaussian complex 3x3; rows 0,1 Gram-Schmidt orthonormalised;
// row 2 = conj(row0 x row1) (det = 1).
template <int PREC, int RECON>
__global__ void k_gauge_random(void *dst, long Vh, uint64_t seed) {
    long l = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= 8 * Vh) return;
    long i = l >> 2;
    int mu = (int)(l & 3);
    int par = i >= Vh;
    long h = i - par * Vh;
    cx<double> U[9];
#pragma unroll
    for (int e = 0; e < 6; e++) {
        double2 g = philox_gaussian_pair(seed, (uint64_t)i, kTagGauge + mu, (uint32_t)e);
        U[e] = {g.x, g.y};
    }
    double n0 = 0;
#pragma unroll
    for (int b = 0; b < 3; b++) n0 += U[b].re * U[b].re + U[b].im * U[b].im;
    n0 = rsqrt(n0);
#pragma unroll
    for (int b = 0; b < 3; b++) U[b] = {U[b].re * n0, U[b].im * n0};
    cx<double> d = {0, 0};  // <row0, row1>
#pragma unroll
    for (int b = 0; b < 3; b++) d = cadd(d, conjmul(U[b], U[3 + b]));
#pragma unroll
    for (int b = 0; b < 3; b++) U[3 + b] = csub(U[3 + b], cmul(d, U[b]));
    double n1 = 0;
#pragma unroll
    for (int b = 0; b < 3; b++) n1 += U[3 + b].re * U[3 + b].re + U[3 + b].im * U[3 + b].im;
    n1 = rsqrt(n1);
#pragma unroll
    for (int b = 0; b < 3; b++) U[3 + b] = {U[3 + b].re * n1, U[3 + b].im * n1};
    reconstruct_row2(U);
    LinkIO<PREC, RECON>::store(dst, Vh, par, mu, h, U);
}

template <int PREC, int RECON>
__global__ void k_gauge_unit(void *dst, long Vh) {
    long l = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= 8 * Vh) return;
    long i = l >> 2;
    int mu = (int)(l & 3);
    int par = i >= Vh;
    long h = i - par * Vh;
    cx<double> U[9];
#pragma unroll
    for (int e = 0; e < 9; e++) U[e] = {(e % 4 == 0) ? 1.0 : 0.0, 0.0};
    LinkIO<PREC, RECON>::store(dst, Vh, par, mu, h, U);
}

template <int DP, int DR, int SP, int SR>
__global__ void k_gauge_copy(void *dst, const void *src, long Vh) {
    long l = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= 8 * Vh) return;
    long i = l >> 2;
    int mu = (int)(l & 3);
    int par = i >= Vh;
    long h = i - par * Vh;
    using R = typename LinkIO<SP, SR>::real;
    cx<R> U[9];
    LinkIO<SP, SR>::load(src, Vh, par, mu, h, U);
    cx<double> D[9];
#pragma unroll
    for (int e = 0; e < 9; e++) D[e] = {(double)U[e].re, (double)U[e].im};
    LinkIO<DP, DR>::store(dst, Vh, par, mu, h, D);
}

}  // namespace dev

// ---- dispatch helpers ------------------------------------------------------------

#define PLQCD_SPINOR_SWITCH(prec, F)                          \
    switch (prec) {                                           \
        case PLQCD_F64: F(PLQCD_F64); break;                  \
        case PLQCD_F32: F(PLQCD_F32); break;                  \
        case PLQCD_F16: F(PLQCD_F16); break;                  \
        case PLQCD_BF16: F(PLQCD_BF16); break;                \
        default: return set_error(PLQCD_ERR_ARG, "unknown spinor precision %d", prec); \
    }

#define PLQCD_GAUGE_SWITCH(prec, recon, F)                                       \
    switch ((prec) * 100 + (recon)) {                                            \
        case PLQCD_F64 * 100 + 18: F(PLQCD_F64, 18); break;                      \
        case PLQCD_F64 * 100 + 12: F(PLQCD_F64, 12); break;                      \
        case PLQCD_F32 * 100 + 18: F(PLQCD_F32, 18); break;                      \
        case PLQCD_F32 * 100 + 12: F(PLQCD_F32, 12); break;                      \
        case PLQCD_F16 * 100 + 12: F(PLQCD_F16, 12); break;                      \
        case PLQCD_BF16 * 100 + 12: F(PLQCD_BF16, 12); break;                    \
        default: return set_error(PLQCD_ERR_ARG, "unsupported gauge format %d/%d", prec, recon); \
    }

int launch_spinor_import(const Geom &g, cudaStream_t s, const void *aos, int parity, void *dst, int prec, long first,
                         long count) {
    PLQCD_TRY(check_field_ptr(aos, "spinor import (API layout)"));
    PLQCD_TRY(check_field_ptr(dst, "spinor import"));
    if (count < 0) count = g.Vh - first;
    if (count < 1) return set_error(PLQCD_ERR_ARG, "spinor import: %ld sites", count);
    const unsigned nb = (unsigned)((count + dev::kSpinorSites - 1) / dev::kSpinorSites);
#define F(P) dev::k_spinor_import<P><<<nb, dev::kSpinorSites, 0, s>>>((const double2 *)aos, g.Vh, parity, dst, first, count)
    PLQCD_SPINOR_SWITCH(prec, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_spinor_export(const Geom &g, cudaStream_t s, const void *src, int prec, int parity, void *aos, long first,
                         long count) {
    PLQCD_TRY(check_field_ptr(src, "spinor export"));
    PLQCD_TRY(check_field_ptr(aos, "spinor export (API layout)"));
    if (count < 0) count = g.Vh - first;
    if (count < 1) return set_error(PLQCD_ERR_ARG, "spinor export: %ld sites", count);
    const unsigned nb = (unsigned)((count + dev::kSpinorSites - 1) / dev::kSpinorSites);
#define F(P) dev::k_spinor_export<P><<<nb, dev::kSpinorSites, 0, s>>>(src, g.Vh, parity, (double2 *)aos, first, count)
    PLQCD_SPINOR_SWITCH(prec, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_spinor_import_split(const Geom &g, cudaStream_t s, const double *re, const double *im, void *dst,
                               int prec) {
#define F(P) dev::k_spinor_import_split<P><<<dev::nblocks(g.Vh), dev::kBlock, 0, s>>>(re, im, g.Vh, dst)
    PLQCD_SPINOR_SWITCH(prec, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_spinor_export_split(const Geom &g, cudaStream_t s, const void *src, int prec, double *re, double *im) {
#define F(P) dev::k_spinor_export_split<P><<<dev::nblocks(g.Vh), dev::kBlock, 0, s>>>(src, g.Vh, re, im)
    PLQCD_SPINOR_SWITCH(prec, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_gauge_import_split(const Geom &g, cudaStream_t s, const double *re, const double *im, long first, long n,
                              void *dst, int prec, int recon) {
#define F(P, R) dev::k_gauge_import_split<P, R><<<dev::nblocks(n), dev::kBlock, 0, s>>>(re, im, first, n, g.Vh, dst)
    PLQCD_GAUGE_SWITCH(prec, recon, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_spinor_convert(const Geom &g, cudaStream_t s, void *dst, int dprec, const void *src, int sprec) {
    PLQCD_TRY(check_field_ptr(dst, "spinor convert"));
    PLQCD_TRY(check_field_ptr(src, "spinor convert"));
#define G(DP, SP) dev::k_spinor_convert<DP, SP><<<dev::nblocks(g.Vh), dev::kBlock, 0, s>>>(dst, src, g.Vh)
#define F(DP)                                                  \
    switch (sprec) {                                           \
        case PLQCD_F64: G(DP, PLQCD_F64); break;               \
        case PLQCD_F32: G(DP, PLQCD_F32); break;               \
        case PLQCD_F16: G(DP, PLQCD_F16); break;               \
        case PLQCD_BF16: G(DP, PLQCD_BF16); break;             \
        default: return set_error(PLQCD_ERR_ARG, "unknown spinor precision %d", sprec); \
    }
    PLQCD_SPINOR_SWITCH(dprec, F)
#undef F
#undef G
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_spinor_gaussian(const Geom &g, cudaStream_t s, void *dst, int prec, int parity, uint64_t seed) {
    PLQCD_TRY(check_field_ptr(dst, "spinor gaussian"));
#define F(P) dev::k_spinor_gaussian<P><<<dev::nblocks(g.Vh), dev::kBlock, 0, s>>>(dst, g.Vh, parity, seed)
    PLQCD_SPINOR_SWITCH(prec, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_gauge_import(const Geom &g, cudaStream_t s, const void *aos, long first, long n, void *dst, int prec,
                        int recon) {
    PLQCD_TRY(check_field_ptr(aos, "gauge import (API layout)"));
    if (first < 0 || n < 4 || first % 4 || n % 4 || first + n > 8 * g.Vh)
        return set_error(PLQCD_ERR_ARG, "gauge import: links [%ld, %ld) are not whole sites", first, first + n);
    const unsigned nb = (unsigned)((n / 4 + dev::kLinkSites - 1) / dev::kLinkSites);
#define F(P, R) dev::k_gauge_import<P, R><<<nb, 4 * dev::kLinkSites, 0, s>>>((const double2 *)aos, first / 4, n / 4, g.Vh, dst)
    PLQCD_GAUGE_SWITCH(prec, recon, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_gauge_export(const Geom &g, cudaStream_t s, const void *src, int prec, int recon, void *aos) {
#define F(P, R) dev::k_gauge_export<P, R><<<dev::nblocks(8 * g.Vh), dev::kBlock, 0, s>>>(src, g.Vh, (double2 *)aos)
    PLQCD_GAUGE_SWITCH(prec, recon, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_gauge_random(const Geom &g, cudaStream_t s, void *dst, int prec, int recon, uint64_t seed) {
#define F(P, R) dev::k_gauge_random<P, R><<<dev::nblocks(8 * g.Vh), dev::kBlock, 0, s>>>(dst, g.Vh, seed)
    PLQCD_GAUGE_SWITCH(prec, recon, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_gauge_unit(const Geom &g, cudaStream_t s, void *dst, int prec, int recon) {
#define F(P, R) dev::k_gauge_unit<P, R><<<dev::nblocks(8 * g.Vh), dev::kBlock, 0, s>>>(dst, g.Vh)
    PLQCD_GAUGE_SWITCH(prec, recon, F)
#undef F
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

int launch_gauge_copy(const Geom &g, cudaStream_t s, void *dst, int dprec, int drecon, const void *src, int sprec,
                      int srecon) {
#define G(DP, DR, SP, SR) dev::k_gauge_copy<DP, DR, SP, SR><<<dev::nblocks(8 * g.Vh), dev::kBlock, 0, s>>>(dst, src, g.Vh)
#define F(SP, SR)                                                                    \
    switch (dprec * 100 + drecon) {                                                  \
        case PLQCD_F64 * 100 + 18: G(PLQCD_F64, 18, SP, SR); break;                  \
        case PLQCD_F64 * 100 + 12: G(PLQCD_F64, 12, SP, SR); break;                  \
        case PLQCD_F32 * 100 + 18: G(PLQCD_F32, 18, SP, SR); break;                  \
        case PLQCD_F32 * 100 + 12: G(PLQCD_F32, 12, SP, SR); break;                  \
        case PLQCD_F16 * 100 + 12: G(PLQCD_F16, 12, SP, SR); break;                  \
        case PLQCD_BF16 * 100 + 12: G(PLQCD_BF16, 12, SP, SR); break;                \
        default: return set_error(PLQCD_ERR_ARG, "unsupported gauge format %d/%d", dprec, drecon); \
    }
    PLQCD_GAUGE_SWITCH(sprec, srecon, F)
#undef F
#undef G
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

// ---- sizes -------------------------------------------------------------------------
size_t spinor_parity_bytes(long Vh, int prec) {
    switch (prec) {
        case PLQCD_F64: return (size_t)Vh * 192;
        case PLQCD_F32: return (size_t)Vh * 96;
        case PLQCD_F16:
        case PLQCD_BF16: return (size_t)Vh * 52;
        default: return 0;
    }
}

bool gauge_format_ok(int prec, int recon) {
    if (prec == PLQCD_F64 || prec == PLQCD_F32) return recon == 18 || recon == 12;
    if (prec == PLQCD_F16 || prec == PLQCD_BF16) return recon == 12;
    return false;
}

size_t gauge_elem_bytes(int prec, int recon) {
    if (prec == PLQCD_F64) return 16;
    if (prec == PLQCD_F32) return recon == 18 ? 8 : 16;
    return 8;
}

int gauge_elems(int prec, int recon) {
    if (prec == PLQCD_F64) return recon == 18 ? 9 : 6;
    if (prec == PLQCD_F32) return recon == 18 ? 9 : 3;
    return 3;
}

size_t gauge_total_bytes(long Vh, int prec, int recon) {
    if (!gauge_format_ok(prec, recon)) return 0;
    return (size_t)8 * Vh * gauge_elems(prec, recon) * gauge_elem_bytes(prec, recon);
}

}  // namespace plqcd
