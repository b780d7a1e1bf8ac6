// dslash_mrhs_links.cu -- FP64 multi-RHS hop: the links of a block's sites in
// shared memory, the spinors ahead in registers (sm_100a).
//
// A block of n warps covers 32 output sites for n right-hand sides (warp =
// RHS, lane = site). The warps share out the eight directions and copy their
// links into shared memory once (cp.async, each lane its own site's slots);
// after one barrier every warp computes its RHS, the next direction's
// neighbour spinor (and at the end the xpay operand) on its way into
// registers meanwhile. A link crosses L2->SM once per n RHS, which with the
// spinors is what bounds the hop beside latency at 8 warps per SM: at 16^3x32
// with 12 RHS and n = 2, 1.9 kB per site and RHS, 10.9 TB/s. Same arithmetic, so
// the same bits, as the other kernels. Threads past the last site or RHS copy
// in-bounds data and store nothing.
//
// Two or four RHS per block (222 registers, 8 warps per SM in blocks whose
// start-ups overlap), the tuner decides. us at 16^3x32 with 12 RHS and at
// 24^3x48 with 4 RHS, xpay, short bursts / back to back under the power cap:
// 2: 130 / 148 and 233 / 273, 4: 130 / 145 and 231 / 265, 8: 159 / 166; one RHS
// per block 172 and 319 (one measurement). Before: the TMA kernel with RHS
// tiles 142 / 157, one thread per RHS 261 / 297 at 24^3x48; links in shared
// memory with the spinors beside them 263 and 650.
#include <cuda_runtime.h>

#include "blas.cuh"
#include "dslash_core.cuh"
#include "hop_sum.cuh"
#include "internal.h"
#include "mrhs_core.cuh"
#include "pdl.cuh"
#include "raw_loads.cuh"

namespace plqcd {
namespace dev {

struct LinksSum {  // SUM of k_mrhs_links_f64
    HopSumKind kind;
    int out_prec;
    const char *c;
    size_t out_fbytes;
    double *partials;
};

constexpr int kLinkSlots = 8 * 9 * 32;  // 16-byte slots: [direction of dir_at][element][site]

// the links of the directions in `mine` at the block's 32 sites, copied by
// the calling warp (its lanes are the sites)
template <class LIO>
__device__ __forceinline__ void issue_links(uint4 *lk, unsigned mine, const void *gauge, long Vh, int par, int h,
                                            const int nb[8]) {
    const uint32_t s0 = smem_addr(lk) + (threadIdx.x & 31) * 16;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int d = dir_at(k);
        if (mine >> k & 1)
            LIO::issue(gauge, Vh, d < 4 ? par : par ^ 1, d & 3, d < 4 ? h : nb[d], s0 + k * (9 * 32 * 16), 32 * 16);
    }
    cp_async_commit();
}

// waits for them, rebuilds row 2 of 12-real links in place, and for the block
template <class LIO>
__device__ __forceinline__ void finish_links(uint4 *lk, unsigned mine) {
    const int lane = threadIdx.x & 31;
    cp_async_wait<0>();
    if constexpr (LIO::NSLOT < 9)
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (!(mine >> k & 1)) continue;
            uint4 *p = lk + k * (9 * 32) + lane;
            cx<double> U[9];
            LIO::load_staged(p, 32, U);
#pragma unroll
            for (int e = 6; e < 9; e++) *reinterpret_cast<double2 *>(p + e * 32) = make_double2(U[e].re, U[e].im);
        }
    __syncthreads();
}

// SUM (0: none): HOP_RESID or HOP_CHECK of blas.cuh per RHS, c and (in the
// format OP) the output being blocks of fields; the site blocks' sums go to
// the partials [RHS][site block], HOP_CHECK's second ones after them
template <class LIO, bool XPAY, int SUM = 0, int OP = PLQCD_F64>
__global__ void __maxnreg__(232) k_mrhs_links_f64(const MrhsArgs a, const LinksSum q) {
    using SIO = SpinorIO<PLQCD_F64>;
    __shared__ uint4 lk[kLinkSlots];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int grp = blockIdx.x % a.ntiles, sb = blockIdx.x / a.ntiles;
    const int r = grp * nw + w;
    const bool valid = sb * 32 + lane < a.Vh;
    const int h = valid ? sb * 32 + lane : (int)a.Vh - 1;
    const int par = a.out_parity;
    const long Vh = a.Vh;
    const Coords c = site_coords(h, par, a.L0h, a.L1, a.L2);
    const int xh = h - c.row * a.L0h;
    int nb[8];
    neighbour_sites(c, xh, a.L0, a.L0h, a.L1, a.L2, a.L3, nb);
    unsigned mine = 0;
    for (int k = w; k < 8; k += nw) mine |= 1u << k;
    pdl_start();
    issue_links<LIO>(lk, mine, a.gauge, Vh, par, h, nb);
    const bool has = r < a.nrhs;
    const char *in = a.in + (size_t)(has ? r : 0) * a.fbytes;
    const char *x = XPAY ? a.x + (size_t)(has ? r : 0) * a.fbytes : nullptr;
    RawSpinor<SIO> rs[2];
    auto issue = [&](int k) {
        if (k < 8)
            rs[k & 1].load(in, Vh, nb[dir_at(k)]);
        else if (XPAY)
            rs[0].load(x, Vh, h);
    };
    issue(0);
    finish_links<LIO>(lk, mine);
    if (!has || (SUM == 0 && !valid)) return;
    const double sg = a.g5_in;
    cx<double> acc[12];
#pragma unroll
    for (int k = 0; k < 12; k++) acc[k] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 8; k++) {
        issue(k + 1);
        cx<double> U[9], s[12];
        double n;
#pragma unroll
        for (int e = 0; e < 9; e++) {
            const double2 v = *reinterpret_cast<const double2 *>(lk + (k * 9 + e) * 32 + lane);
            U[e] = {v.x, v.y};
        }
        rs[k & 1].get(s, n);
        compute_dir_n<false, false, double>(dir_at(k), acc, s, U, sg, n);
    }
    const double aup = a.a_up, alow = a.a_low;
    if (XPAY) {
        cx<double> xv[12];
        double n;
        rs[0].get(xv, n);
        const double b = a.b;
#pragma unroll
        for (int k = 0; k < 12; k++) {
            const double ak = k < 6 ? aup : alow;
            acc[k] = {fma(ak, acc[k].re, b * xv[k].re), fma(ak, acc[k].im, b * xv[k].im)};
        }
    } else {
#pragma unroll
        for (int k = 0; k < 12; k++) {
            const double ak = k < 6 ? aup : alow;
            acc[k] = {ak * acc[k].re, ak * acc[k].im};
        }
    }
    if constexpr (SUM == 0) {
        SIO::store(a.out + (size_t)r * a.fbytes, Vh, h, acc);
    } else {
        double v = 0, u = 0;
        if (valid) {
            cx<double> cv[12];
            load_coherent<SIO>(q.c + (size_t)r * a.fbytes, Vh, h, cv);
            if (SUM == HOP_CHECK) u = site_norm2(cv);
#pragma unroll
            for (int k = 0; k < 12; k++) cv[k] = csub(cv[k], acc[k]);
            v = site_norm2(cv);
            if constexpr (SUM == HOP_RESID) {
                using RO = typename SpinorIO<OP>::real;
                cx<RO> z[12];
#pragma unroll
                for (int k = 0; k < 12; k++) z[k] = {(RO)cv[k].re, (RO)cv[k].im};
                SpinorIO<OP>::store(a.out + (size_t)r * q.out_fbytes, Vh, h, z);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_xor_sync(0xffffffffu, v, o);
            if (SUM == HOP_CHECK) u += __shfl_xor_sync(0xffffffffu, u, o);
        }
        if (lane == 0) {
            const size_t nsb = gridDim.x / a.ntiles;
            q.partials[(size_t)r * nsb + sb] = v;
            if (SUM == HOP_CHECK) q.partials[((size_t)a.nrhs + r) * nsb + sb] = u;
        }
    }
}

// one block per RHS (and second sum): its nsb partials in a fixed order
__global__ void __launch_bounds__(256) k_links_sum_finish(const double *partials, int nsb, double *out) {
    __shared__ double ws[8];
    const double *p = partials + (size_t)blockIdx.x * nsb;
    double t = 0;
#pragma unroll 4
    for (int i = threadIdx.x; i < nsb; i += 256) t += p[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x != 0) return;
    t = 0;
    for (int i = 0; i < 8; i++) t += ws[i];
    out[blockIdx.x] = t;
}

template <class L>
static void (*resid_kernel(int prec))(const MrhsArgs, const LinksSum) {
    switch (prec) {
        case PLQCD_F64: return k_mrhs_links_f64<L, true, HOP_RESID, PLQCD_F64>;
        case PLQCD_F32: return k_mrhs_links_f64<L, true, HOP_RESID, PLQCD_F32>;
        case PLQCD_F16: return k_mrhs_links_f64<L, true, HOP_RESID, PLQCD_F16>;
        case PLQCD_BF16: return k_mrhs_links_f64<L, true, HOP_RESID, PLQCD_BF16>;
        default: return nullptr;
    }
}

template <int RC>
static int launch_links(const Geom &g, cudaStream_t s, MrhsArgs a, int warps, bool xpay, const LinksSum *q = nullptr) {
    using L = LinkIO<PLQCD_F64, RC>;
    a.ntiles = (a.nrhs + warps - 1) / warps;
    const long nblk = (g.Vh + 31) / 32 * a.ntiles;
    if (nblk > 0x7fffffffL) return set_error(PLQCD_ERR_ARG, "dslash_mrhs: grid too large");
    auto k = xpay ? k_mrhs_links_f64<L, true> : k_mrhs_links_f64<L, false>;
    if (q) k = q->kind == HOP_CHECK ? k_mrhs_links_f64<L, true, HOP_CHECK> : resid_kernel<L>(q->out_prec);
    if (!k) return set_error(PLQCD_ERR_ARG, "dslash_mrhs: unknown precision %d", q->out_prec);
    return launch_overlapped(k, (unsigned)nblk, 32 * warps, s, a, q ? *q : LinksSum{});
}

}  // namespace dev

// FP64 hop of `warps` (1 to 8) RHS per block
int launch_mrhs_links(const Geom &g, cudaStream_t s, int recon, const dev::MrhsArgs &a, int warps, bool xpay) {
    if (warps < 1 || warps > 8) return set_error(PLQCD_ERR_ARG, "dslash_mrhs: %d RHS per block", warps);
    return recon == 18 ? dev::launch_links<18>(g, s, a, warps, xpay) : dev::launch_links<12>(g, s, a, warps, xpay);
}

int launch_mrhs_links_sum(const Geom &g, cudaStream_t s, const plqcd_gauge *gf, void *out, const void *in, int nrhs,
                          int out_parity, double a, const void *x, double b, const HopSum &h, double *partials,
                          double *sums) {
    dev::MrhsArgs m;
    PLQCD_TRY(mrhs_args(g, gf->data, PLQCD_F64, out, in, nrhs, out_parity, 0, a, x, b, m));
    PLQCD_TRY(check_field_ptr(h.c, "dslash_mrhs"));
    if (gf->prec != PLQCD_F64 || !x || (h.kind != HOP_RESID && h.kind != HOP_CHECK))
        return set_error(PLQCD_ERR_ARG, "dslash_mrhs: no such hop with sums");
    dev::LinksSum q;
    q.kind = h.kind;
    q.out_prec = h.out_prec;
    q.c = static_cast<const char *>(h.c);
    q.out_fbytes = spinor_parity_bytes(g.Vh, h.out_prec);
    q.partials = partials;
    // (two per block: four come out even where they fill it, and leave more
    // idle warps where they don't)
    const int warps = 2, sets = h.kind == HOP_CHECK ? 2 : 1;
    PLQCD_TRY(gf->recon == 18 ? dev::launch_links<18>(g, s, m, warps, true, &q)
                              : dev::launch_links<12>(g, s, m, warps, true, &q));
    dev::k_links_sum_finish<<<sets * nrhs, 256, 0, s>>>(partials, (int)((g.Vh + 31) / 32), sums);
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

// loads what launch_mrhs_links_sum runs for HOP_RESID (with lazy loading a
// kernel is otherwise loaded by its first launch, which may be captured)
int preload_mrhs_links_resid(int recon, int out_prec) {
    cudaFuncAttributes at;
    auto k = recon == 18 ? dev::resid_kernel<dev::LinkIO<PLQCD_F64, 18>>(out_prec)
                         : dev::resid_kernel<dev::LinkIO<PLQCD_F64, 12>>(out_prec);
    if (!k) return set_error(PLQCD_ERR_ARG, "dslash_mrhs: unknown precision %d", out_prec);
    PLQCD_CUDA_TRY(cudaFuncGetAttributes(&at, (const void *)k));
    PLQCD_CUDA_TRY(cudaFuncGetAttributes(&at, (const void *)dev::k_links_sum_finish));
    return PLQCD_OK;
}

}  // namespace plqcd
