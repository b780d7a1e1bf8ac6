// dslash_ahead.cu -- hopping matrix with the next directions' data in
// registers (sm_100a).
//
// Same operator and arithmetic order as the other kernels (lib/dirac.c:35-408
// eo, 414-791 oe; the same bits). One thread per output site, direct loads;
// before a direction is computed, the stored form of the spinor and link of
// the direction DEPTH steps later is already on its way into registers
// (raw_loads.cuh). Compared with the cp.async pipeline a staged byte does
// not pass the L1 data pipe a second and third time (written to and read
// from shared memory), and L1 stays a cache; compared with loading at the
// use, a thread waits for one latency per site instead of eight.
//
// Blocks are 64 threads; the register budget follows from the format:
// - FP64: the data of two directions and the accumulator take ~250
//   registers: 8 warps per SM, each with 336 bytes per lane in flight;
// - FP32: depth 1 or 2 at 128 registers (16 warps);
// - 16-bit: depth 1 at 96 registers (20 warps), the two FMA pipes being the
//   nearest bound (65% of the heavy one at 24^3x48, a third of it for the
//   conversions), or depth 2 at 128 for small lattices.
//
// What bounds it, and what it measured (us, before = the best kernel so far,
// three sets of fields in turn):
//   F32-18 xpay 32^3x64   175 -> 135   DRAM: 6.7 TB/s of its 864 bytes per site
//   F32-18 full 32^3x64   231 -> 180   DRAM and L2
//   F32-12 48^3x96        571 -> 527   DRAM: 5.8 TB/s
//   F16 xpay 32^3x64       96 -> 90    FMA pipes and latency
//   F64-18 xpay 24^3x48    97 -> 93    DRAM: 6.2 TB/s
//   F64-18 full 32^3x64   446 -> 441   latency at 8 warps; in a long run, where
//                         484 -> 430   the power cap lowers the clock
#include <cuda_runtime.h>

#include "dslash_core.cuh"
#include "internal.h"
#include "raw_loads.cuh"

namespace plqcd {
namespace dev {

constexpr int kAheadBlock = 64;

// Site number s of the full-lattice tile order: tiles of 2x2x2 rows in
// (y, z, t), y fastest within a tile and over the tiles. Every extent is
// even, so the tiles cover any lattice.
__device__ __forceinline__ Coords tiled_coords(int s, int par, int L0h, int L1, int L2, int *xh) {
    const int r = s / L0h;
    *xh = s - r * L0h;
    const int tile = r >> 3, n1 = L1 >> 1, n2 = L2 >> 1;
    const int q = tile / n1, t = q / n2;
    Coords c;
    c.y = 2 * (tile - q * n1) + (r & 1);
    c.z = 2 * (q - t * n2) + (r >> 1 & 1);
    c.t = 2 * t + (r >> 2 & 1);
    c.row = c.y + L1 * (c.z + L2 * c.t);
    c.x = 2 * *xh + ((c.y + c.z + c.t + par) & 1);
    return c;
}

// MODE 0: one parity; 1: with the xpay epilogue; 2: full lattice, the two
// parities of the same sites in neighbouring blocks; 3: full lattice, the
// two parities of 32 sites in one block (one warp each), sites in the 2x2x2
// tile order: the link a parity loads for its forward term is in L1 when
// the other one needs it for its backward term, and a tile's neighbour rows
// are loaded by blocks that run together (F64 at 32^3x64, long run: 429 us
// against 451 with the parities joined in the plain order and 462 in mode 2;
// 4x2x2 430, 2x4x4 447, 4x4x4 453, 2x8x8 452, half of z x all of t 445;
// short run 441 against 452 in mode 2).
template <class SIO, class LIO, int MODE, int DEPTH, int MINB>
__global__ void __launch_bounds__(kAheadBlock, MINB) k_dslash_ahead(const DslashArgs a) {
    using R = typename SIO::real;
    constexpr bool XPAY = MODE == 1, FULL = MODE >= 2;
    int par;
    long h;
    if (MODE == 3) {
        par = threadIdx.x >> 5;
        h = (long)blockIdx.x * 32 + (threadIdx.x & 31);
    } else if (MODE == 2) {
        par = blockIdx.x & 1;
        h = (long)(blockIdx.x >> 1) * kAheadBlock + threadIdx.x;
    } else {
        par = a.out_parity;
        h = a.h_begin + (long)(blockIdx.x / a.nrhs) * kAheadBlock + threadIdx.x;
    }
    if (h >= a.h_end) return;
    const int opp = par ^ 1;
    // selects, not a dynamic index into the parameter arrays (which would
    // copy them to local memory)
    const long roff = FULL ? 0 : (long)(blockIdx.x % a.nrhs) * a.fbytes;  // RHS of this block
    const void *in = (FULL && par == 0) ? a.in[1] : static_cast<const char *>(a.in[0]) + roff;
    void *out = (FULL && par == 1) ? a.out[1] : static_cast<char *>(a.out[0]) + roff;
    const long Vh = a.Vh;
    Coords c;
    int xh;
    if (MODE == 3) {
        c = tiled_coords((int)h, par, a.L0h, a.L1, a.L2, &xh);
        h = c.row * a.L0h + xh;
    } else {
        c = site_coords(h, par, a.L0h, a.L1, a.L2);
        xh = (int)(h - c.row * a.L0h);
    }
    int nb[8];
    neighbour_sites(c, xh, a.L0, a.L0h, a.L1, a.L2, a.L3, nb);

    constexpr int S = DEPTH + 1;
    RawSpinor<SIO> rs[S];
    RawLink<LIO> rl[S];
    // k-th direction of dir_at into slot k % S; k = 8: the xpay operand
    auto issue = [&](int k) {
        if (k < 8) {
            const int d = dir_at(k);
            rs[k % S].load(in, Vh, nb[d]);
            if (d < 4)
                rl[k % S].load(a.gauge, Vh, par, d, (int)h);
            else
                rl[k % S].load(a.gauge, Vh, opp, d - 4, nb[d]);
        } else if (XPAY && k == 8) {
            rs[8 % S].load(static_cast<const char *>(a.x) + roff, Vh, (int)h);
        }
    };
    cx<R> acc[12];
#pragma unroll
    for (int k = 0; k < 12; k++) acc[k] = {R(0), R(0)};
    const R sg = (R)a.g5_in;
#pragma unroll
    for (int k = 0; k < DEPTH; k++) issue(k);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        issue(k + DEPTH);
        cx<R> s[12], U[9];
        R n;
        rs[k % S].get(s, n);
        rl[k % S].get(U);
        compute_dir_n<false, SIO::kScaled, R, true>(dir_at(k), acc, s, U, sg, n);
    }
    const R aup = (R)a.a_up, alow = (R)a.a_low;
    if (XPAY) {
        cx<R> xv[12];
        R n;
        rs[8 % S].get(xv, n);
        const R b = (R)a.b;
#pragma unroll
        for (int k = 0; k < 12; k++) {
            const R ak = k < 6 ? aup : alow;
            if (SIO::kScaled) xv[k] = {xv[k].re * n, xv[k].im * n};
            acc[k] = {fma(ak, acc[k].re, b * xv[k].re), fma(ak, acc[k].im, b * xv[k].im)};
        }
    } else {
#pragma unroll
        for (int k = 0; k < 12; k++) {
            const R ak = k < 6 ? aup : alow;
            acc[k] = {ak * acc[k].re, ak * acc[k].im};
        }
    }
    SIO::store(out, Vh, h, acc);
}

template <class SIO, class LIO, int MODE, int DEPTH, int MINB>
static int launch_ahead_t(cudaStream_t s, const DslashArgs &a) {
    const long per = MODE == 3 ? 32 : kAheadBlock;
    const long nblk = (a.h_end - a.h_begin + per - 1) / per * (MODE == 2 ? 2 : a.nrhs);
    if (nblk > 0x7fffffffL) return set_error(PLQCD_ERR_ARG, "dslash: grid too large");
    k_dslash_ahead<SIO, LIO, MODE, DEPTH, MINB><<<(unsigned)nblk, kAheadBlock, 0, s>>>(a);
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

template <int P, int RC, int MODE>
static int launch_ahead_m(cudaStream_t s, const DslashArgs &a, bool deep) {
    using S = SpinorIO<P>;
    using L = LinkIO<P, RC>;
    if constexpr (P == PLQCD_F64) {
        return launch_ahead_t<S, L, MODE, 1, 4>(s, a);
    } else {
        if (deep) return launch_ahead_t<S, L, MODE, 2, 8>(s, a);
        return launch_ahead_t<S, L, MODE, 1, P == PLQCD_F32 ? 8 : 10>(s, a);
    }
}

template <int P, int RC>
static int launch_ahead_pr(cudaStream_t s, const DslashArgs &a, bool xpay, bool full, bool joined, bool deep) {
    if (full) {
        if constexpr (P == PLQCD_F64)
            if (joined) return launch_ahead_m<P, RC, 3>(s, a, false);
        return launch_ahead_m<P, RC, 2>(s, a, deep);
    }
    if (xpay) return launch_ahead_m<P, RC, 1>(s, a, deep);
    return launch_ahead_m<P, RC, 0>(s, a, deep);
}

}  // namespace dev

// deep: depth 2 (the FP32-computing formats; FP64 always loads one ahead);
// joined: mode 3 for the FP64 full lattice (without effect elsewhere)
int launch_dslash_ahead(cudaStream_t s, const dev::DslashArgs &a, int prec, int recon, bool xpay, bool full,
                        bool joined, bool deep) {
    switch (prec * 100 + recon) {
        case PLQCD_F64 * 100 + 18: return dev::launch_ahead_pr<PLQCD_F64, 18>(s, a, xpay, full, joined, deep);
        case PLQCD_F64 * 100 + 12: return dev::launch_ahead_pr<PLQCD_F64, 12>(s, a, xpay, full, joined, deep);
        case PLQCD_F32 * 100 + 18: return dev::launch_ahead_pr<PLQCD_F32, 18>(s, a, xpay, full, joined, deep);
        case PLQCD_F32 * 100 + 12: return dev::launch_ahead_pr<PLQCD_F32, 12>(s, a, xpay, full, joined, deep);
        case PLQCD_F16 * 100 + 12: return dev::launch_ahead_pr<PLQCD_F16, 12>(s, a, xpay, full, joined, deep);
        case PLQCD_BF16 * 100 + 12: return dev::launch_ahead_pr<PLQCD_BF16, 12>(s, a, xpay, full, joined, deep);
        default:
            return set_error(PLQCD_ERR_ARG, "dslash: unsupported precision/reconstruction %d/%d", prec, recon);
    }
}

}  // namespace plqcd
