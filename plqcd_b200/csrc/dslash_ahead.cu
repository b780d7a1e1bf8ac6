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
// What bounds it, and what it measured: us per launch on three sets of fields
// in turn, in short bursts at full clock / back to back for a second, where
// the power cap lowers the clock; before = the tuner's choice among cp.async,
// TMA and direct loads:
//   F32-18 xpay 32^3x64   146 / 160 -> 133 / 145   DRAM: 6.8 TB/s of its 864 bytes per site
//   F32-18 full 32^3x64   213 / 243 -> 182 / 215   DRAM and L2
//   F32-12 48^3x96        496 / 574 -> 483 / 561   DRAM: 6.3 / 5.5 TB/s
//   F16 xpay 32^3x64     85.7 / 96.6 -> 86.9 / 94.4   FMA pipes and latency
//   BF16 xpay 32^3x64    88.9 / 97.8 -> 84.1 / 90.6   the same
//   F64-18 xpay 24^3x48  92.0 / 102.6 -> 87.2 / 94.6   DRAM: 6.6 / 6.1 TB/s
//   F64-18 full 32^3x64   395 / 460 -> 390 / 456   latency at 8 warps
#include <cuda_runtime.h>

#include "blas.cuh"
#include "dslash_core.cuh"
#include "hop_sum.cuh"
#include "internal.h"
#include "pdl.cuh"
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

// Grids of at most this many blocks finish their sums in the last block to
// arrive, sparing a launch (2.5 us); above, its 64 threads would take longer
// over the partials than a kernel of one block of 1024 threads (4 us for the
// 16384 partials of 32^3x64).
constexpr long kSumInKernel = 512;

// block sums of (v, w) into the partials [block], [gridDim + block]; every
// thread of the block takes part
__device__ __forceinline__ void hop_sum_block(const SumArgs &q, double v, double w, bool two) {
    __shared__ double ws[2][2];
    __shared__ bool last;
    auto warp_sum = [](double t) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        return t;
    };
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    auto block_sum = [&](double t, double u) {
        t = warp_sum(t);
        if (two) u = warp_sum(u);
        __syncthreads();
        if (lane == 0) {
            ws[0][wp] = t;
            ws[1][wp] = u;
        }
        __syncthreads();
    };
    block_sum(v, w);
    CgState st;  // (no other block changes the state before every block has arrived)
    if (threadIdx.x == 0) {
        if (q.in_kernel) st = *q.red.state;
        q.red.partials[blockIdx.x] = ws[0][0] + ws[0][1];
        if (two) q.red.partials[gridDim.x + blockIdx.x] = ws[1][0] + ws[1][1];
        last = false;
        if (q.in_kernel) {
            __threadfence();
            last = atomicAdd(q.red.counter, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0, u = 0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
        t += __ldcg(q.red.partials + k);
        if (two) u += __ldcg(q.red.partials + gridDim.x + k);
    }
    block_sum(t, u);
    if (threadIdx.x == 0) {
        red_apply(q.op, ws[0][0] + ws[0][1], ws[1][0] + ws[1][1], st, q.red.state, q.report);
        *q.red.counter = 0;  // ready for the next sum on this scratch
    }
}

// the n partials (of one or two sums) in a fixed order, then the state update
__global__ void __launch_bounds__(1024) k_hop_sum_finish(RedScratch red, CgReport *report, int n, int two, RedOp op,
                                                         const int *halt) {
    __shared__ double ws[2][32];
    pdl_start();
    if (halt && *halt) return;
    CgState st;
    if (threadIdx.x == 0) st = *red.state;
    double t = 0, u = 0;
#pragma unroll 8
    for (int k = threadIdx.x; k < n; k += 1024) t += red.partials[k];
    if (two)
        for (int k = threadIdx.x; k < n; k += 1024) u += red.partials[n + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(0xffffffffu, t, o);
        u += __shfl_xor_sync(0xffffffffu, u, o);
    }
    if ((threadIdx.x & 31) == 0) {
        ws[0][threadIdx.x >> 5] = t;
        ws[1][threadIdx.x >> 5] = u;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    t = u = 0;
    for (int i = 0; i < 32; i++) {
        t += ws[0][i];
        u += ws[1][i];
    }
    red_apply(op, t, u, st, red.state, report);
}

// MODE 0: one parity; 1: with the xpay epilogue; 2: full lattice, the two
// parities of the same sites in neighbouring blocks; 3: full lattice, the
// two parities of 32 sites in one block (one warp each), sites in the 2x2x2
// tile order: the link a parity loads for its forward term is in L1 when
// the other one needs it for its backward term, and a tile's neighbour rows
// are loaded by blocks that run together (F64 at 32^3x64, long run: 429 us
// against 451 with the parities joined in the plain order; 4x2x2 430, 2x4x4
// 447, 4x4x4 453, 2x8x8 452, half of z x all of t 445). Modes 2 and 3 are a
// near-tie that the tuner decides: 3 took 429 against 462 us on one box, 463
// against 457 (short bursts 399 against 390) on another.
// SUM (mode 1, whole fields): a HopSumKind; OP: the format of its output.
// Threads past the last site compute on it and add nothing.
template <class SIO, class LIO, int MODE, int DEPTH, int MINB, int SUM = 0, int OP = PLQCD_F64>
__global__ void __launch_bounds__(kAheadBlock, MINB) k_dslash_ahead(const DslashArgs a, const SumArgs q) {
    using R = typename SIO::real;
    static_assert(SUM == 0 || MODE == 1, "sums belong to the xpay epilogue");
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
    const bool valid = h < a.h_end;
    if (!valid) {
        if (SUM == 0) {
            pdl_start();
            return;
        }
        h = a.h_end - 1;
    }
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
    pdl_start();
    if (a.halt && *a.halt) return;  // (an earlier kernel writes the flag: never read ahead of the wait)

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
    if constexpr (SUM == 0) {
        SIO::store(out, Vh, h, acc);
    } else {
        double v = 0, w = 0;
        if (valid) sum_epilogue<SIO, SUM, OP>(q, out, Vh, h, acc, v, w);
        hop_sum_block(q, v, w, SUM == HOP_CHECK);
    }
}

template <class SIO, class LIO, int MODE, int DEPTH, int MINB>
static int launch_ahead_t(cudaStream_t s, const DslashArgs &a) {
    const long per = MODE == 3 ? 32 : kAheadBlock;
    const long nblk = (a.h_end - a.h_begin + per - 1) / per * (MODE == 2 ? 2 : a.nrhs);
    if (nblk > 0x7fffffffL) return set_error(PLQCD_ERR_ARG, "dslash: grid too large");
    return launch_overlapped(k_dslash_ahead<SIO, LIO, MODE, DEPTH, MINB>, (unsigned)nblk, kAheadBlock, s, a, SumArgs{});
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
static int launch_sum_pr(cudaStream_t s, const DslashArgs &a, const SumArgs &q, unsigned nblk, const HopSum &h) {
    using S = SpinorIO<P>;
    using L = LinkIO<P, RC>;
    // Depth by format alone: in FP32 the two are within 2% in a solve from
    // 12^3x24 to 32^3x64 (depth 1 0.998 to 1.002 of depth 2 with 18-real
    // links, 8^3x16 1.03). In 16 bits depth 1 is the better one from 24^3x48
    // on (F16 solve at 32^3x64 12.87 ms against 13.06, BF16 52.7 against
    // 53.7), depth 2 below (F16 16^3x32 1.32 ms against 1.39, 8^3x16 0.76
    // against 0.77); the plain hops between these choose by the tuner.
    constexpr int D = P == PLQCD_F32 ? 2 : 1, B = P == PLQCD_F64 ? 4 : P == PLQCD_F32 ? 8 : 10;
    void (*k)(const DslashArgs, const SumArgs) = nullptr;
    if (h.kind == HOP_NORM) k = k_dslash_ahead<S, L, 1, D, B, HOP_NORM>;
    if (h.kind == HOP_UPDATE) k = k_dslash_ahead<S, L, 1, D, B, HOP_UPDATE>;
    if constexpr (P == PLQCD_F64) {
        if (h.kind == HOP_CHECK) k = k_dslash_ahead<S, L, 1, D, B, HOP_CHECK>;
        if (h.kind == HOP_RESID) switch (h.out_prec) {
                case PLQCD_F64: k = k_dslash_ahead<S, L, 1, D, B, HOP_RESID, PLQCD_F64>; break;
                case PLQCD_F32: k = k_dslash_ahead<S, L, 1, D, B, HOP_RESID, PLQCD_F32>; break;
                case PLQCD_F16: k = k_dslash_ahead<S, L, 1, D, B, HOP_RESID, PLQCD_F16>; break;
                case PLQCD_BF16: k = k_dslash_ahead<S, L, 1, D, B, HOP_RESID, PLQCD_BF16>; break;
            }
    }
    if (!k) return set_error(PLQCD_ERR_ARG, "hop with a sum: kind %d not available for precision %d", (int)h.kind, P);
    return launch_overlapped(k, nblk, kAheadBlock, s, a, q);
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

size_t hop_sum_partials(long Vh) { return 2 * (size_t)((Vh + dev::kAheadBlock - 1) / dev::kAheadBlock); }

int build_args(const Geom &g, const DslashCall &c, dev::DslashArgs &a);

int launch_hop_sum(const Geom &g, cudaStream_t s, const DslashCall &c, const HopSum &h, const RedScratch &r) {
    dev::DslashArgs a{};
    PLQCD_TRY(build_args(g, c, a));
    if (!c.x || c.full || c.nrhs != 1 || a.h_begin != 0 || a.h_end != g.Vh || (c.flags & PLQCD_DSLASH_COMPAT))
        return set_error(PLQCD_ERR_ARG, "hop with a sum: whole one-parity fields with an xpay operand only");
    if ((h.kind == HOP_UPDATE && !h.rvec) || ((h.kind == HOP_RESID || h.kind == HOP_CHECK) && !h.c))
        return set_error(PLQCD_ERR_ARG, "hop with a sum: operand missing");
    const long nblk = (g.Vh + dev::kAheadBlock - 1) / dev::kAheadBlock;
    const dev::SumArgs q{h.c, h.rvec, r, h.report, h.op, nblk <= dev::kSumInKernel};
    int rc;
    switch (c.prec * 100 + c.recon) {
        case PLQCD_F64 * 100 + 18: rc = dev::launch_sum_pr<PLQCD_F64, 18>(s, a, q, (unsigned)nblk, h); break;
        case PLQCD_F64 * 100 + 12: rc = dev::launch_sum_pr<PLQCD_F64, 12>(s, a, q, (unsigned)nblk, h); break;
        case PLQCD_F32 * 100 + 18: rc = dev::launch_sum_pr<PLQCD_F32, 18>(s, a, q, (unsigned)nblk, h); break;
        case PLQCD_F32 * 100 + 12: rc = dev::launch_sum_pr<PLQCD_F32, 12>(s, a, q, (unsigned)nblk, h); break;
        case PLQCD_F16 * 100 + 12: rc = dev::launch_sum_pr<PLQCD_F16, 12>(s, a, q, (unsigned)nblk, h); break;
        case PLQCD_BF16 * 100 + 12: rc = dev::launch_sum_pr<PLQCD_BF16, 12>(s, a, q, (unsigned)nblk, h); break;
        default:
            return set_error(PLQCD_ERR_ARG, "dslash: unsupported precision/reconstruction %d/%d", c.prec, c.recon);
    }
    if (rc == PLQCD_OK && !q.in_kernel)
        rc = launch_overlapped(dev::k_hop_sum_finish, 1, 1024, s, r, h.report, (int)nblk, h.kind == HOP_CHECK, h.op, c.halt);
    return rc;
}

}  // namespace plqcd
