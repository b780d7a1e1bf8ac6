// dslash.cu -- the Wilson hopping matrix on device fields (sm_100a).
//
// Gather form of the reference's four-pass hopping pair
// (lib/dirac.c:35-408 eo, 414-791 oe): one thread per output site reads its
// eight neighbours and the eight links directly, so the phip/phim buffers
// of the reference (include/plqcd_global_params.h:170-173) and their write /
// read-back traffic disappear. Per direction:
//   forward, neighbour x+mu:  chi  = U_mu(x)        h,  h  = upper((1 - g_mu) psi(x+mu))
//   backward, neighbour x-mu: chi' = U_mu(x-mu)^dag h', h' = upper((1 + g_mu) psi(x-mu))
// and the lower two spins are rebuilt from chi by the sign / i pattern of
// lib/dirac.c:269-311 (forward) and 371-398 (backward). The periodic wrap
// replaces the reference's MPI face exchange (lib/dirac.c:124-131, 203-228)
// for a lattice held by one GPU.
//
// Memory traffic is the bound (HBM roofline). Compulsory bytes per output
// site for one parity: input spinor once (neighbour re-reads hit L2), the 8
// links, the output spinor: 192 + 8*144 + 192 = 1536 B in FP64/18-real. The
// full-lattice kernel (FULL=true) produces both parities in one launch so
// each link, used by the forward term of x and the backward term of x+mu,
// is read from HBM once: 192 + 4*144 + 192 = 960 B per site.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "dslash_core.cuh"
#include "internal.h"
#include "tune.h"

namespace plqcd {

int launch_dslash_ahead(cudaStream_t s, const dev::DslashArgs &a, int prec, int recon, bool xpay, bool full,
                        bool joined, bool deep);
int build_args(const Geom &g, const DslashCall &c, dev::DslashArgs &a);

namespace dev {

// Direct loads at the use, for the reference's as-shipped results (COMPAT,
// FP64, one parity): a check, not a path whose speed matters. Everything
// else loads ahead (dslash_ahead.cu).
template <class SIO, class LIO>
__global__ void __launch_bounds__(256) k_dslash_compat(const DslashArgs a) {
    using R = typename SIO::real;
    const int par = a.out_parity;
    const long h = a.h_begin + (long)(blockIdx.x / a.nrhs) * blockDim.x + threadIdx.x;
    if (h >= a.h_end) return;
    const long roff = (long)(blockIdx.x % a.nrhs) * a.fbytes;  // RHS of this block
    const void *in = static_cast<const char *>(a.in[0]) + roff;
    void *out = static_cast<char *>(a.out[0]) + roff;
    const long Vh = a.Vh;
    const Coords c = site_coords(h, par, a.L0h, a.L1, a.L2);
    const int xh = (int)(h - c.row * a.L0h);
    int nb[8];
    neighbour_sites(c, xh, a.L0, a.L0h, a.L1, a.L2, a.L3, nb);

    const R sg = (R)a.g5_in;
    const int opp = par ^ 1;
    // as shipped, oe takes forward links of odd site h from the even site
    // with the same half index (lib/dirac.c:643)
    const int fpar = 0;

    cx<R> acc[12];
#pragma unroll
    for (int k = 0; k < 12; k++) acc[k] = {R(0), R(0)};
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int d = dir_at(k);
        cx<R> s[12], U[9];
        R n;
        SIO::load_raw(in, Vh, nb[d], s, n);
        if (d < 4)
            LIO::load(a.gauge, Vh, fpar, d, h, U);
        else
            LIO::load(a.gauge, Vh, opp, d - 4, nb[d], U);
        compute_dir_n<true, SIO::kScaled, R>(d, acc, s, U, sg, n);
    }
    const R aup = (R)a.a_up, alow = (R)a.a_low;
#pragma unroll
    for (int k = 0; k < 12; k++) {
        const R ak = k < 6 ? aup : alow;
        acc[k] = {ak * acc[k].re, ak * acc[k].im};
    }
    SIO::store(out, Vh, h, acc);
}

// Pipelined variant: the neighbour spinor and link of each of the 8
// directions are copied global->shared with cp.async, ST directions ahead of
// the one being computed, into slots private to the thread (no block-level
// synchronisation). The register file then only holds the direction being
// computed, while ST directions' loads are in flight per thread.
// Shared memory per block: ST * (spinor + link slots) * 16 bytes * blockDim.
template <class SIO, class LIO, int ST, bool COMPAT, bool XPAY, bool FULL>
__global__ void __launch_bounds__(256) k_dslash_pipe(const DslashArgs a) {
    using R = typename SIO::real;
    extern __shared__ uint4 smem[];
    constexpr int NS = SIO::NSLOT + LIO::NSLOT;
    const int B = blockDim.x;
    if (!COMPAT && !FULL && a.halt && *a.halt) return;
    int par;
    long h;
    if (FULL) {
        par = blockIdx.x & 1;
        h = (long)(blockIdx.x >> 1) * B + threadIdx.x;
    } else {
        par = a.out_parity;
        h = a.h_begin + (long)(blockIdx.x / a.nrhs) * B + threadIdx.x;
    }
    if (h >= a.h_end) return;  // no block-level barrier below
    const long roff = FULL ? 0 : (long)(blockIdx.x % a.nrhs) * a.fbytes;  // RHS of this block
    const void *in = (FULL && par == 0) ? a.in[1] : static_cast<const char *>(a.in[0]) + roff;
    void *out = (FULL && par == 1) ? a.out[1] : static_cast<char *>(a.out[0]) + roff;
    const long Vh = a.Vh;
    const int L0h = a.L0h, L1 = a.L1, L2 = a.L2, L3 = a.L3;
    const Coords c = site_coords(h, par, L0h, L1, L2);
    const int xh = (int)(h - c.row * L0h);
    int nb[8];
    neighbour_sites(c, xh, a.L0, L0h, L1, L2, L3, nb);
    const int opp = par ^ 1;
    const int fpar = (COMPAT && par == 1) ? 0 : par;

    const int stride = B * 16;  // bytes between consecutive slots of one thread
    const uint32_t s_thread = smem_addr(smem) + threadIdx.x * 16;
    // k-th direction of dir_at into slot k % ST
    auto issue = [&](int k) {
        const int d = dir_at(k);
        const uint32_t s0 = s_thread + (uint32_t)((k % ST) * NS) * stride;
        SIO::issue(in, Vh, nb[d], s0, stride);
        if (d < 4)
            LIO::issue(a.gauge, Vh, fpar, d, h, s0 + SIO::NSLOT * stride, stride);
        else
            LIO::issue(a.gauge, Vh, opp, d - 4, nb[d], s0 + SIO::NSLOT * stride, stride);
    };
#pragma unroll
    for (int k = 0; k < ST; k++) {
        issue(k);
        cp_async_commit();
    }
    cx<R> acc[12];
#pragma unroll
    for (int k = 0; k < 12; k++) acc[k] = {R(0), R(0)};
    const R sg = (R)a.g5_in;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        cp_async_wait<ST - 1>();
        const uint4 *s0 = smem + threadIdx.x + (k % ST) * NS * B;
        cx<R> s[12], U[9];
        R n;
        SIO::load_staged_raw(s0, B, s, n);
        LIO::load_staged(s0 + SIO::NSLOT * B, B, U);
        compute_dir_n<COMPAT, SIO::kScaled, R, true>(dir_at(k), acc, s, U, sg, n);
        // the slot just consumed is refilled only after its values were used
        if (k + ST < 8) issue(k + ST);
        cp_async_commit();
    }

    const R aup = (R)a.a_up, alow = (R)a.a_low;
    if (XPAY) {
        cx<R> xv[12];
        SIO::load(static_cast<const char *>(a.x) + roff, Vh, h, xv);
        const R b = (R)a.b;
#pragma unroll
        for (int k = 0; k < 12; k++) {
            const R ak = k < 6 ? aup : alow;
            acc[k] = {fma(ak, acc[k].re, b * xv[k].re), fma(ak, acc[k].im, b * xv[k].im)};
        }
    } else {
#pragma unroll
        for (int k = 6; k < 12; k++) acc[k] = {alow * acc[k].re, alow * acc[k].im};
#pragma unroll
        for (int k = 0; k < 6; k++) acc[k] = {aup * acc[k].re, aup * acc[k].im};
    }
    SIO::store(out, Vh, h, acc);
}

template <class SIO, class LIO, int ST, bool COMPAT, bool XPAY, bool FULL>
static int launch_pipe(const Geom &g, cudaStream_t s, const DslashArgs &a, int block) {
    long nblk = (a.h_end - a.h_begin + block - 1) / block * a.nrhs;
    if (FULL) nblk *= 2;
    constexpr int NS = SIO::NSLOT + LIO::NSLOT;
    const size_t smem = (size_t)ST * NS * 16 * block;
    auto k = k_dslash_pipe<SIO, LIO, ST, COMPAT, XPAY, FULL>;
    PLQCD_TRY(smem_optin((const void *)k, 227 * 1024));
    if (smem > 227 * 1024) return set_error(PLQCD_ERR_ARG, "dslash: %zu bytes of shared memory requested", smem);
    k<<<(unsigned)nblk, block, smem, s>>>(a);
    PLQCD_CUDA_TRY(cudaGetLastError());
    return PLQCD_OK;
}

// variant 2, 3: cp.async pipeline of that depth; anything else: loads ahead
// in registers (0 and 21 of dslash_ahead.cu; tuning files may still hold 12
// and 13, kernels of two sites per thread that it replaced where they existed)
template <class SIO, class LIO, bool COMPAT, bool XPAY, bool FULL>
static int launch_t(const Geom &g, cudaStream_t s, const DslashArgs &a, int prec, int recon, int variant, int block) {
    if (variant == 2) return launch_pipe<SIO, LIO, 2, COMPAT, XPAY, FULL>(g, s, a, block);
    if (variant == 3) return launch_pipe<SIO, LIO, 3, COMPAT, XPAY, FULL>(g, s, a, block);
    if ((variant == 12 || variant == 13) && (COMPAT || FULL || std::is_same<typename SIO::real, double>::value))
        return set_error(PLQCD_ERR_ARG, "dslash: two sites per thread exists for 32/16-bit single-parity calls");
    if constexpr (COMPAT) {
        const long nblk = (a.h_end - a.h_begin + block - 1) / block * a.nrhs;
        k_dslash_compat<SIO, LIO><<<(unsigned)nblk, block, 0, s>>>(a);
        PLQCD_CUDA_TRY(cudaGetLastError());
        return PLQCD_OK;
    } else {
        return launch_dslash_ahead(s, a, prec, recon, XPAY, FULL, variant == 21, block == 128);
    }
}

template <int PREC, int RECON>
static int launch_pr(const Geom &g, cudaStream_t s, const DslashArgs &a, int variant, int block, bool compat,
                     bool xpay, bool full) {
    using S = SpinorIO<PREC>;
    using L = LinkIO<PREC, RECON>;
    if (full) return launch_t<S, L, false, false, true>(g, s, a, PREC, RECON, variant, block);
    if (compat) {
        if (PREC == PLQCD_F64 && RECON == 18) return launch_t<S, L, true, false, false>(g, s, a, PREC, RECON, variant, block);
        return set_error(PLQCD_ERR_ARG, "dslash: the bug-compatible mode exists for F64 18-real links only");
    }
    if (xpay) return launch_t<S, L, false, true, false>(g, s, a, PREC, RECON, variant, block);
    return launch_t<S, L, false, false, false>(g, s, a, PREC, RECON, variant, block);
}

}  // namespace dev

int launch_dslash_tma(const Geom &g, cudaStream_t s, const dev::DslashArgs &a, int prec, int recon, bool full,
                      bool xpay, int kind, int nstage, int ny);

static int env_int(const char *name, int dflt) {
    const char *e = getenv(name);
    return (e && *e) ? atoi(e) : dflt;  // unset or empty: the default
}

static int dispatch(const Geom &g, cudaStream_t s, const DslashCall &c, const dev::DslashArgs &a, int variant,
                    int block);

static int tune_dslash(const Geom &g, cudaStream_t s, const DslashCall &c, const dev::DslashArgs &a,
                       const char *key);

// one launch with an explicit configuration (no tuning)
int launch_dslash_config(const Geom &g, cudaStream_t s, const DslashCall &c, int variant, int block) {
    dev::DslashArgs a{};
    PLQCD_TRY(build_args(g, c, a));
    return dispatch(g, s, c, a, variant, block);
}

int launch_dslash(const Geom &g, cudaStream_t s, const DslashCall &c) {
    dev::DslashArgs a{};
    PLQCD_TRY(build_args(g, c, a));
    const bool compat = (c.flags & PLQCD_DSLASH_COMPAT) != 0;

    // explicit configuration (block from the call, or the environment for
    // experiments) bypasses the tuner
    int env_block = env_int("PLQCD_DSLASH_BLOCK", 0), env_var = env_int("PLQCD_DSLASH_STAGES", -1);
    // PLQCD_DSLASH_FULL_STAGES: the variant of full-lattice F64 calls only
    if (c.full && c.prec == PLQCD_F64 && env_int("PLQCD_DSLASH_FULL_STAGES", -1) >= 0) {
        env_var = env_int("PLQCD_DSLASH_FULL_STAGES", -1);
        if (env_block <= 0) env_block = 64;
    }
    if (c.block > 0 || env_block > 0 || env_var >= 0) {
        int block = c.block > 0 ? c.block : (env_block > 0 ? env_block : 128);
        return dispatch(g, s, c, a, env_var >= 0 ? env_var : 2, block);
    }
    // a partial site range (the drop-in path's t-slab chunks) is a separate
    // entry: its best kernel need not be that of whole fields
    const bool part = a.h_begin != 0 || a.h_end != g.Vh;
    const TuneId id = tune_id(kTuneDslash, c.prec, c.recon, c.full | (c.x ? 2 : 0) | (compat ? 4 : 0) | (part ? 8 : 0),
                              c.nrhs, g.L);
    TuneResult known;
    if (tune_recall(id, &known)) return dispatch(g, s, c, a, known.variant, known.block);
    char key[256];
    snprintf(key, sizeof key, "%sdslash|p%d|r%d|%s%s%s%s|%dx%dx%dx%d|n%d%s", device_tag().c_str(), c.prec, c.recon,
             c.full ? "full" : "half", c.x ? "+xpay" : "", compat ? "+compat" : "", part ? "+range" : "", g.L[0],
             g.L[1], g.L[2], g.L[3], c.nrhs, kTuneListTag);
    const int rc = tune_dslash(g, s, c, a, key);
    tune_remember(id, key);
    return rc;
}

int build_args(const Geom &g, const DslashCall &c, dev::DslashArgs &a) {
    PLQCD_TRY(check_field_ptr(c.out, "dslash"));
    PLQCD_TRY(check_field_ptr(c.in, "dslash"));
    if (c.full) {
        PLQCD_TRY(check_field_ptr(c.out2, "dslash_full"));
        PLQCD_TRY(check_field_ptr(c.in2, "dslash_full"));
    }
    if (c.x) PLQCD_TRY(check_field_ptr(c.x, "dslash_xpay"));
    a.gauge = c.gauge;
    if (c.nrhs < 1 || (c.full && c.nrhs != 1)) return set_error(PLQCD_ERR_ARG, "dslash: nrhs = %d invalid", c.nrhs);
    a.nrhs = c.nrhs;
    a.fbytes = (long)spinor_parity_bytes(g.Vh, c.prec);
    if (c.full) {
        a.in[0] = c.in;
        a.in[1] = c.in2;
        a.out[0] = c.out;
        a.out[1] = c.out2;
    } else {
        a.in[0] = c.in;
        a.out[0] = c.out;
    }
    a.x = c.x;
    a.halt = c.halt;
    a.Vh = g.Vh;
    a.h_begin = c.h_begin;
    a.h_end = c.h_count < 0 ? g.Vh : c.h_begin + c.h_count;
    if (a.h_begin < 0 || a.h_end > g.Vh || a.h_end <= a.h_begin || (c.full && (a.h_begin != 0 || a.h_end != g.Vh)))
        return set_error(PLQCD_ERR_ARG, "dslash: site range [%ld, %ld) invalid", a.h_begin, a.h_end);
    a.L0 = g.L[0];
    a.L0h = g.L0h;
    a.L1 = g.L[1];
    a.L2 = g.L[2];
    a.L3 = g.L[3];
    a.out_parity = c.out_parity;
    a.a_up = c.a_up;
    a.a_low = (c.flags & PLQCD_DSLASH_G5_OUT) ? -c.a_low : c.a_low;
    a.b = c.b;
    a.g5_in = (c.flags & PLQCD_DSLASH_G5_IN) ? -1.0 : 1.0;
    const bool compat = (c.flags & PLQCD_DSLASH_COMPAT) != 0;
    if (c.full && (compat || c.x || (c.flags & (PLQCD_DSLASH_G5_IN | PLQCD_DSLASH_G5_OUT))))
        return set_error(PLQCD_ERR_ARG, "dslash_full: flags and xpay are not supported in full-lattice mode");
    return PLQCD_OK;
}

static int tune_dslash(const Geom &g, cudaStream_t s, const DslashCall &c, const dev::DslashArgs &a,
                       const char *key) {
    // loads ahead in registers (0: a block of 64 stands for depth 1, one of
    // 128 for depth 2; 21: joined parities), cp.async pipeline depth (2, 3) x
    // block size. The first one runs where tuning is not possible.
    std::vector<TuneResult> cands;
    const bool compat = (c.flags & PLQCD_DSLASH_COMPAT) != 0;
    auto add = [&](int variant, int block) {
        TuneResult r;
        r.variant = variant;
        r.block = block;
        cands.push_back(r);
    };
    if (compat) {
        // (larger blocks too: 256 threads at 16^3x32 17.6 us, 64 threads 18.7)
        for (int v : {2, 0, 3})
            for (int b : {64, 128, 256}) add(v, b);
    } else {
        if (c.full && c.prec == PLQCD_F64) add(21, 64);
        if (c.prec != PLQCD_F64) add(0, 128);
        add(0, 64);
        for (int v : {2, 3})
            for (int b : {64, 128, 256}) add(v, b);
    }
    // TMA-staged rows: ring depth x rows per tile, where the tile fits, for
    // the FP64 full lattice. (With loads ahead in registers the other forms
    // lose at every measured size, e.g. F64 xpay at 32^3x64 295 us against
    // 270, F32-18 full lattice 296 against 180; a near-tie is left at 16^3x32,
    // 32.5 against 32.8. They run when the environment or an older tuning
    // file names them.)
    if (c.full && c.prec == PLQCD_F64 && getenv("PLQCD_NO_TMA") == nullptr)
        // (kinds 3 and 5, two own-line buffers, lost to 2 and 4 at every
        // measured point and are not tried). The own-line kernels (4, 2)
        // come first, so they keep a near-tie: they stage fewer bytes per
        // site and hold a higher rate once the power cap settles the clock
        // (FP64 full lattice at 32^3x64, 4 s back to back: 4304 0.666 of
        // HBM against 0.651 for 1204, at 1515 / 1470 MHz)
        for (int kind : {4, 2, 1})
            for (int ny : {4, 8, 16, 2})
                for (int ns : {1, 2, 3, 4, 6}) {
                    if (kind == 2 ? ns == 6 : ns == 1) continue;
                    int blk = 0;
                    if (dslash_tma_plan(g, c.prec, c.recon, kind, ns, ny, &blk, nullptr) != PLQCD_OK) {
                        clear_error();
                        continue;
                    }
                    add(1000 * kind + 100 * ns + ny, blk);
                }
    // trial launches write into scratch outputs: an xpay whose output aliases
    // its x operand must not be applied more than once
    void *scratch[2] = {nullptr, nullptr};
    std::vector<int> tma_checked;
    auto run = [&](const TuneResult &r, bool trial) -> int {
        if (!trial) return dispatch(g, s, c, a, r.variant, r.block);
        if (r.variant >= 1000 && std::find(tma_checked.begin(), tma_checked.end(), r.variant) == tma_checked.end()) {
            // first trial of a TMA configuration: run it alone and check that
            // no stage wait ran out before it is timed
            tma_checked.push_back(r.variant);
            dev::DslashArgs t = a;
            size_t bytes = spinor_parity_bytes(g.Vh, c.prec);
            for (int k = 0; k < (c.full ? 2 : 1); k++)
                if (!scratch[k] && cudaMalloc(&scratch[k], bytes) != cudaSuccess) {
                    cudaGetLastError();
                    return set_error(PLQCD_ERR_NOMEM, "tune: scratch allocation failed");
                }
            t.out[0] = scratch[0];
            if (c.full) t.out[1] = scratch[1];
            t.halt = nullptr;
            PLQCD_TRY(dispatch(g, s, c, t, r.variant, r.block));
            PLQCD_CUDA_TRY(cudaStreamSynchronize(s));
            if (dslash_tma_status(true)) return set_error(PLQCD_ERR_CUDA, "dslash: TMA stage wait timed out");
        }
        size_t bytes = spinor_parity_bytes(g.Vh, c.prec) * c.nrhs;
        for (int k = 0; k < (c.full ? 2 : 1); k++)
            if (!scratch[k] && cudaMalloc(&scratch[k], bytes) != cudaSuccess) {
                cudaGetLastError();
                return set_error(PLQCD_ERR_NOMEM, "tune: scratch allocation failed");
            }
        dev::DslashArgs t = a;
        t.out[0] = scratch[0];
        if (c.full) t.out[1] = scratch[1];
        t.halt = nullptr;
        return dispatch(g, s, c, t, r.variant, r.block);
    };
    int rc = tune_launch(key, s, cands, run);
    for (void *p : scratch)
        if (p) {
            cudaStreamSynchronize(s);
            cudaFree(p);
        }
    return rc;
}

static int dispatch(const Geom &g, cudaStream_t s, const DslashCall &c, const dev::DslashArgs &a, int variant,
                    int block) {
    const bool compat = (c.flags & PLQCD_DSLASH_COMPAT) != 0;
    const bool xpay = c.x != nullptr;
    if (variant >= 1000) {  // TMA-staged rows; the block follows from the tile
        if (compat) return set_error(PLQCD_ERR_ARG, "dslash: no bug-compatible TMA kernel");
        return launch_dslash_tma(g, s, a, c.prec, c.recon, c.full, xpay, variant / 1000, (variant / 100) % 10,
                                 variant % 100);
    }
    if (block % 32 || block < 32 || block > 256) return set_error(PLQCD_ERR_ARG, "dslash: block size %d invalid", block);
    switch (c.prec * 100 + c.recon) {
        case PLQCD_F64 * 100 + 18: return dev::launch_pr<PLQCD_F64, 18>(g, s, a, variant, block, compat, xpay, c.full);
        case PLQCD_F64 * 100 + 12: return dev::launch_pr<PLQCD_F64, 12>(g, s, a, variant, block, compat, xpay, c.full);
        case PLQCD_F32 * 100 + 18: return dev::launch_pr<PLQCD_F32, 18>(g, s, a, variant, block, compat, xpay, c.full);
        case PLQCD_F32 * 100 + 12: return dev::launch_pr<PLQCD_F32, 12>(g, s, a, variant, block, compat, xpay, c.full);
        case PLQCD_F16 * 100 + 12: return dev::launch_pr<PLQCD_F16, 12>(g, s, a, variant, block, compat, xpay, c.full);
        case PLQCD_BF16 * 100 + 12: return dev::launch_pr<PLQCD_BF16, 12>(g, s, a, variant, block, compat, xpay, c.full);
        default:
            return set_error(PLQCD_ERR_ARG, "dslash: unsupported precision/reconstruction %d/%d", c.prec, c.recon);
    }
}

}  // namespace plqcd
