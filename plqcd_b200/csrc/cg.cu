// cg.cu -- even/odd preconditioned CG for the Wilson operator, FP64 and
// mixed precision with reliable updates.
//
// The reference stops at the hopping matrix (its operator and solver
// parameters are placeholders, include/plqcd_global_params.h:197-201); this
// solver builds on the same operator:
//   D = 1 - kappa H,   D [x_e; x_o] = [b_e; b_o]
//   Mhat = 1 - kappa^2 H_eo H_oe   (Schur complement on even sites)
//   b'   = b_e + kappa H_eo b_o,   Mhat x_e = b',   x_o = b_o + kappa H_oe x_e
// CG runs on the normal equations Mhat^dag Mhat x_e = Mhat^dag b' with
// Mhat^dag = g5 Mhat g5 (gamma5 folded into the hopping kernels).
//
// Mixed precision (Clark et al., "Solving Lattice QCD systems of equations
// using mixed precision solvers on GPUs", 2010): the recursion runs with a
// sloppy operator and sloppy vectors; whenever |r_sloppy| has dropped by
// `delta` since the last update, or looks converged, a reliable update adds
// the sloppy solution into the FP64 solution and recomputes the true
// residual with the FP64 operator (defect correction). Convergence is
// declared on the FP64 Schur residual |b' - Mhat x| / |b'| only; the final
// full-lattice residual |b - D x| / |b| is reported as well. All
// reductions accumulate in FP64 on the device and finalise alpha / beta
// there; the host reads one small state block per iteration to steer.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "blas.cuh"
#include "internal.h"

using namespace plqcd;

namespace plqcd {

int lattice_workspace(plqcd_lattice *lat, size_t bytes, void **out) {
    if (lat->ws_bytes < bytes) {
        if (lat->ws) {
            cudaStreamSynchronize(lat->stream);
            cudaFree(lat->ws);
            lat->ws = nullptr;
            lat->ws_bytes = 0;
        }
        if (cudaMalloc(&lat->ws, bytes) != cudaSuccess) {
            cudaGetLastError();
            return set_error(PLQCD_ERR_NOMEM, "solver workspace of %zu bytes", bytes);
        }
        lat->ws_bytes = bytes;
    }
    *out = lat->ws;
    return PLQCD_OK;
}

int lattice_staging(plqcd_lattice *lat, size_t bytes, void **out) {
    if (bytes > kStagingBytes) return set_error(PLQCD_ERR_ARG, "staging of %zu bytes", bytes);
    if (lat->staging_bytes < bytes) {
        if (lat->staging) {
            cudaStreamSynchronize(lat->stream);
            cudaFree(lat->staging);
            lat->staging = nullptr;
            lat->staging_bytes = 0;
        }
        if (cudaMalloc(&lat->staging, bytes) != cudaSuccess) {
            cudaGetLastError();
            return set_error(PLQCD_ERR_NOMEM, "staging of %zu bytes", bytes);
        }
        lat->staging_bytes = bytes;
    }
    *out = lat->staging;
    return PLQCD_OK;
}

int lattice_host_block(plqcd_lattice *lat, void **out) {
    if (!lat->host_block && cudaHostAlloc(&lat->host_block, kHostBlockBytes, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        lat->host_block = nullptr;
        return set_error(PLQCD_ERR_NOMEM, "page-locked block of %zu bytes", kHostBlockBytes);
    }
    *out = lat->host_block;
    return PLQCD_OK;
}

}  // namespace plqcd

namespace {

struct Op {
    const Geom &g;
    cudaStream_t s;
    double kappa;
    const RedScratch &red;
    static DslashCall call(const plqcd_gauge *gf, void *out, const void *in, int out_parity, unsigned flags,
                           const void *x, double a, double b, const int *halt) {
        DslashCall c;
        c.gauge = gf->data;
        c.prec = gf->prec;
        c.recon = gf->recon;
        c.out = out;
        c.in = in;
        c.out_parity = out_parity;
        c.flags = flags;
        c.x = x;
        c.a_up = c.a_low = a;
        c.b = b;
        c.halt = halt;
        return c;
    }
    // out_parity-specific hopping with epilogue
    int hop(const plqcd_gauge *gf, void *out, const void *in, int out_parity, unsigned flags, const void *x = nullptr,
            double a = 1.0, double b = 0.0, const int *halt = nullptr) const {
        return launch_dslash(g, s, call(gf, out, in, out_parity, flags, x, a, b, halt));
    }
    // out = Mhat in (dagger: g5 Mhat g5 in); tmp_o: odd scratch
    int mhat(const plqcd_gauge *gf, void *out, const void *in, void *tmp_o, bool dagger) const {
        unsigned fin = dagger ? PLQCD_DSLASH_G5_IN : 0u, fout = dagger ? PLQCD_DSLASH_G5_OUT : 0u;
        PLQCD_TRY(hop(gf, tmp_o, in, PLQCD_ODD, fin));
        return hop(gf, out, tmp_o, PLQCD_EVEN, fout, in, -kappa * kappa, 1.0);
    }
    // the same with the sum h in the second hop's epilogue
    int mhat_sum(const plqcd_gauge *gf, void *out, const void *in, void *tmp_o, bool dagger, const HopSum &h,
                 const int *halt = nullptr) const {
        unsigned fin = dagger ? PLQCD_DSLASH_G5_IN : 0u, fout = dagger ? PLQCD_DSLASH_G5_OUT : 0u;
        PLQCD_TRY(hop(gf, tmp_o, in, PLQCD_ODD, fin, nullptr, 1.0, 0.0, halt));
        return launch_hop_sum(g, s, call(gf, out, tmp_o, PLQCD_EVEN, fout, in, -kappa * kappa, 1.0, halt), h, red);
    }
};

HopSum sum_of(HopSumKind kind, RedOp op, const void *c = nullptr, void *rvec = nullptr, int out_prec = PLQCD_F64,
              CgReport *report = nullptr) {
    HopSum h;
    h.report = report;
    h.kind = kind;
    h.op = op;
    h.c = c;
    h.rvec = rvec;
    h.out_prec = out_prec;
    return h;
}

}  // namespace

extern "C" void plqcd_cg_param_default(plqcd_cg_param *p) {
    if (!p) return;
    memset(p, 0, sizeof *p);
    p->kappa = 0.12;
    p->tol = 1e-10;
    p->max_iter = 10000;
    p->sloppy_prec = PLQCD_F64;
    p->delta = 0.01;
    p->verbose = 0;
}

extern "C" int plqcd_invert_cg(plqcd_lattice *lat, const plqcd_gauge *g64, const plqcd_gauge *gs, void *x_even,
                               void *x_odd, const void *b_even, const void *b_odd, const plqcd_cg_param *prm,
                               plqcd_cg_info *info) {
    clear_error();
    if (!lat || !g64 || !x_even || !x_odd || !b_even || !b_odd || !prm)
        return set_error(PLQCD_ERR_ARG, "plqcd_invert_cg: null argument");
    if (!gs) gs = g64;
    PLQCD_CUDA_TRY(cudaSetDevice(lat->device));
    if (g64->prec != PLQCD_F64) return set_error(PLQCD_ERR_ARG, "plqcd_invert_cg: the reliable gauge field must be F64");
    if (gs->prec != prm->sloppy_prec)
        return set_error(PLQCD_ERR_ARG, "plqcd_invert_cg: sloppy gauge precision %d != sloppy_prec %d", gs->prec,
                         prm->sloppy_prec);
    if (g64->lat->geom.Vh != lat->geom.Vh || gs->lat->geom.Vh != lat->geom.Vh)
        return set_error(PLQCD_ERR_ARG, "plqcd_invert_cg: gauge fields belong to another lattice");
    if (!(prm->tol > 0) || prm->max_iter <= 0) return set_error(PLQCD_ERR_ARG, "plqcd_invert_cg: bad tol / max_iter");

    const Geom &g = lat->geom;
    cudaStream_t s = lat->stream;
    const int ps = prm->sloppy_prec;
    const int xprec = (ps == PLQCD_F64) ? PLQCD_F64 : PLQCD_F32;
    const size_t b64 = spinor_parity_bytes(g.Vh, PLQCD_F64);
    const size_t bs = spinor_parity_bytes(g.Vh, ps);
    const size_t bx = spinor_parity_bytes(g.Vh, xprec);
    auto al = [](size_t n) { return (n + 255) & ~(size_t)255; };
    const size_t need = 3 * al(b64) + 5 * al(bs) + al(bx) + al(red_scratch_bytes(g.Vh));
    void *ws = nullptr;
    PLQCD_TRY(lattice_workspace(lat, need, &ws));
    char *w = static_cast<char *>(ws);
    auto take = [&](size_t n) {
        void *p = w;
        w += al(n);
        return p;
    };
    void *bprime = take(b64), *t64 = take(b64), *tmp64 = take(b64);
    void *rs = take(bs), *p = take(bs), *Ap = take(bs), *t = take(bs), *tmps = take(bs);
    void *xs = take(bx);
    void *redmem = take(red_scratch_bytes(g.Vh));
    PLQCD_CUDA_TRY(cudaMemsetAsync(redmem, 0, red_scratch_bytes(g.Vh), s));
    RedScratch red = red_scratch_from(redmem, g.Vh);
    // page-locked: the state as last read, its start values, and one report
    // per iteration in flight
    void *hblock = nullptr;
    PLQCD_TRY(lattice_host_block(lat, &hblock));
    static_assert(2 * sizeof(CgState) + 2 * sizeof(CgReport) <= kHostBlockBytes, "solver states");
    CgState *hst = static_cast<CgState *>(hblock);
    CgReport *report = reinterpret_cast<CgReport *>(hst + 2);
    auto read_state = [&]() -> int {
        PLQCD_CUDA_TRY(cudaMemcpyAsync(hst, red.state, sizeof(CgState), cudaMemcpyDeviceToHost, s));
        PLQCD_CUDA_TRY(cudaStreamSynchronize(s));
        return PLQCD_OK;
    };

    Op op{g, s, prm->kappa, red};
    cudaEvent_t e0 = lat->ev0, e1 = lat->ev1;
    for (cudaEvent_t &ev : lat->iter_event)
        if (!ev) PLQCD_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    cudaEventRecord(e0, s);
    int rc = PLQCD_OK;
    plqcd_cg_info inf;
    memset(&inf, 0, sizeof inf);
    double bp2 = 0, sr2 = 0;
    bool end_recorded = false;  // device time covers the solve, not the verification

    do {
        const bool mixed = ps != PLQCD_F64;
        CgState *init = hst + 1;
        memset(init, 0, sizeof *init);
        init->target = prm->tol * prm->tol;  // RED_RR_INIT makes it tol^2 |rhs|^2
        init->delta2 = prm->delta * prm->delta;
        init->mixed = mixed;
        // a sloppy recursion that stops reducing its residual (16-bit storage
        // with a tiny delta) would never trigger an update: force one after
        // this many iterations without
        init->max_run = 100;
        if (cudaMemcpyAsync(red.state, init, sizeof *init, cudaMemcpyHostToDevice, s) != cudaSuccess) {
            rc = set_error(PLQCD_ERR_CUDA, "plqcd_invert_cg: state upload failed");
            break;
        }
        // b' = b_e + kappa H_eo b_o ; r = p = rhs = Mhat^dag b'
        if ((rc = launch_hop_sum(g, s, Op::call(g64, bprime, b_odd, PLQCD_EVEN, 0, b_even, prm->kappa, 1.0, nullptr),
                                 sum_of(HOP_NORM, RED_AUX), red)))
            break;
        const HopSum rhs_sum = sum_of(HOP_NORM, RED_RR_INIT);
        if (mixed) {
            // the sloppy recursion starts from rhs in sloppy precision, so
            // the sloppy operator computes it; convergence is decided on the
            // FP64 Schur residual of b', which does not use rhs
            if ((rc = launch_spinor_convert(g, s, t, ps, bprime, PLQCD_F64))) break;
            if ((rc = op.mhat_sum(gs, rs, t, tmps, true, rhs_sum))) break;
            inf.sloppy_hops += 2;
        } else if ((rc = op.mhat_sum(g64, rs, bprime, tmp64, true, rhs_sum))) {
            break;
        }
        if (cudaMemcpyAsync(p, rs, bs, cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
            rc = set_error(PLQCD_ERR_CUDA, "plqcd_invert_cg: device copy failed");
            break;
        }
        cudaMemsetAsync(x_even, 0, b64, s);
        if ((rc = read_state())) break;
        bp2 = hst->aux;
        if (!(bp2 > 0)) {  // zero source: zero solution
            rc = op.hop(g64, x_odd, x_even, PLQCD_ODD, 0, b_odd, prm->kappa, 1.0);
            inf.sloppy_hops = 0;
            inf.converged = 1;
            break;
        }

        // One iteration, all of it queued at once: Ap = Mhat^dag Mhat p with
        // |t|^2 = |Mhat p|^2 and r -= alpha Ap, |r|^2 in the hops' epilogues,
        // then x_s += alpha p, p = r + beta p. The |r|^2 sum decides whether
        // a reliable update is due; then the p step, and every kernel of the
        // iteration queued after, does nothing. So the host queues iteration
        // it + 1 before it reads what iteration `it` came to, and the device
        // does not wait for it. The outcome reaches the host as a store of the
        // summing kernel to page-locked memory: a copy between the kernels
        // held up the stream for 5 us.
        // The sloppy solution x_s is not cleared: while `fresh` it counts as
        // zero, and its next update writes it unread.
        const int *halt = &red.state->halt;
        auto queue = [&](int it, bool fresh) -> int {
            PLQCD_TRY(op.mhat_sum(gs, t, p, tmps, false, sum_of(HOP_NORM, RED_ALPHA), halt));
            PLQCD_TRY(op.mhat_sum(gs, Ap, t, tmps, true,
                                  sum_of(HOP_UPDATE, RED_RR, nullptr, rs, ps, &report[it & 1]), halt));
            PLQCD_CUDA_TRY(cudaEventRecord(lat->iter_event[it & 1], s));
            return blas_cg_p_x(g, s, p, rs, ps, xs, xprec, fresh ? 1 : 2, red);
        };
        bool fresh = true;  // before the iteration whose outcome is read next
        if ((rc = queue(1, fresh))) break;
        for (int it = 1; it <= prm->max_iter; it++) {
            if (it < prm->max_iter && (rc = queue(it + 1, false))) break;
            const cudaError_t e = cudaEventSynchronize(lat->iter_event[it & 1]);
            if (e != cudaSuccess) {
                rc = set_error(PLQCD_ERR_CUDA, "plqcd_invert_cg: %s", cudaGetErrorString(e));
                break;
            }
            const CgReport now = report[it & 1];
            inf.sloppy_hops += 4;
            inf.iterations = it;
            if (!std::isfinite(now.rr)) {
                rc = set_error(PLQCD_ERR_NOCONV, "plqcd_invert_cg: residual is not finite at iteration %d", it);
                break;
            }
            if (!now.halt) {
                fresh = false;
                continue;
            }
            // reliable update, defect correction: x += x_s + alpha p, then
            // the Schur residual b' - Mhat x in FP64, stored in the sloppy
            // format (the restart needs nothing more)
            if ((rc = blas_accum(g, s, x_even, xs, xprec, fresh, p, ps, red))) break;
            fresh = true;
            if ((rc = op.mhat_sum(g64, t, x_even, tmp64, false, sum_of(HOP_RESID, RED_SR2, bprime, nullptr, ps)))) break;
            inf.f64_hops += 2;
            inf.reliable_updates++;
            if ((rc = read_state())) break;
            sr2 = hst->sr2;
            if (prm->verbose)
                fprintf(stderr, "plqcd cg: it %d reliable update, |r_schur|/|b'| = %.3e\n", it, sqrt(sr2 / bp2));
            if (sr2 <= prm->tol * prm->tol * bp2) {
                inf.converged = 1;
                break;
            }
            // restart the recursion from r = Mhat^dag (b' - Mhat x). The FP64
            // residual above decides convergence; the restart direction only
            // needs the sloppy operator's accuracy
            if ((rc = op.mhat_sum(mixed ? gs : g64, rs, t, tmps, true, sum_of(HOP_NORM, RED_RR_TRUE)))) break;
            (mixed ? inf.sloppy_hops : inf.f64_hops) += 2;
            if ((rc = blas_cg_p_x(g, s, p, rs, ps, xs, xprec, 0, red))) break;
            if (it < prm->max_iter && (rc = queue(it + 1, fresh))) break;
        }
        if (rc) break;
        if (!inf.converged) {
            // fold in what the sloppy recursion has so far
            if ((rc = blas_accum(g, s, x_even, xs, xprec, fresh, nullptr, ps, red))) break;
        }
        // x_o = b_o + kappa H_oe x_e
        if ((rc = op.hop(g64, x_odd, x_even, PLQCD_ODD, 0, b_odd, prm->kappa, 1.0))) break;
        // the solve ends here; what follows is the verification
        cudaEventRecord(e1, s);
        end_recorded = true;
        // full-lattice residual |b - D x| / |b|, D x = x - kappa H x
        if ((rc = launch_hop_sum(g, s, Op::call(g64, t64, x_odd, PLQCD_EVEN, 0, x_even, -prm->kappa, 1.0, nullptr),
                                 sum_of(HOP_CHECK, RED_CHECK_E, b_even), red)))
            break;
        if ((rc = launch_hop_sum(g, s, Op::call(g64, t64, x_even, PLQCD_ODD, 0, x_odd, -prm->kappa, 1.0, nullptr),
                                 sum_of(HOP_CHECK, RED_CHECK_O, b_odd), red)))
            break;
        if ((rc = read_state())) break;
        inf.true_residual = sqrt((hst->check[0] + hst->check[2]) / (hst->check[1] + hst->check[3]));
        inf.schur_residual = sqrt(sr2 / bp2);
    } while (0);

    if (!end_recorded) cudaEventRecord(e1, s);
    // nothing queued is left behind: an iteration queued ahead still reads x
    // and writes the page-locked reports
    cudaStreamSynchronize(s);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    inf.seconds = ms / 1e3;
    // a hop whose staged loads never arrived leaves a flag, not a CUDA error
    if (!rc && dslash_tma_status(true))
        rc = set_error(PLQCD_ERR_TIMEOUT, "plqcd_invert_cg: a TMA stage wait of a hop ran out");
    if (info) *info = inf;
    if (rc) return rc;
    if (!inf.converged)
        return set_error(PLQCD_ERR_NOCONV, "plqcd_invert_cg: not converged after %d iterations (|r|/|b'| = %.3e)",
                         inf.iterations, inf.schur_residual);
    return PLQCD_OK;
}
