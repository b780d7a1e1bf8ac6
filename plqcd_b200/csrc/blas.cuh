// blas.cuh -- vector kernels and FP64 reductions for the solvers.
#pragma once

#include <cuda_runtime.h>

#include "internal.h"

namespace plqcd {

// Solver scalars kept in device memory. Reductions finalise them on the
// device (last block of the reducing kernel, or a kernel of one block after
// it), so kernels read alpha / beta from here, and whether the iteration
// needs a reliable update is decided here too (RED_RR): the host queues the
// next iteration before it has read the outcome of this one, and the kernels
// of an iteration queued past a halt do nothing.
struct CgState {
    double rr;       // |r_sloppy|^2 (iterated), or |r|^2 after a reliable update
    double rr_old;   // previous rr
    double pAp;      // <p, A p> = |Mhat p|^2
    double alpha;    // rr / pAp
    double beta;     // rr / rr_old
    double sr2;      // |b' - Mhat x|^2 at the last reliable update (Schur residual)
    double aux;      // last plain reduction result
    double check[4]; // |b - D x|^2, |b|^2 of the even and the odd sites
    double maxrr, target, delta2;  // largest rr since the last update, trigger for a convergence check, delta^2
    int halt;        // a reliable update is due (or rr is not finite)
    int run;         // iterations since the last reliable update
    int mixed;
    int max_run;     // update after this many iterations without one
};

// what the host needs to know of an iteration, stored by the sum RED_RR
struct CgReport {
    double rr;
    int halt;
    int pad;
};

// Reduction scratch: per-block partials, the arrival counter of the
// last-block pattern, and the CgState block.
struct RedScratch {
    double *partials = nullptr;  // hop_sum_partials(Vh) doubles, at least kMaxRedBlocks
    unsigned *counter = nullptr;
    CgState *state = nullptr;
};
constexpr int kMaxRedBlocks = 1184;  // 8 x 148 SMs
constexpr int kBlasBlock = 256;
size_t red_scratch_bytes(long Vh);
// carve a RedScratch out of `mem` (red_scratch_bytes(), zero-initialised)
RedScratch red_scratch_from(void *mem, long Vh);

enum RedOp : int {
    RED_AUX = 0,     // state.aux = sum
    RED_ALPHA = 1,   // state.pAp = sum; state.alpha = state.rr / sum
    RED_RR = 2,      // state.rr_old = state.rr; state.rr = sum; state.beta = sum / state.rr_old; decide halt
    RED_SR2 = 3,     // state.sr2 = sum
    RED_RR_TRUE = 4, // the restart of a reliable update: state.rr = sum; state.beta = sum / state.rr_old; halt = 0
    RED_RR_INIT = 5, // state.rr = state.rr_old = state.maxrr = sum; state.target *= sum
    RED_CHECK_E = 6, // state.check[0], [1] = two sums
    RED_CHECK_O = 7, // state.check[2], [3] = two sums
};

#ifdef __CUDACC__
// st: the state as it was when the launch began, loaded beforehand (one
// round trip to L2 instead of one per field); out: where the new values go
__device__ __forceinline__ void red_apply(RedOp op, double sum, double sum2, const CgState &st, CgState *out,
                                          CgReport *report) {
    switch (op) {
        case RED_AUX: out->aux = sum; break;
        case RED_ALPHA:
            out->pAp = sum;
            out->alpha = sum > 0 ? st.rr / sum : 0.0;
            break;
        case RED_RR: {
            const int run = st.run + 1;
            const int halt = (st.mixed && sum < st.delta2 * st.maxrr) || sum <= st.target || !isfinite(sum) ||
                             run >= st.max_run;
            if (report) *report = CgReport{sum, halt, 0};
            out->halt = halt;
            out->run = run;
            out->rr_old = st.rr;
            out->rr = sum;
            out->beta = st.rr > 0 ? sum / st.rr : 0.0;
            if (!halt) out->maxrr = fmax(st.maxrr, sum);
            break;
        }
        case RED_SR2: out->sr2 = sum; break;
        case RED_RR_TRUE:
            out->rr = sum;
            out->beta = st.rr_old > 0 ? sum / st.rr_old : 0.0;
            out->maxrr = sum;
            if (sum <= st.target) out->target = 0.25 * st.target;
            out->run = 0;
            out->halt = 0;
            break;
        case RED_RR_INIT:
            out->rr = sum;
            out->rr_old = sum;
            out->maxrr = sum;
            out->target = st.target * sum;
            break;
        case RED_CHECK_E:
            out->check[0] = sum;
            out->check[1] = sum2;
            break;
        case RED_CHECK_O:
            out->check[2] = sum;
            out->check[3] = sum2;
            break;
    }
}
#endif

// A hop out = a H in + b x with a sum over its sites, taken in its epilogue
// (dslash_ahead.cu); `red` needs hop_sum_partials(Vh) partials.
//   HOP_NORM:   out stored; |out|^2
//   HOP_UPDATE: out not stored; rvec -= alpha out in place; |rvec|^2
//   HOP_RESID:  z = c - out stored to `out` in the format out_prec; |z|^2 (F64 hops)
//   HOP_CHECK:  z = c - out, nothing stored; |z|^2 and |c|^2 (F64 hops)
enum HopSumKind : int { HOP_NORM = 1, HOP_UPDATE = 2, HOP_RESID = 3, HOP_CHECK = 4 };
struct HopSum {
    HopSumKind kind = HOP_NORM;
    RedOp op = RED_AUX;
    const void *c = nullptr;
    void *rvec = nullptr;
    int out_prec = PLQCD_F64;
    CgReport *report = nullptr;  // RED_RR: page-locked host memory, written by the device
};
size_t hop_sum_partials(long Vh);

// |x_f|^2 of nf fields stored back to back; scratch: nf * norm2_blocks(Vh)
// partials and nf counters (zero on entry, left zero on exit)
int norm2_blocks(long Vh);
int preload_norm2_multi();
int launch_norm2_multi(const Geom &g, cudaStream_t s, const void *fields, int prec, int nf, double *partials,
                       unsigned *counters, double *out);
// xmode 1: x_s = alpha p, 2: x_s += alpha p, 0: no x update; then p = r + beta p
// (xmode 1 and 2, an iteration's update, do nothing once the state has halted)
int blas_cg_p_x(const Geom &g, cudaStream_t s, void *p, const void *rs, int prec, void *xs, int xprec, int xmode,
                const RedScratch &r);
// x64 += x_s (fresh: x_s counts as zero) [+ alpha p when p != null, with p in prec]
int blas_accum(const Geom &g, cudaStream_t s, void *x64, const void *xs, int xprec, bool fresh, const void *p,
               int prec, const RedScratch &r);
// c.x must be set; with c.halt the launch does nothing once *c.halt is set
int launch_hop_sum(const Geom &g, cudaStream_t s, const DslashCall &c, const HopSum &h, const RedScratch &r);

// FP64 multi-RHS hop with HOP_RESID or HOP_CHECK per RHS (dslash_mrhs_links.cu):
// out, in, x and h.c are blocks of nrhs fields (out in the format h.out_prec;
// not written by HOP_CHECK); sums[nrhs] (HOP_CHECK: sums[2 * nrhs], |z|^2
// then |c|^2). partials: nrhs * ceil(Vh / 32) doubles, twice that for
// HOP_CHECK. Meant for nrhs >= 2.
int launch_mrhs_links_sum(const Geom &g, cudaStream_t s, const plqcd_gauge *gf, void *out, const void *in, int nrhs,
                          int out_parity, double a, const void *x, double b, const HopSum &h, double *partials,
                          double *sums);

int preload_mrhs_links_resid(int recon, int out_prec);

}  // namespace plqcd
