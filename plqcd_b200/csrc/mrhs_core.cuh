// mrhs_core.cuh -- arguments and epilogue shared by the multi-RHS kernels
// (dslash_mrhs.cu, dslash_mrhs_links.cu).
#pragma once

#include "dslash_core.cuh"
#include "internal.h"
#include "raw_loads.cuh"

namespace plqcd {
namespace dev {

struct MrhsArgs {
    const void *gauge;
    const char *in;
    char *out;
    const char *x;
    size_t fbytes;
    int nrhs, ntiles;
    long Vh;
    int L0, L0h, L1, L2, L3;
    int out_parity;
    double a_up, a_low, b, g5_in;
    RhsSink sink;  // fused CG sums (RHS-pair kernels, epi > 0)
};

__device__ __forceinline__ double sq_sum(const cx<float> v[12]) {
    double s = 0;
#pragma unroll
    for (int k = 0; k < 12; k++) s += (double)v[k].re * v[k].re + (double)v[k].im * v[k].im;
    return s;
}

// epilogue of the RHS-pair kernels: scale (and xpay with x from xload(j,
// xv)), then EPI 0 / 1: store (1: v = |out|^2 per RHS); EPI 2: r -= alpha
// out in place, v = |r|^2 (out is not stored). Threads past the last
// site (valid false) only take part in the sums.
template <class SIO, bool XPAY, int EPI, class XLoad>
__device__ __forceinline__ void pair_epilogue(const MrhsArgs &a, int r0, bool two, int h, bool valid,
                                              const cx<f2> acc[12], XLoad xload, double v[2]) {
    const float aup = (float)a.a_up, alow = (float)a.a_low, b = (float)a.b;
    v[0] = v[1] = 0.0;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        if ((j == 1 && !two) || !valid) break;
        cx<float> o[12];
#pragma unroll
        for (int k = 0; k < 12; k++) o[k] = lane(acc[k], j);
        if (XPAY) {
            cx<float> xv[12];
            xload(j, xv);
#pragma unroll
            for (int k = 0; k < 12; k++) {
                const float ak = k < 6 ? aup : alow;
                o[k] = {fmaf(ak, o[k].re, b * xv[k].re), fmaf(ak, o[k].im, b * xv[k].im)};
            }
        } else {
#pragma unroll
            for (int k = 0; k < 12; k++) {
                const float ak = k < 6 ? aup : alow;
                o[k] = {ak * o[k].re, ak * o[k].im};
            }
        }
        if (EPI == 2) {
            const int f = r0 + j;
            if (a.sink.active[f]) {
                const float al = (float)a.sink.alpha[f];
                char *rf = a.sink.rvec + (size_t)f * a.fbytes;
                cx<float> rv[12];
                load_coherent<SIO>(rf, a.Vh, h, rv);
#pragma unroll
                for (int k = 0; k < 12; k++) rv[k] = {fmaf(-al, o[k].re, rv[k].re), fmaf(-al, o[k].im, rv[k].im)};
                SIO::store(rf, a.Vh, h, rv);
                v[j] = sq_sum(rv);
            }
        } else {
            SIO::store(a.out + (size_t)(r0 + j) * a.fbytes, a.Vh, h, o);
            if (EPI == 1 || EPI == 3) v[j] = sq_sum(o);
        }
    }
}

}  // namespace dev

// checked arguments of a multi-RHS launch (dslash_mrhs.cu)
int mrhs_args(const Geom &g, const void *gauge, int prec, void *out, const void *in, int nrhs, int out_parity,
              unsigned flags, double a, const void *x, double b, dev::MrhsArgs &m);

}  // namespace plqcd
