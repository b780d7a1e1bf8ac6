// hop_sum.cuh -- epilogue of the hops that carry a sum (HopSum).
#pragma once

#include "blas.cuh"
#include "device_fields.cuh"
#include "raw_loads.cuh"

namespace plqcd {
namespace dev {

// What a hop with a sum in its epilogue needs besides its arguments (HopSum)
struct SumArgs {
    const void *c;
    void *rvec;
    RedScratch red;
    CgReport *report;
    RedOp op;
    int in_kernel;  // the last block adds the partials (small grids); else k_hop_sum_finish does
};

// (four partial sums: a single chain of 48 dependent FP64 operations takes
// longer than the loads of a small launch)
template <typename R>
__device__ __forceinline__ double site_norm2(const cx<R> v[12]) {
    double s[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 12; k++) s[k & 3] = fma((double)v[k].re, (double)v[k].re, fma((double)v[k].im, (double)v[k].im, s[k & 3]));
    return (s[0] + s[1]) + (s[2] + s[3]);
}

// one site: out is the hop's result with the xpay applied; v (and w for
// HOP_CHECK) receive the site's terms of the sums
template <class SIO, int SUM, int OP, typename R>
__device__ __forceinline__ void sum_epilogue(const SumArgs &q, void *out, long Vh, long h, const cx<R> acc[12],
                                             double &v, double &w) {
    if constexpr (SUM == HOP_NORM) {
        SIO::store(out, Vh, h, acc);
        v = site_norm2(acc);
    } else if constexpr (SUM == HOP_UPDATE) {
        const R al = (R)q.red.state->alpha;
        cx<R> rv[12];
        load_coherent<SIO>(q.rvec, Vh, h, rv);
#pragma unroll
        for (int k = 0; k < 12; k++) rv[k] = {fma(-al, acc[k].re, rv[k].re), fma(-al, acc[k].im, rv[k].im)};
        SIO::store(q.rvec, Vh, h, rv);
        v = site_norm2(rv);
    } else {
        cx<R> cv[12];
        load_coherent<SIO>(q.c, Vh, h, cv);
        if (SUM == HOP_CHECK) w = site_norm2(cv);
#pragma unroll
        for (int k = 0; k < 12; k++) cv[k] = csub(cv[k], acc[k]);
        v = site_norm2(cv);
        if constexpr (SUM == HOP_RESID) {
            using RO = typename SpinorIO<OP>::real;
            cx<RO> z[12];
#pragma unroll
            for (int k = 0; k < 12; k++) z[k] = {(RO)cv[k].re, (RO)cv[k].im};
            SpinorIO<OP>::store(out, Vh, h, z);
        }
    }
}

}  // namespace dev
}  // namespace plqcd
