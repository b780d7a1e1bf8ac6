// raw_loads.cuh -- loads of a site's stored bits into registers, apart from
// their conversion.
//
// A kernel that issues the loads of the next direction before it computes
// the current one keeps the stored form in registers meanwhile: a 16-bit
// spinor takes 13 registers, its converted form 24. The loads are volatile
// asm statements, so they stay in the order written (ahead of the
// arithmetic) instead of being moved down to their uses, and ordinary ones
// (not the non-coherent path), so a kernel may read what the one it overlaps
// with has written (pdl.cuh).
#pragma once

#include "device_fields.cuh"

namespace plqcd {
namespace dev {

__device__ __forceinline__ uint4 ld_v4(const void *p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_v2(const void *p) {
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double2 ld_d2(const void *p) {
    double2 v;
    asm volatile("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_f(const void *p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

template <class SIO>
struct RawSpinor;
template <int P>
struct RawSpinor16 {
    uint4 v[3];
    float n;
    __device__ __forceinline__ void load(const void *base, long Vh, int h) {
        const uint4 *p = static_cast<const uint4 *>(base) + h;
#pragma unroll
        for (int k = 0; k < 3; k++) v[k] = ld_v4(p + k * Vh);
        n = ld_f(SpinorIO16<P>::norms(base, Vh) + h);
    }
    __device__ __forceinline__ void get(cx<float> s[12], float &nn) const {
        SpinorIO16<P>::unpack3(v, s);
        nn = n;
    }
};
template <> struct RawSpinor<SpinorIO<PLQCD_F16>> : RawSpinor16<PLQCD_F16> {};
template <> struct RawSpinor<SpinorIO<PLQCD_BF16>> : RawSpinor16<PLQCD_BF16> {};
template <>
struct RawSpinor<SpinorIO<PLQCD_F32>> {
    uint4 v[6];
    __device__ __forceinline__ void load(const void *base, long Vh, int h) {
        const uint4 *p = static_cast<const uint4 *>(base) + h;
#pragma unroll
        for (int k = 0; k < 6; k++) v[k] = ld_v4(p + k * Vh);
    }
    __device__ __forceinline__ void get(cx<float> s[12], float &nn) const {
#pragma unroll
        for (int k = 0; k < 6; k++) {
            s[2 * k] = {__uint_as_float(v[k].x), __uint_as_float(v[k].y)};
            s[2 * k + 1] = {__uint_as_float(v[k].z), __uint_as_float(v[k].w)};
        }
        nn = 1.f;
    }
};
template <>
struct RawSpinor<SpinorIO<PLQCD_F64>> {
    double2 v[12];
    __device__ __forceinline__ void load(const void *base, long Vh, int h) {
        const double2 *p = static_cast<const double2 *>(base) + h;
#pragma unroll
        for (int k = 0; k < 12; k++) v[k] = ld_d2(p + k * Vh);
    }
    __device__ __forceinline__ void get(cx<double> s[12], double &nn) const {
#pragma unroll
        for (int k = 0; k < 12; k++) s[k] = {v[k].x, v[k].y};
        nn = 1.0;
    }
};
template <class LIO>
struct RawLink;
template <int R>
struct RawLink64 {
    double2 v[R / 2];
    __device__ __forceinline__ void load(const void *base, long Vh, int par, int mu, int h) {
        const double2 *p = static_cast<const double2 *>(base) + (long)(par * 4 + mu) * (R / 2) * Vh + h;
#pragma unroll
        for (int e = 0; e < R / 2; e++) v[e] = ld_d2(p + e * Vh);
    }
    __device__ __forceinline__ void get(cx<double> U[9]) const {
#pragma unroll
        for (int e = 0; e < R / 2; e++) U[e] = {v[e].x, v[e].y};
        if (R == 12) reconstruct_row2(U);
    }
};
template <> struct RawLink<LinkIO<PLQCD_F64, 18>> : RawLink64<18> {};
template <> struct RawLink<LinkIO<PLQCD_F64, 12>> : RawLink64<12> {};
template <int P>
struct RawLink16 {
    uint2 v[3];
    __device__ __forceinline__ void load(const void *base, long Vh, int par, int mu, int h) {
        const uint2 *p = static_cast<const uint2 *>(base) + (long)(par * 4 + mu) * 3 * Vh + h;
#pragma unroll
        for (int e = 0; e < 3; e++) v[e] = ld_v2(p + e * Vh);
    }
    __device__ __forceinline__ void get(cx<float> U[9]) const {
#pragma unroll
        for (int e = 0; e < 3; e++) {
            float2 a = Half2<P>::unpack(v[e].x), b = Half2<P>::unpack(v[e].y);
            U[2 * e] = {a.x, a.y};
            U[2 * e + 1] = {b.x, b.y};
        }
        reconstruct_row2(U);
    }
};
template <> struct RawLink<LinkIO<PLQCD_F16, 12>> : RawLink16<PLQCD_F16> {};
template <> struct RawLink<LinkIO<PLQCD_BF16, 12>> : RawLink16<PLQCD_BF16> {};
template <>
struct RawLink<LinkIO<PLQCD_F32, 12>> {
    uint4 v[3];
    __device__ __forceinline__ void load(const void *base, long Vh, int par, int mu, int h) {
        const uint4 *p = static_cast<const uint4 *>(base) + (long)(par * 4 + mu) * 3 * Vh + h;
#pragma unroll
        for (int e = 0; e < 3; e++) v[e] = ld_v4(p + e * Vh);
    }
    __device__ __forceinline__ void get(cx<float> U[9]) const {
#pragma unroll
        for (int e = 0; e < 3; e++) {
            U[2 * e] = {__uint_as_float(v[e].x), __uint_as_float(v[e].y)};
            U[2 * e + 1] = {__uint_as_float(v[e].z), __uint_as_float(v[e].w)};
        }
        reconstruct_row2(U);
    }
};

template <>
struct RawLink<LinkIO<PLQCD_F32, 18>> {
    uint2 v[9];
    __device__ __forceinline__ void load(const void *base, long Vh, int par, int mu, int h) {
        const uint2 *p = static_cast<const uint2 *>(base) + (long)(par * 4 + mu) * 9 * Vh + h;
#pragma unroll
        for (int e = 0; e < 9; e++) v[e] = ld_v2(p + e * Vh);
    }
    __device__ __forceinline__ void get(cx<float> U[9]) const {
#pragma unroll
        for (int e = 0; e < 9; e++) U[e] = {__uint_as_float(v[e].x), __uint_as_float(v[e].y)};
    }
};

// a spinor by ordinary loads, its norm applied
template <class SIO, typename R>
__device__ __forceinline__ void load_coherent(const void *base, long Vh, long h, cx<R> s[12]) {
    RawSpinor<SIO> raw;
    R n;
    raw.load(base, Vh, (int)h);
    raw.get(s, n);
    if (SIO::kScaled)
#pragma unroll
        for (int k = 0; k < 12; k++) s[k] = {s[k].re * n, s[k].im * n};
}

}  // namespace dev
}  // namespace plqcd
