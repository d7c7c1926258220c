// The crater's rim test: which of a sub-facet's 10 x 10 sub-points a direction
// reaches over the rim (sfcpartialshadow, GPU_code.cu:152-210, and the visible
// fractions of calculate_surface_global_viewfactors, main.cpp:1053-1181), shared
// by atpm_crater.cu (the Sun) and atpm_crater_forcing.cu (other facets).
#pragma once
#include <cuda_runtime.h>

#include "atpm_internal.h"

namespace atpm {

template <int MODE> struct Ca;
template <> struct Ca<MODE_REF> {
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
    static __device__ __forceinline__ float sqrt_(float a) { return __fsqrt_rn(a); }
};
template <> struct Ca<MODE_FAST> {
    static __device__ __forceinline__ float add(float a, float b) { return a + b; }
    static __device__ __forceinline__ float sub(float a, float b) { return a - b; }
    static __device__ __forceinline__ float mul(float a, float b) { return a * b; }
    static __device__ __forceinline__ float div(float a, float b) { return a / b; }
    static __device__ __forceinline__ float sqrt_(float a) { return sqrtf(a); }
};

constexpr int kRimPoints = 100;
constexpr int kRimDirs = 4;  // directions a thread tests together, so that a sub-point is placed once for all

// sub-point multipliers and the fraction that is left of a whole sub-facet
// after so many blocked points, per block
struct RimShared {
    float2 cm[kRimPoints];
    float left[kRimPoints + 1];
};

// one blocked point's part of a fraction; an emptied fraction stays empty
template <int MODE>
__device__ __forceinline__ float rim_take(float left, int points) {
    using A = Ca<MODE>;
    if (left < 0.0f) left = 0.0f;
    for (int i = 0; i < points && left != 0.0f; ++i) {
        left = A::sub(left, A::div(1.0f, 100.0f));
        if (left < 0.0f) left = 0.0f;
    }
    return left;
}

template <int MODE>
__device__ __forceinline__ void rim_open(RimShared& r, const CraterDev& c) {
    for (int p = threadIdx.x; p <= kRimPoints; p += blockDim.x) {
        if (p < kRimPoints) r.cm[p] = make_float2(c.cmult[2 * p], c.cmult[2 * p + 1]);
        r.left[p] = rim_take<MODE>(1.0f, p);
    }
    __syncthreads();
}

// A thread's sub-facet.  A point m is blocked in direction (w0, w1) of slope a if
//
//     m2 <= a (u - sqrt(100 - t^2)),  t = w0 m1 - w1 m0,  u = w0 m0 + w1 m1
//
// In real numbers that is z = u - h >= 0, h = m2 / a, and z^2 >= 100 - t^2, and as
// t^2 + u^2 = W r^2, W = w0^2 + w1^2 and r^2 = m0^2 + m1^2,
//
//     by = h (h - 2 u) + W r^2 - 100 >= 0  and  u >= h
//
// without a square root.  Let X = 100 + U^2, U = (|w0| + |w1|) max(|m0| + |m1|).
// Where h^2 <= 4 X, as wherever by is near 0, by is off by less than 2^-18 X, and
// the expression above, rounded operation by operation, draws its line within
// 2^-18 X of by = 0; where h is larger the signs of by and u - h are beyond doubt.
// The sign of u - h matters only where by >= 0, and is in doubt there only if
// 100 - W r^2 is next to nothing.  What 2^-16 X decides is therefore decided as the
// expression decides it; the rest, NaN among it, goes through the expression
// itself.  Only the number of blocked points counts, so their order is free.
template <int MODE>
struct Rim {
    using A = Ca<MODE>;
    float v2[3], t0[3], t1[3], size;

    __device__ __forceinline__ void load(const CraterDev& c, const RimShared& r, int j) {
        float most0 = 0.0f, most1 = 0.0f;
        for (int p = 0; p < kRimPoints; ++p) {
            most0 = fmaxf(most0, fabsf(r.cm[p].x));
            most1 = fmaxf(most1, fabsf(r.cm[p].y));
        }
        size = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v2[k] = c.cverts[3 * c.cfac[3 * j + 2] + k];
            t0[k] = c.ctri[6 * j + k];
            t1[k] = c.ctri[6 * j + 3 + k];
            if (k < 2) size += fabsf(v2[k]) + most0 * fabsf(t0[k]) + most1 * fabsf(t1[k]);
        }
    }

    __device__ __forceinline__ bool blocked(const float (&mp)[3], float w0, float w1, float a) const {
        const float R = 10.0f;
        const float tc1 = A::add(A::mul(A::mul(-1.0f, w1), mp[0]), A::mul(w0, mp[1]));
        const float rad = A::sqrt_(A::sub(A::mul(R, R), A::mul(tc1, tc1)));
        const float tc0 = A::sub(A::add(A::mul(w0, mp[0]), A::mul(w1, mp[1])), rad);
        return mp[2] <= A::mul(a, tc0);
    }

    // blocked points in each direction, two directions to a packed instruction
    __device__ __forceinline__ void count(const RimShared& r, const float (&w0)[kRimDirs], const float (&w1)[kRimDirs],
                                          const float (&a)[kRimDirs], int (&n)[kRimDirs]) const {
        constexpr int P = kRimDirs / 2;
        float2 x0[P], x1[P], ia[P], ww[P], floor_[P];
        auto slope = [](float v) { return v > 1e-30f ? 1.0f / v : __int_as_float(0x7fc00000); };
        auto slack = [&](int d) {
            const float u = (fabsf(w0[d]) + fabsf(w1[d])) * size;
            return (100.0f + u * u) * (1.0f / 65536.0f);
        };
#pragma unroll
        for (int k = 0; k < P; ++k) {
            x0[k] = make_float2(w0[2 * k], w0[2 * k + 1]);
            x1[k] = make_float2(w1[2 * k], w1[2 * k + 1]);
            ia[k] = make_float2(slope(a[2 * k]), slope(a[2 * k + 1]));
            ww[k] = __ffma2_rn(x0[k], x0[k], __fmul2_rn(x1[k], x1[k]));
            floor_[k] = make_float2(slack(2 * k), slack(2 * k + 1));
            n[2 * k] = n[2 * k + 1] = 0;
        }
#pragma unroll 2
        for (int p = 0; p < kRimPoints; ++p) {
            const float2 m = r.cm[p];
            float mp[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) mp[k] = A::add(A::add(v2[k], A::mul(m.x, t0[k])), A::mul(m.y, t1[k]));
            const float rr = __fmaf_rn(mp[0], mp[0], __fmul_rn(mp[1], mp[1]));
            bool hit[kRimDirs], sure[kRimDirs], all = true;
            auto decide = [&](int d, float u, float h, float c, float by, float slack) {
                hit[d] = by >= 0.0f && u >= h;
                sure[d] = fabsf(by) > slack && c < -slack;
                n[d] += hit[d] ? 1 : 0;
                all = all && sure[d];
            };
#pragma unroll
            for (int k = 0; k < P; ++k) {
                const float2 u = __ffma2_rn(x0[k], make_float2(mp[0], mp[0]), __fmul2_rn(x1[k], make_float2(mp[1], mp[1])));
                const float2 h = __fmul2_rn(ia[k], make_float2(mp[2], mp[2]));
                const float2 c = __ffma2_rn(ww[k], make_float2(rr, rr), make_float2(-100.0f, -100.0f));
                const float2 by = __ffma2_rn(h, __ffma2_rn(make_float2(-2.0f, -2.0f), u, h), c);
                decide(2 * k, u.x, h.x, c.x, by.x, floor_[k].x);
                decide(2 * k + 1, u.y, h.y, c.y, by.y, floor_[k].y);
            }
            if (!all) {
#pragma unroll
                for (int d = 0; d < kRimDirs; ++d)
                    if (!sure[d]) n[d] += (blocked(mp, w0[d], w1[d], a[d]) ? 1 : 0) - (hit[d] ? 1 : 0);
            }
        }
    }
};

}  // namespace atpm
