// Sums over view-factor lists of [facet][step] rows, 16 bytes of steps a lane
// (scattered sunlight, atpm_scatter.cu; self-heating, atpm_thermal.cu).
//
// A warp owns one row (facet) and 32 x 16 bytes of its steps.  It reads 32 list
// entries at a time, a lane each, and broadcasts them: an entry then costs one
// 512-byte load of its facet's row and a multiply and an add per step, in list
// order within each step.  With 4 bytes a lane and every lane reading every
// entry the sums were bound by instruction issue and by L1's request rate.
#pragma once
#include <cuda_runtime.h>

#include "atpm_internal.h"

namespace atpm {

// a lane's N consecutive steps
template <class R, int N> struct Steps {
    static __device__ __forceinline__ void get(const R* p, R (&x)[N]) {
        if constexpr (N * sizeof(R) == 16 && sizeof(R) == 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(p));
            x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        } else if constexpr (N * sizeof(R) == 16) {
            const double2 v = __ldg(reinterpret_cast<const double2*>(p));
            x[0] = v.x; x[1] = v.y;
        } else {
            static_assert(N == 1, "16 bytes or one step a lane");
            x[0] = __ldg(p);
        }
    }
    static __device__ __forceinline__ void put(R* p, const R (&x)[N]) {
        if constexpr (N * sizeof(R) == 16 && sizeof(R) == 4)
            *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
        else if constexpr (N * sizeof(R) == 16) *reinterpret_cast<double2*>(p) = make_double2(x[0], x[1]);
        else p[0] = x[0];
    }
};
template <class R> constexpr int kWide = 16 / sizeof(R);  // steps of a 16-byte lane

// 16 bytes a lane while that leaves some 128 warps an SM to hide the gathers
// behind, one step a lane below (tiles: 32 facets x 32 steps).  REFERENCE
// revolutions with one step and with four: 0.44 and 0.55 ms at 2,740 facets x
// 400 steps (1,118 tiles), 1.19 and 0.94 ms at 6,280 x 613 (3,940), 3.40 and
// 1.72 ms at 16,960 x 720 (12,190).
__host__ __forceinline__ bool gather_wide(long long tiles, int wide, int sms) {
    return tiles * 32 / wide >= 128ll * sms;
}

// row stride of [facet][step] arrays that are gathered: every row 16-byte aligned
__host__ __device__ __forceinline__ int gather_ld(int ntau) { return (ntau + 3) & ~3; }

// the list entries [k0, k1) in order: use(i, coefficient, steps of the entry's
// facet), where i is as odd as k - k0 is; `rows` points at facet 0's row at
// this lane's first step, scale(view factor) gives the coefficient.  All 32
// lanes call it together.
template <class R, int N, class Scale, class Use>
__device__ __forceinline__ void gather(const int* idx, const float* vf, int k0, int k1, const R* rows, size_t ld,
                                       Scale&& scale, Use&& use) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int U = N == 1 ? 8 : 4;  // rows in flight (wide: 8 took 0.94 -> 1.00 ms at 6,280 facets, 16 1.04)
    const int lane = threadIdx.x & 31;
    for (int kb = k0; kb < k1; kb += 32) {
        const bool in = kb + lane < k1;
        const int g = in ? __ldg(idx + kb + lane) : 0;
        const R c = in ? scale(__ldg(vf + kb + lane)) : R(0);
        const int n = min(32, k1 - kb);
        int j = 0;
        for (; j + U <= n; j += U) {
            R x[U][N];
#pragma unroll
            for (int u = 0; u < U; ++u) Steps<R, N>::get(rows + (size_t)__shfl_sync(FULL, g, j + u) * ld, x[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) use(u, __shfl_sync(FULL, c, j + u), x[u]);
        }
        for (; j < n; ++j) {
            R x[N];
            Steps<R, N>::get(rows + (size_t)__shfl_sync(FULL, g, j) * ld, x);
            use(j, __shfl_sync(FULL, c, j), x);
        }
    }
}

}  // namespace atpm
