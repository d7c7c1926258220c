// Arithmetic of the depth-column sweeps, shared by the thread-per-facet forms
// (atpm_thermal.cu) and the lane-split form (atpm_conduction_split.cu).
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include "atpm_internal.h"

namespace atpm {

// ------------------------------------------------------------------ arithmetic
template <int MODE> struct Ar;
template <> struct Ar<MODE_REF> {
    using R = float;
    static __device__ __forceinline__ R add(R a, R b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ R sub(R a, R b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ R mul(R a, R b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ R div(R a, R b) { return __fdiv_rn(a, b); }
    static __device__ __forceinline__ R fabs_(R a) { return fabsf(a); }
};
template <> struct Ar<MODE_FP64> {
    using R = double;
    static __device__ __forceinline__ R add(R a, R b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ R sub(R a, R b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ R mul(R a, R b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ R div(R a, R b) { return __ddiv_rn(a, b); }
    static __device__ __forceinline__ R fabs_(R a) { return fabs(a); }
};
template <> struct Ar<MODE_FAST> {
    using R = float;
    static __device__ __forceinline__ R add(R a, R b) { return a + b; }
    static __device__ __forceinline__ R sub(R a, R b) { return a - b; }
    static __device__ __forceinline__ R mul(R a, R b) { return a * b; }
    static __device__ __forceinline__ R div(R a, R b) { return a / b; }
    static __device__ __forceinline__ R fabs_(R a) { return fabsf(a); }
};

template <int MODE> struct Pw;
template <> struct Pw<MODE_REF> {
    static __device__ __forceinline__ float p4(const PowTab& t, float x, int* st) { return libm_pow4(t, x, st); }
    static __device__ __forceinline__ float p3(const PowTab& t, float x, int* st) { return libm_pow3(t, x, st); }
};
template <> struct Pw<MODE_FP64> {
    static __device__ __forceinline__ double p4(const PowTab&, double x, int*) {
        double t2 = __dmul_rn(x, x);
        return __dmul_rn(t2, t2);
    }
    static __device__ __forceinline__ double p3(const PowTab&, double x, int*) { return __dmul_rn(__dmul_rn(x, x), x); }
};
template <> struct Pw<MODE_FAST> {
    static __device__ __forceinline__ float p4(const PowTab&, float x, int*) { float t2 = x * x; return t2 * t2; }
    static __device__ __forceinline__ float p3(const PowTab&, float x, int*) { return x * x * x; }
};

// per-mode scalar views of DevSolve
template <int MODE> struct Sc {
    using R = typename Ar<MODE>::R;
    R ti, oma, es, es4, m1, r, tacc, tacc10, esw;
    __device__ __forceinline__ void load(const DevSolve& s) {
        if constexpr (MODE == MODE_FP64) {
            ti = s.ti_d; oma = s.oma_d; es = s.es_d; es4 = s.es4_d; m1 = s.m1_d; r = s.r_d;
            tacc = s.tacc_d; tacc10 = s.tacc10_d; esw = s.es_w_d;
        } else {
            ti = s.ti; oma = s.oma; es = s.es; es4 = s.es4; m1 = s.m1; r = s.r;
            tacc = s.tacc; tacc10 = s.tacc10; esw = s.es_w;
        }
    }
    // facet f's own rotation rate (the secondary of a non-synchronous binary)
    __device__ __forceinline__ void body(const DevSolve& s, int f) {
        if (f < s.fsplit) return;
        if constexpr (MODE == MODE_FP64) { m1 = s.m1_2_d; r = s.r2_d; }
        else { m1 = s.m1_2; r = s.r2; }
    }
};

// FAST arithmetic is written with explicitly rounded operations (the _rn
// intrinsics are never contracted into a multiply-add), so the scalar, the
// lane-split and the paired forms of the sweep round alike, operation by
// operation, whatever the compiler schedules.
// eps sigma T^4 (with the IR absorptivity folded into es_w)
__device__ __forceinline__ float fast_w(float es_w, float t) {
    const float t2 = __fmul_rn(t, t);
    return __fmul_rn(es_w, __fmul_rn(t2, t2));
}
// the BF16 pair of W: hi = bf16(w), lo = bf16(w - hi)
__device__ __forceinline__ __nv_bfloat16 w_lo(float w, __nv_bfloat16 hi) {
    return __float2bfloat16_rn(__fsub_rn(w, __bfloat162float(hi)));
}

// FAST + tensor-core self-heating: eps*sigma*T^4 of the new surface
// temperature goes straight into the hi/lo BF16 tiles the next revolution's
// product reads (atpm_spmm_tc.cu), so no separate pass re-reads stemp1.
struct WOut {
    __nv_bfloat16* tiles;  // null: no tensor-core tiles
    float* w32;            // facet's row, null without a sparse remainder
    float es_w;
    int n;
    uint32_t col;          // f & 63
    size_t row;            // the facet's column block's first tile
    __device__ __forceinline__ void open(const DevSolve& sv, int f) {
        tiles = static_cast<__nv_bfloat16*>(sv.Wb);
        if (!tiles) return;
        es_w = sv.es_w;
        n = sv.tc_n;
        col = (uint32_t)(f & 63);
        row = (size_t)(f >> 6) * sv.tc_nchunks * (size_t)2 * n * 64;
        w32 = sv.W32 ? sv.W32 + (size_t)f * sv.w32_ld : nullptr;
    }
    __device__ __forceinline__ void store(int s, float t) const {
        const float w = fast_w(es_w, t);
        const uint32_t c = (uint32_t)s / (uint32_t)n;
        __nv_bfloat16* d = tiles + row + (size_t)c * 2 * n * 64 + swz((uint32_t)s - c * n, col);
        const __nv_bfloat16 hi = __float2bfloat16_rn(w);
        d[0] = hi;
        d[(size_t)n * 64] = w_lo(w, hi);
        if (w32) w32[s] = w;
    }
};

// One FTCS node update and one Newton step of the FAST sweep, shared by the
// thread-per-facet and the lane-split forms so both round alike.
// (up + dn) - 2 t is formed as one fma: 2 t is exact, so this is the
// rounding of the plain expression
__device__ __forceinline__ float ftcs_node(float r, float up, float dn, float t) {
    return __fmaf_rn(r, __fmaf_rn(-2.0f, t, __fadd_rn(up, dn)), t);
}

// x / y for a normal y: one approximate reciprocal and a product, the bits of
// __fdividef there (5.2e9 random pairs, y in [2^-20, 2^30)) without its range
// handling; y is m1 + 4 eps sigma T^3, a few W/m^2/K to some thousands
__device__ __forceinline__ float quotient(float x, float y) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    return __fmul_rn(x, r);
}

// one Newton step on theta_0: sbc = (m1 (t1 - th) + a) - es TR^4 with the
// emission folded into one multiply-add
// (TR: the temperature Tref + th)
__device__ __forceinline__ float newton_at(float th, float TR, float t1, float a, float m1, float es, float es4,
                                           float& DT) {
    const float t2 = __fmul_rn(TR, TR);
    const float sbc = __fmaf_rn(-es, __fmul_rn(t2, t2), __fmaf_rn(m1, __fsub_rn(t1, th), a));
    const float sbcd = __fmaf_rn(es4, __fmul_rn(t2, TR), m1);
    const float th1 = __fadd_rn(th, quotient(sbc, sbcd));
    DT = fabsf(__fsub_rn(th1, th));
    return th1;
}
__device__ __forceinline__ float newton_fast(float th, float Tref, float t1, float a, float m1, float es, float es4,
                                             float& DT) {
    return newton_at(th, __fadd_rn(Tref, th), t1, a, m1, es, es4, DT);
}

// ------------------------------------------------ lanes per facet (split form)
// lanes sharing a facet: at most `want`, and few enough that a lane has 3 nodes
__host__ __device__ constexpr int split_lanes(int nx, int want) {
    int l = want;
    while (l > 1 && (nx + l - 1) / l < 3) l >>= 1;
    return l;
}
constexpr int kFewLanes = 4, kFewestLanes = 16;

// a list of the solve's active facets is kept for this revolution
__device__ __forceinline__ bool active_listed(const DevSolve& sv, int rev) {
    return sv.freeze && rev >= 7 && sv.act_cnt[2 + (rev & 1)] == rev;
}

}  // namespace atpm
