// Per-revolution thermal kernels, batched over solves.
//
// One revolution of the reference (inertiadifference,
// 3905/Thermal/NominalPole/main.cpp:1473-1557) advances every non-converged
// facet through NTAU steps of FTCS conduction + a Newton-Raphson radiative
// surface boundary.  Its self-heating flux reads only previous-revolution
// surface temperatures (main.cpp:1505-1527), so the revolution splits into
//
//   k_selfheat_w   W[f][s] = eps*sigma*T_{r-1}[s][f]^4          (transpose)
//   k_selfheat_q   Q[s][f] = sum_k W[g_k][s] * vf_k  (list order)  -- A6
//                  (FAST: the tensor-core product of atpm_spmm_tc.cu)
//   k_conduction   depth column in registers, NTAU steps, Newton BC -- A1
//                  (FAST: over the active-facet list once at most half a
//                  solve is active)
//   k_prepare, k_conduction_few   FAST revolutions with few advancing facets:
//                  several lanes per facet (atpm_conduction_split.cu, as the
//                  REFERENCE and FP64 sweeps)
//   k_converge     shape_converged (main.cpp:1876-1909)             -- A4
//                  (+ the active-facet lists and row-block activity)
//   advance        revolution counter / stop rule (main.cpp:2522-2539)
//
// All of them read the per-solve control word and return at once for solves
// that have stopped, so the same launch sequence (or a captured graph of it)
// can be replayed until every solve in the batch is done.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "atpm_column.cuh"
#include "atpm_gather.cuh"
#include "atpm_internal.h"

namespace atpm {

// ------------------------------------------------------------- self-heating
// W[f][s] = (eps*sigma) * T[s][f]^4 over a 32x32 tile, transposed in shared memory
template <int MODE>
__global__ void __launch_bounds__(256) k_selfheat_w(Batch b) {
    using A = Ar<MODE>;
    using R = typename A::R;
    const int4 t = b.wmap[blockIdx.x];
    const DevSolve& sv = b.tab[t.x];
    if (!sv.ctl->active || sv.nnz == 0) return;
    __shared__ R sm[32][33];
    const int nf = sv.nf, ntau = sv.ntau;
    const R* T = static_cast<const R*>(sv.stemp1);
    R* W = static_cast<R*>(sv.W);
    Sc<MODE> c;
    c.load(sv);
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int s = t.z + j, f = t.y + threadIdx.x;
        R v = R(0);
        if (s < ntau && f < nf) v = A::mul(c.esw, Pw<MODE>::p4(b.p4, T[(size_t)s * nf + f], sv.status));
        sm[j][threadIdx.x] = v;
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int f = t.y + j, s = t.z + threadIdx.x;
        if (f < nf && s < ntau) W[(size_t)f * gather_ld(ntau) + s] = sm[threadIdx.x][j];
    }
}

// Q[s][f] = sum over f's list of W[g][s] * vf, accumulated in list order
// (main.cpp:1519-1529), a warp per facet over rows of W (atpm_gather.cuh).  The
// map's tiles of 32 facets x 32 steps are regrouped: the tiles of one span of
// 32 lanes' steps (four in 32 bits, two in 64; fewer at the end) share its
// facets.  Last facets first: a binary's secondary comes last and has its
// longest rows.  REFERENCE, 6,280 facets, 613 steps: 0.44 -> 0.19 ms.
template <int MODE, int N>
__global__ void __launch_bounds__(N == 1 ? 1024 : 256) k_selfheat_q(Batch b) {
    using A = Ar<MODE>;
    using R = typename A::R;
    constexpr int SPAN = 32 * N, WARPS = N == 1 ? 32 : 8;
    const int4 t = b.wmap[gridDim.x - 1 - blockIdx.x];
    const DevSolve& sv = b.tab[t.x];
    if (!sv.ctl->active) return;
    __shared__ R sm[SPAN][33];
    const int nf = sv.nf, ntau = sv.ntau, ld = gather_ld(ntau);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile = t.z / 32, span = tile / N, share = min(N, (ntau + 31) / 32 - span * N);
    const int f0 = t.y + 32 * (tile % N) / share, f1 = min(nf, t.y + 32 * (tile % N + 1) / share);
    const int s0 = span * SPAN, s = s0 + lane * N;
    const bool inst = (MODE == MODE_FP64) ? (sv.ti_d == 0.0) : (sv.ti == 0.0f);
    const R* rows = static_cast<const R*>(sv.W) + (s < ntau ? s : 0);
    for (int f = f0 + warp; f < f1; f += WARPS) {
        R q[N] = {};
        if (inst || !sv.freeze || !sv.conv[f])
            gather<R, N>(sv.dep_idx, sv.dep_vf, sv.dep_ptr[f], sv.dep_ptr[f + 1], rows, ld, [](float v) { return (R)v; },
                      [&](int, R c, const R(&x)[N]) {
#pragma unroll
                          for (int u = 0; u < N; ++u) q[u] = A::add(q[u], A::mul(x[u], c));
                      });
#pragma unroll
        for (int u = 0; u < N; ++u) sm[lane * N + u][f - f0] = q[u];
    }
    __syncthreads();
    const int nw = f1 - f0;
    for (int i = threadIdx.x; i < SPAN * 32; i += 32 * WARPS) {
        const int so = i >> 5, fo = i & 31;
        if (fo < nw && s0 + so < ntau) static_cast<R*>(sv.Q)[(size_t)(s0 + so) * nf + f0 + fo] = sm[so][fo];
    }
}

// --------------------------------------------------------------- conduction
// REFERENCE and FP64 run the lane-split sweep (atpm_conduction_split.cu).  The
// sweeps record whether |stemp1-stemp0| >= TACC at some step (the
// shape_converged test), so no stemp history has to be re-read.
//
// FAST precision: the same update, scheduled for the FP32 pipes.
//  * The column is advanced as offsets theta_i = T_i - T_ref from a per-facet
//    reference (the bottom node at the start of the revolution).  The FTCS
//    Laplacian is translation-invariant, so each step rounds to the ulp of
//    theta (a few K) instead of the ulp of T (~300 K): 10-100x less roundoff
//    than the reference's absolute FP32 update, which is what keeps the FAST
//    path within 0.01 K of FP64 over hundreds of revolutions.
//  * Node 1 is advanced first (the boundary solve needs it); the Newton
//    boundary runs two iterations unconditionally (more only while the change
//    is still >= TACC/10), and the update of nodes 2..NX-1 -- independent of
//    the boundary result -- sits in the same basic block, so the scheduler
//    overlaps it with the Newton dependency chain.
// per-thread asynchronous copies (cp.async, 4 bytes) for the step prefetch of
// the FAST sweep: each thread copies and later reads only its own words, so
// no block barrier is involved
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int kFastPrefetch = 8;  // steps of forcing / flux / previous temperature in flight per facet

template <int NX>
__device__ __forceinline__ void column_revolution_fast(const DevSolve& sv, int f) {
    const int nf = sv.nf, ntau = sv.ntau;
    const bool sec = f >= sv.fsplit;  // non-synchronous secondary: its own rotation rate
    const float r = sec ? sv.r2 : sv.r, oma = sv.oma, es = sv.es, es4 = sv.es4, m1 = sec ? sv.m1_2 : sv.m1,
                tacc = sv.tacc, tacc10 = sv.tacc10;
    float* temp = static_cast<float*>(sv.temp);
    const float* __restrict__ E = static_cast<const float*>(sv.E);
    const float* __restrict__ Q = static_cast<const float*>(sv.Q);
    float* __restrict__ S0 = static_cast<float*>(sv.stemp0);
    float* __restrict__ S1 = static_cast<float*>(sv.stemp1);
    float T[NX + 1];
    const float Tref = temp[(size_t)NX * nf + f];
    // W tile addressing, advanced incrementally (no per-step division)
    __nv_bfloat16* Wb = static_cast<__nv_bfloat16*>(sv.Wb);
    const int N = sv.tc_n;
    const size_t chunk = (size_t)2 * N * 64;
    size_t wrow = Wb ? (size_t)(f >> 6) * sv.tc_nchunks * chunk : 0;
    const uint32_t kc = (uint32_t)(f & 63) >> 3, k7 = (uint32_t)f & 7u;
    int wn = 0;
#pragma unroll
    for (int i = 0; i <= NX; ++i) T[i] = __fsub_rn(temp[(size_t)i * nf + f], Tref);
    bool hot = false;
    int flags = 0;
    const int cap = sv.newton_cap;
    // E, Q and the previous temperature of step s + kFastPrefetch are copied
    // into this thread's shared-memory slots while step s computes: in the
    // late revolutions a few active facets per SM cannot hide DRAM latency
    // behind other warps
    constexpr int D = kFastPrefetch;
    __shared__ float pre[D][3][128];
    // the last 8 values of eps sigma T^4, written to this facet's W32 row
    // as two 16-byte stores per 8 steps (one full 32-byte sector)
    __shared__ float w8[8][128];
    float* W32 = Wb ? sv.W32 : nullptr;
    float* w32row = W32 ? W32 + (size_t)f * sv.w32_ld : nullptr;
    const int lt = threadIdx.x;
    for (int j = 0; j < D; ++j) {
        if (j < ntau) {
            const size_t oj = (size_t)j * nf + f;
            cp_async4(&pre[j][0][lt], E + oj);
            cp_async4(&pre[j][1][lt], Q + oj);
            cp_async4(&pre[j][2][lt], S1 + oj);
        }
        cp_async_commit();
    }
    size_t o = (size_t)f;
    int slot = 0;
    for (int s = 0; s < ntau; ++s, o += nf) {
        cp_async_wait<D - 1>();  // the copies of step s have landed
        const float e = pre[slot][0][lt], q = pre[slot][1][lt], old = pre[slot][2][lt];
        S0[o] = old;
        const float t1 = T[1];
        T[1] = ftcs_node(r, T[2], T[0], t1);
        const float a = __fmaf_rn(oma, e, q);
        // Newton iterations 1 and 2 on theta_0 (T_0 = Tref + theta_0)
        float DT;
        float th1 = newton_fast(T[0], Tref, T[1], a, m1, es, es4, DT);
        if (DT >= tacc10) th1 = newton_fast(th1, Tref, T[1], a, m1, es, es4, DT);
        // remaining nodes (independent of the boundary result)
        float tm = t1;
#pragma unroll
        for (int i = 2; i < NX; ++i) {
            const float ti = T[i];
            T[i] = ftcs_node(r, T[i + 1], tm, ti);
            tm = ti;
        }
        int it = 2;
        while (DT >= tacc10) {
            if (it >= cap) { flags |= ST_NEWTON_CAP; break; }
            th1 = newton_fast(th1, Tref, T[1], a, m1, es, es4, DT);
            ++it;
        }
        T[0] = th1;
        const float Tsurf = __fadd_rn(Tref, th1);
        S1[o] = Tsurf;
        if (Wb) {
            const float w = fast_w(sv.es_w, Tsurf);
            const uint32_t off = (uint32_t)wn * 64u + ((kc ^ ((uint32_t)wn & 7u)) << 3) + k7;
            const __nv_bfloat16 hi = __float2bfloat16_rn(w);
            Wb[wrow + off] = hi;
            Wb[wrow + (size_t)N * 64 + off] = w_lo(w, hi);
            if (++wn == N) { wn = 0; wrow += chunk; }
            if (w32row) {
                w8[s & 7][lt] = w;
                if ((s & 7) == 7) {
                    float4* d = reinterpret_cast<float4*>(w32row + (s - 7));
                    d[0] = make_float4(w8[0][lt], w8[1][lt], w8[2][lt], w8[3][lt]);
                    d[1] = make_float4(w8[4][lt], w8[5][lt], w8[6][lt], w8[7][lt]);
                }
            }
        }
        T[NX] = T[NX - 1];
        hot = hot || (fabsf(__fsub_rn(Tsurf, old)) >= tacc);
        // refill the slot just read (its words are consumed) with step s + D
        if (s + D < ntau) {
            const size_t od = o + (size_t)D * nf;
            cp_async4(&pre[slot][0][lt], E + od);
            cp_async4(&pre[slot][1][lt], Q + od);
            cp_async4(&pre[slot][2][lt], S1 + od);
        }
        cp_async_commit();
        if (++slot == D) slot = 0;
    }
    cp_async_wait<0>();
    if (w32row)  // the steps after the last full group of 8
        for (int s = ntau & ~7; s < ntau; ++s) w32row[s] = w8[s & 7][lt];
    if (!isfinite(__fadd_rn(T[0], Tref))) flags |= ST_NONFINITE;
#pragma unroll
    for (int i = 0; i <= NX; ++i) temp[(size_t)i * nf + f] = __fadd_rn(Tref, T[i]);
    sv.hot[f] = hot ? 1 : 0;
    if (flags) atomicOr(sv.status, flags);
}

// FAST, two adjacent facets per thread.  The sweep is issue-bound, so the
// pair is advanced with the packed FP32 instructions (fma/add/mul .f32x2):
// each lane of a pair is the scalar sweep's operation sequence with the same
// roundings, so both facets end bit-identical to column_revolution_fast.  The
// two facets' words sit side by side in every [step][facet] and
// [depth][facet] array (f even, nf even), so their loads and stores are
// 8-byte accesses and the two W tile entries one BF16x2 store.  The Newton
// solve runs while either lane still needs a step; a lane that has stopped
// keeps its value (per-lane select), so each facet takes its own iterations.
__device__ __forceinline__ float2 f2fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 f2add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 f2mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
// a - b with one rounding (b * -1 is exact), the value of __fsub_rn(a, b)
__device__ __forceinline__ float2 f2sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }

__device__ __forceinline__ float2 ftcs_node2(float2 r, float2 up, float2 dn, float2 t) {
    return f2fma(r, f2fma(make_float2(-2.0f, -2.0f), t, f2add(up, dn)), t);
}

// newton_fast on both lanes (nes = -es)
__device__ __forceinline__ float2 newton_fast2(float2 th, float2 Tref, float2 t1, float2 a, float2 m1, float2 nes,
                                               float2 es4, float2& DT) {
    const float2 TR = f2add(Tref, th);
    const float2 t2 = f2mul(TR, TR);
    const float2 sbc = f2fma(nes, f2mul(t2, t2), f2fma(m1, f2sub(t1, th), a));
    const float2 sbcd = f2fma(es4, f2mul(t2, TR), m1);
    const float2 th1 = f2add(th, make_float2(quotient(sbc.x, sbcd.x), quotient(sbc.y, sbcd.y)));
    const float2 d = f2sub(th1, th);
    DT = make_float2(fabsf(d.x), fabsf(d.y));
    return th1;
}

__device__ __forceinline__ void cp_async8(float2* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

template <int NX>
__device__ __forceinline__ void column_revolution_fast2(const DevSolve& sv, int f) {
    const int nf = sv.nf, ntau = sv.ntau;
    const bool sec0 = f >= sv.fsplit, sec1 = f + 1 >= sv.fsplit;
    const float2 r = make_float2(sec0 ? sv.r2 : sv.r, sec1 ? sv.r2 : sv.r);
    const float2 m1 = make_float2(sec0 ? sv.m1_2 : sv.m1, sec1 ? sv.m1_2 : sv.m1);
    const float2 oma = make_float2(sv.oma, sv.oma), nes = make_float2(-sv.es, -sv.es),
                 es4 = make_float2(sv.es4, sv.es4), esw = make_float2(sv.es_w, sv.es_w);
    const float tacc = sv.tacc, tacc10 = sv.tacc10;
    float* temp = static_cast<float*>(sv.temp);
    const float* __restrict__ E = static_cast<const float*>(sv.E);
    const float* __restrict__ Q = static_cast<const float*>(sv.Q);
    float* __restrict__ S0 = static_cast<float*>(sv.stemp0);
    float* __restrict__ S1 = static_cast<float*>(sv.stemp1);
    float2 T[NX + 1];
    const float2 Tref = *reinterpret_cast<const float2*>(temp + (size_t)NX * nf + f);
    __nv_bfloat16* Wb = static_cast<__nv_bfloat16*>(sv.Wb);
    const int N = sv.tc_n;
    const size_t chunk = (size_t)2 * N * 64;
    size_t wrow = Wb ? (size_t)(f >> 6) * sv.tc_nchunks * chunk : 0;
    const uint32_t kc = (uint32_t)(f & 63) >> 3, k7 = (uint32_t)f & 7u;  // f even: f + 1 is the next BF16
    int wn = 0;
#pragma unroll
    for (int i = 0; i <= NX; ++i) T[i] = f2sub(*reinterpret_cast<const float2*>(temp + (size_t)i * nf + f), Tref);
    bool hot0 = false, hot1 = false;
    int flags = 0;
    const int cap = sv.newton_cap;
    constexpr int D = kFastPrefetch;
    __shared__ float2 pre2[D][3][64];
    __shared__ float2 w8p[8][64];
    float* W32 = Wb ? sv.W32 : nullptr;
    float* w32r0 = W32 ? W32 + (size_t)f * sv.w32_ld : nullptr;
    float* w32r1 = W32 ? w32r0 + sv.w32_ld : nullptr;
    const int lt = threadIdx.x;
    for (int j = 0; j < D; ++j) {
        if (j < ntau) {
            const size_t oj = (size_t)j * nf + f;
            cp_async8(&pre2[j][0][lt], E + oj);
            cp_async8(&pre2[j][1][lt], Q + oj);
            cp_async8(&pre2[j][2][lt], S1 + oj);
        }
        cp_async_commit();
    }
    size_t o = (size_t)f;
    int slot = 0;
    for (int s = 0; s < ntau; ++s, o += nf) {
        cp_async_wait<D - 1>();
        const float2 e = pre2[slot][0][lt], q = pre2[slot][1][lt], old = pre2[slot][2][lt];
        *reinterpret_cast<float2*>(S0 + o) = old;
        const float2 t1 = T[1];
        T[1] = ftcs_node2(r, T[2], T[0], t1);
        const float2 a = f2fma(oma, e, q);
        float2 DT;
        float2 th1 = newton_fast2(T[0], Tref, T[1], a, m1, nes, es4, DT);
        {
            const bool n0 = DT.x >= tacc10, n1 = DT.y >= tacc10;
            if (n0 || n1) {
                float2 d2;
                const float2 t = newton_fast2(th1, Tref, T[1], a, m1, nes, es4, d2);
                if (n0) { th1.x = t.x; DT.x = d2.x; }
                if (n1) { th1.y = t.y; DT.y = d2.y; }
            }
        }
        float2 tm = t1;
#pragma unroll
        for (int i = 2; i < NX; ++i) {
            const float2 ti = T[i];
            T[i] = ftcs_node2(r, T[i + 1], tm, ti);
            tm = ti;
        }
        for (int it = 2;; ++it) {
            const bool n0 = DT.x >= tacc10, n1 = DT.y >= tacc10;
            if (!n0 && !n1) break;
            if (it >= cap) { flags |= ST_NEWTON_CAP; break; }
            float2 d2;
            const float2 t = newton_fast2(th1, Tref, T[1], a, m1, nes, es4, d2);
            if (n0) { th1.x = t.x; DT.x = d2.x; }
            if (n1) { th1.y = t.y; DT.y = d2.y; }
        }
        T[0] = th1;
        const float2 Tsurf = f2add(Tref, th1);
        *reinterpret_cast<float2*>(S1 + o) = Tsurf;
        if (Wb) {
            const float2 t2s = f2mul(Tsurf, Tsurf);
            const float2 w = f2mul(esw, f2mul(t2s, t2s));
            const uint32_t off = (uint32_t)wn * 64u + ((kc ^ ((uint32_t)wn & 7u)) << 3) + k7;
            const __nv_bfloat162 hi = __floats2bfloat162_rn(w.x, w.y);
            const float2 lo = f2sub(w, __bfloat1622float2(hi));
            *reinterpret_cast<__nv_bfloat162*>(Wb + wrow + off) = hi;
            *reinterpret_cast<__nv_bfloat162*>(Wb + wrow + (size_t)N * 64 + off) = __floats2bfloat162_rn(lo.x, lo.y);
            if (++wn == N) { wn = 0; wrow += chunk; }
            if (w32r0) {
                w8p[s & 7][lt] = w;
                if ((s & 7) == 7) {
                    float4* d0 = reinterpret_cast<float4*>(w32r0 + (s - 7));
                    float4* d1 = reinterpret_cast<float4*>(w32r1 + (s - 7));
                    d0[0] = make_float4(w8p[0][lt].x, w8p[1][lt].x, w8p[2][lt].x, w8p[3][lt].x);
                    d0[1] = make_float4(w8p[4][lt].x, w8p[5][lt].x, w8p[6][lt].x, w8p[7][lt].x);
                    d1[0] = make_float4(w8p[0][lt].y, w8p[1][lt].y, w8p[2][lt].y, w8p[3][lt].y);
                    d1[1] = make_float4(w8p[4][lt].y, w8p[5][lt].y, w8p[6][lt].y, w8p[7][lt].y);
                }
            }
        }
        T[NX] = T[NX - 1];
        const float2 dT = f2sub(Tsurf, old);
        hot0 = hot0 || (fabsf(dT.x) >= tacc);
        hot1 = hot1 || (fabsf(dT.y) >= tacc);
        if (s + D < ntau) {
            const size_t od = o + (size_t)D * nf;
            cp_async8(&pre2[slot][0][lt], E + od);
            cp_async8(&pre2[slot][1][lt], Q + od);
            cp_async8(&pre2[slot][2][lt], S1 + od);
        }
        cp_async_commit();
        if (++slot == D) slot = 0;
    }
    cp_async_wait<0>();
    if (w32r0)
        for (int s = ntau & ~7; s < ntau; ++s) {
            w32r0[s] = w8p[s & 7][lt].x;
            w32r1[s] = w8p[s & 7][lt].y;
        }
    const float2 t0 = f2add(T[0], Tref);
    if (!isfinite(t0.x) || !isfinite(t0.y)) flags |= ST_NONFINITE;
#pragma unroll
    for (int i = 0; i <= NX; ++i) *reinterpret_cast<float2*>(temp + (size_t)i * nf + f) = f2add(Tref, T[i]);
    sv.hot[f] = hot0 ? 1 : 0;
    sv.hot[f + 1] = hot1 ? 1 : 0;
    if (flags) atomicOr(sv.status, flags);
}

// How a FAST revolution's depth sweep runs, decided once per revolution from
// the facets that advance (one warp, over the solves): with few of them the
// lane-split sweep takes every solve (k_conduction_few; its warps are dealt
// out here, solve by solve), else the thread-per-facet kernels do.  The answer
// goes to the batch's first solve, where all of them read it: exactly one of
// the forms advances each facet.
__device__ __forceinline__ void tail_mode(const Batch& b) {
    const int lane = threadIdx.x & 31;
    auto advancing = [&](int i) {
        if (i >= b.n) return 0;
        const DevSolve& s = b.tab[i];
        if (!s.ctl->active || s.ti == 0.0f) return 0;
        const int rev = s.ctl->rev;
        return active_listed(s, rev) ? s.act_cnt[rev & 1] : s.nf;
    };
    int total = 0;
    for (int i = lane; i < b.n; i += 32) total += advancing(i);
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    int lanes = 0;
    if (b.warp_tail && total <= b.few_limit) lanes = split_lanes(b.nx, total <= b.tail_limit ? kFewestLanes : kFewLanes);
    int start = 0;
    if (lanes) {
        const int per = 32 / lanes;  // facets per warp
        for (int i0 = 0; i0 < b.n; i0 += 32) {
            const int w = (advancing(i0 + lane) + per - 1) / per;
            int x = w;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (i0 + lane < b.n) b.tab[i0 + lane].act_cnt[ACT_START] = start + x - w;
            start += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    if (lane == 0) {
        b.tab[0].act_cnt[ACT_LANES] = lanes;
        b.tab[0].act_cnt[ACT_WARPS] = start;
    }
}

// What a FAST revolution needs to know before it runs, in one block: how its
// depth sweep runs, and the product's work items whose row block has an active
// facet, in map order, so that tickets are spent on work only.  A kernel for
// each and a memset of the counters cost a few us apiece in revolutions of
// some 140 (single solves, late revolutions): with the end of the revolution in
// k_converge, 1,280 facets 140.5 -> 137.5 us.
// A small block, which starts beside the other group's kernels: one of 1,024
// threads waited for a whole SM and held the sweep of eight inertias up 6 %.
constexpr int kPrepThreads = 256, kPrepWarps = kPrepThreads / 32;
constexpr int kPrepItems = 16;  // items a thread looks at in one pass

__global__ void __launch_bounds__(kPrepThreads) k_prepare(Batch b) {
    constexpr int PER = kPrepItems * kPrepWarps / 32;
    __shared__ int at[kPrepItems * kPrepWarps];
    __shared__ int count;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == kPrepWarps - 1) tail_mode(b);
    if (b.nq == 0) return;
    int base = 0;
    for (int i0 = 0; i0 < b.nq; i0 += kPrepThreads * kPrepItems) {
        unsigned mine = 0;  // the items of this thread that are in
#pragma unroll 8
        for (int k = 0; k < kPrepItems; ++k) {
            const int i = i0 + k * kPrepThreads + threadIdx.x;
            bool use = false;
            if (i < b.nq) {
                const int4 it = b.qmap[i];
                const DevSolve& sv = b.tab[it.x];
                const bool everyone = !sv.freeze || sv.ti == 0.0f;
                use = sv.ctl->active && sv.tc_tiles && (everyone || sv.rb_act[it.y]);
            }
            const unsigned m = __ballot_sync(0xffffffffu, use);
            if (lane == 0) at[k * kPrepWarps + warp] = __popc(m);
            mine |= use ? 1u << k : 0u;
        }
        __syncthreads();
        if (warp == 0) {  // exclusive sums of the counts, PER consecutive ones a lane
            int c[PER], sum = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                c[k] = at[lane * PER + k];
                sum += c[k];
            }
            int x = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) count = x;
            x += base - sum;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                at[lane * PER + k] = x;
                x += c[k];
            }
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < kPrepItems; ++k) {
            const bool use = (mine >> k) & 1u;
            const unsigned m = __ballot_sync(0xffffffffu, use);
            if (use)
                b.tc_list[at[k * kPrepWarps + warp] + __popc(m & ((1u << lane) - 1u))] =
                    b.qmap[i0 + k * kPrepThreads + threadIdx.x];
        }
        base += count;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        b.tc_work[0] = base;  // list length
        b.tc_work[1] = 0;     // next ticket
        // parts an item is dealt out in: as many as the SMs take in one wave
        // (a second wave reads every V tile again).  us a revolution whole and
        // dealt out: 90.2 and 80.6 at 320 facets x 300 steps, 132.6 and 130 at
        // 2,740 x 400, 137.6 and 134.3 at 1,280 x 720; half a wave 80, 132 and 137.5.
        b.tc_work[2] = max(1, min(b.tc_nmax / 16, base ? b.sms / base : 1));
    }
}

__device__ __forceinline__ bool few_now(const Batch& b) { return b.tab[0].act_cnt[ACT_LANES] != 0; }

// instequilibrium (main.cpp:1563-1612): every facet, every step, no depth
__device__ __forceinline__ void column_equilibrium_fast(const DevSolve& sv, int f) {
    const int nf = sv.nf, ntau = sv.ntau;
    const float* E = static_cast<const float*>(sv.E);
    const float* Q = static_cast<const float*>(sv.Q);
    float* S0 = static_cast<float*>(sv.stemp0);
    float* S1 = static_cast<float*>(sv.stemp1);
    bool hot = false;
    WOut w;
    w.open(sv, f);
    for (int s = 0; s < ntau; ++s) {
        const size_t o = (size_t)s * nf + f;
        const float old = S1[o];
        S0[o] = old;
        const float tn = dev_qroot((sv.oma * E[o] + Q[o]) / sv.es);
        S1[o] = tn;
        if (w.tiles) w.store(s, tn);
        hot = hot || (fabsf(tn - old) >= sv.tacc);
    }
    sv.hot[f] = hot ? 1 : 0;
}

// the solve sweeps its list of active facets this revolution (at most half
// of them active, freeze protocol, list built for this revolution)
__device__ __forceinline__ bool list_mode(const Batch& b, const DevSolve& sv) {
    const int rev = sv.ctl->rev;
    return b.warp_tail && active_listed(sv, rev) && 2 * sv.act_cnt[rev & 1] <= sv.nf;
}
// the facet-range sweep of this solve runs as pairs (variant 4, even facet
// count) while at least 90 % of its facets are active: once facets freeze,
// pairs split and their other halves would fall to the scalar sweep, so the
// whole range goes back to it.  Both kernels read the same list count
// (written by the previous revolution's convergence test), so exactly one
// of them takes each facet.
__device__ __forceinline__ bool pairs_here(const Batch& b, const DevSolve& sv) {
    if (b.cond_variant != 4 || (sv.nf & 1)) return false;
    const int rev = sv.ctl->rev;
    // no count for this revolution (every facet active before revolution 7,
    // or no lists kept): pairs; split pairs fall to the scalar sweep
    if (!active_listed(sv, rev)) return true;
    return 10 * sv.act_cnt[rev & 1] >= 9 * sv.nf;
}

// MINB: minimum resident blocks per SM requested from the register allocator
// (the variants trade registers for occupancy, picked at run time)
template <int NX, int MINB>
__global__ void __launch_bounds__(128, MINB) k_conduction(Batch b) {
    const int2 fb = b.fmap[blockIdx.x];
    const DevSolve& sv = b.tab[fb.x];
    if (!sv.ctl->active) return;
    if (sv.ti != 0.0f) {
        if (few_now(b)) return;  // k_conduction_few runs this revolution
        // at most half the facets active: the solve's blocks sweep its
        // list of active facets instead of its facet range, so active
        // facets fill whole warps and the remaining blocks exit
        const int rev = sv.ctl->rev;
        if (list_mode(b, sv)) {
            const int k = fb.y + threadIdx.x;
            if (k >= sv.act_cnt[rev & 1]) return;
            column_revolution_fast<NX>(sv, sv.act_list[(size_t)(rev & 1) * sv.nf + k]);
            return;
        }
    }
    const int f = fb.y + threadIdx.x;
    if (f >= sv.nf) return;
    // k_conduction_pairs sweeps the pairs whose facets are both active;
    // a facet whose partner is frozen is swept here
    if (sv.ti != 0.0f && pairs_here(b, sv) && !(sv.freeze && sv.conv[f ^ 1])) return;
    if (sv.ti == 0.0f) { column_equilibrium_fast(sv, f); return; }
    if (sv.freeze && sv.conv[f]) return;
    column_revolution_fast<NX>(sv, f);
}

// FAST conduction variant 4: the facet-range sweep (every revolution before
// the active list or the lane-split form takes over) as pairs of adjacent
// facets, 64 threads per 128-facet block.  Only pairs with both facets
// active are swept here: k_conduction, launched beside it, takes a facet
// whose partner is frozen (the freeze flags do not change during the sweep),
// and every facet of a solve with an odd facet count.
template <int NX>
__global__ void __launch_bounds__(64, 4) k_conduction_pairs(Batch b) {
    const int2 fb = b.fmap[blockIdx.x];
    const DevSolve& sv = b.tab[fb.x];
    if (!sv.ctl->active || sv.ti == 0.0f || !pairs_here(b, sv) || few_now(b) || list_mode(b, sv)) return;
    const int f = fb.y + 2 * threadIdx.x;
    if (f >= sv.nf || (sv.freeze && (sv.conv[f] || sv.conv[f + 1]))) return;
    column_revolution_fast2<NX>(sv, f);
}

// -------------------------------------------------------------- convergence
// the end of a solve's revolution
__device__ __forceinline__ void advance(const DevSolve& sv) {
    Ctl* ctl = sv.ctl;
    if (!ctl->active) return;
    const int rev = ctl->rev;
    if (rev > 5) {
        const int n = __ldcg(&sv.counts[rev]);
        ctl->numconv = n;
        ctl->converged = (n == sv.nf) ? 1 : 0;
    } else {
        sv.counts[rev] = ctl->numconv;
    }
    // read by this revolution's conduction; k_converge of rev + 1 refills it
    sv.act_cnt[rev & 1] = 0;
    sv.act_cnt[2 + (rev & 1)] = -1;
    ctl->rev = rev + 1;
    if (ctl->converged || rev + 1 >= sv.revcap || (*sv.status & ST_NONFINITE)) ctl->active = 0;
}

__device__ __forceinline__ void converge(const Batch& b) {
    const int2 fb = b.fmap[blockIdx.x];
    const DevSolve& sv = b.tab[fb.x];
    if (!sv.ctl->active) return;
    const int rev = sv.ctl->rev;
    if (rev <= 5) return;
    const int f = fb.y + threadIdx.x;
    int c = 0;
    if (f < sv.nf) {
        const bool ok = !sv.hot[f];
        if (ok) { sv.conv[f] = 1; c = 1; }
    }
    c = __syncthreads_count(c);
    if (threadIdx.x == 0 && c) atomicAdd(&sv.counts[rev], c);
    // row-block activity read by the next revolution's tensor-core product
    // (blocks of this kernel are the product's 128-facet row blocks)
    const int any = __syncthreads_or(f < sv.nf && !sv.conv[f]);
    if (threadIdx.x == 0) sv.rb_act[fb.y >> 7] = any ? 1 : 0;
    // list of the facets still active for the next revolution (FAST, freeze):
    // each block appends its active facets as one segment in facet order, so
    // a sweep over the list keeps runs of neighbouring facets together
    if (b.mode == MODE_FAST && sv.freeze) {
        __shared__ int wcnt[4], base;
        const bool act = f < sv.nf && !sv.conv[f];
        const unsigned m = __ballot_sync(0xffffffffu, act);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (lane == 0) wcnt[warp] = __popc(m);
        __syncthreads();
        if (threadIdx.x == 0) {
            const int t = wcnt[0] + wcnt[1] + wcnt[2] + wcnt[3];
            base = t ? atomicAdd(&sv.act_cnt[(rev + 1) & 1], t) : 0;
            if (fb.y == 0) sv.act_cnt[2 + ((rev + 1) & 1)] = rev + 1;
        }
        __syncthreads();
        int off = base;
        for (int w = 0; w < warp; ++w) off += wcnt[w];
        if (act) sv.act_list[(size_t)((rev + 1) & 1) * sv.nf + off + __popc(m & ((1u << lane) - 1u))] = f;
    }
}

// The convergence test, and with the last block to finish the end of the
// revolution for every solve (a kernel of its own took 3 to 5 us).  The ticket
// counter, of the batch's first solve, wraps to zero with the last block.
__global__ void __launch_bounds__(128) k_converge(Batch b) {
    __shared__ bool last;
    converge(b);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned* ticket = reinterpret_cast<unsigned*>(&b.tab[0].act_cnt[ACT_TICKET]);
        last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = threadIdx.x; i < b.n; i += blockDim.x) advance(b.tab[i]);
}

// ------------------------------------------------------------- initial state
// initialisetemperatures (main.cpp:1439-1467): the facet's mean absorbed flux,
// summed in step order, -> T0 = ((1 - A) mean / (eps sigma))^0.25 everywhere in
// its column and at every step; FAST's W (BF16 tiles and FP32 rows) with it.
// A block owns 64 facets and a span of steps.  Its threads bring E in through
// shared memory, kInitSteps steps at a time with the next ones in flight, and
// one thread a facet sums them: a thread a facet on its own waited for E 720
// times over.  W is constant over the steps, so it is packed once and stored
// 16 bytes a lane.  Bound by the stores; FAST, 21,760 facets x 720 steps with
// the W kernels 199 -> 77 us a call, 1,280 facets 53 -> 25.
constexpr int kInitFacets = 64, kInitSteps = 32;

template <int MODE>
__global__ void __launch_bounds__(256) k_initial(DevSolve sv, PowTab pq) {
    using A = Ar<MODE>;
    using R = typename A::R;
    constexpr int PER = kInitFacets * kInitSteps / 256;  // elements a thread brings in at a time
    __shared__ R e[kInitSteps][kInitFacets];
    __shared__ R t0[kInitFacets];
    __shared__ float w0[kInitFacets];
    __shared__ __align__(16) __nv_bfloat16 wt[2][kInitFacets];
    const int nf = sv.nf, ntau = sv.ntau, f0 = blockIdx.x * kInitFacets;
    const int col = threadIdx.x % kInitFacets, row = threadIdx.x / kInitFacets, f = f0 + col;
    constexpr int ROWS = 256 / kInitFacets;
    const R* E = static_cast<const R*>(sv.E);
    R next[PER];
    auto fetch = [&](int s0) {
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int s = s0 + row + j * ROWS;
            next[j] = (f < nf && s < ntau) ? __ldg(E + (size_t)s * nf + f) : R(0);
        }
    };
    const R inv = A::div(R(1), (R)ntau);
    R m = R(0);
    fetch(0);
    for (int s0 = 0; s0 < ntau; s0 += kInitSteps) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < PER; ++j) e[row + j * ROWS][col] = next[j];
        __syncthreads();
        fetch(s0 + kInitSteps);
        if (row == 0) {
            if (s0 + kInitSteps <= ntau) {
#pragma unroll
                for (int j = 0; j < kInitSteps; ++j) m = A::add(m, A::mul(inv, e[j][col]));
            } else {
                for (int j = 0; s0 + j < ntau; ++j) m = A::add(m, A::mul(inv, e[j][col]));
            }
        }
    }
    if (row == 0) {
        R v = R(0);
        if (f < nf) {
            if constexpr (MODE == MODE_FP64) {
                v = sqrt(sqrt(__ddiv_rn(__dmul_rn(sv.oma_d, m), sv.es_d)));
            } else {
                const float x = __fdiv_rn(__fmul_rn(sv.oma, m), sv.es);
                v = (MODE == MODE_REF) ? libm_qroot(pq, x, sv.status) : dev_qroot(x);  // powf(x, 0.25f)
            }
        }
        t0[col] = v;
        if constexpr (MODE == MODE_FAST) {
            const float w = f < nf ? fast_w(sv.es_w, v) : 0.0f;
            const __nv_bfloat16 hi = __float2bfloat16_rn(w);
            w0[col] = w;
            wt[0][col] = hi;
            wt[1][col] = w_lo(w, hi);
        }
    }
    __syncthreads();
    // this block's steps [b0, b1): whole multiples of 32 up to the last
    const int span = ((ntau + 31) / 32 + gridDim.y - 1) / gridDim.y * 32;
    const int b0 = blockIdx.y * span, b1 = min(ntau, b0 + span);
    const R v = t0[col];
    if (f < nf) {
        R* S0 = static_cast<R*>(sv.stemp0);
        R* S1 = static_cast<R*>(sv.stemp1);
        for (int s = b0 + row; s < b1; s += ROWS) {
            S0[(size_t)s * nf + f] = v;
            S1[(size_t)s * nf + f] = v;
        }
        R* temp = static_cast<R*>(sv.temp);
        if (blockIdx.y == 0)
            for (int i = row; i <= sv.nx; i += ROWS) temp[(size_t)i * nf + f] = v;
    }
    if constexpr (MODE == MODE_FAST) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (sv.Wb) {  // eight lanes a step's row of 64 facets, swizzled
            uint4* Wb = static_cast<uint4*>(sv.Wb) + (size_t)blockIdx.x * sv.tc_nchunks * sv.tc_n * 16;
            const uint4* hi = reinterpret_cast<const uint4*>(wt[0]);
            const uint4* lo = reinterpret_cast<const uint4*>(wt[1]);
            for (int s = b0 + threadIdx.x / 8; s < b1; s += 32) {
                const int n = s % sv.tc_n, at = lane & 7;
                uint4* d = Wb + (size_t)(s / sv.tc_n) * sv.tc_n * 16 + n * 8 + at;
                d[0] = hi[at ^ (n & 7)];
                d[sv.tc_n * 8] = lo[at ^ (n & 7)];
            }
        }
        if (sv.W32)
            for (int r = warp; r < min(kInitFacets, nf - f0); r += 8) {
                float* d = sv.W32 + (size_t)(f0 + r) * sv.w32_ld;
                const float w = w0[r];
                for (int s = b0 + 4 * lane; s < b1; s += 128) {
                    if (s + 4 <= b1) *reinterpret_cast<float4*>(d + s) = make_float4(w, w, w, w);
                    else
                        for (int u = s; u < b1; ++u) d[u] = w;
                }
            }
    }
}

// FP64 energy balance of the current revolution: sums over facets and steps
// of absorbed flux (1-A)E + Q, emitted eps*sigma*T^4 and T.
template <int MODE>
__global__ void k_energy(DevSolve sv) {
    using R = typename Ar<MODE>::R;
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    double ab = 0.0, em = 0.0, tm = 0.0;
    if (f < sv.nf) {
        const R* E = static_cast<const R*>(sv.E);
        const R* Q = static_cast<const R*>(sv.Q);
        const R* S1 = static_cast<const R*>(sv.stemp1);
        const double oma = 1.0 - (double)sv.alb_d, es = sv.es_d;
        for (int s = 0; s < sv.ntau; ++s) {
            const size_t o = (size_t)s * sv.nf + f;
            const double T = (double)S1[o];
            ab += oma * (double)E[o] + (double)Q[o];
            em += es * (T * T) * (T * T);
            tm += T;
        }
    }
    for (int d = 16; d > 0; d >>= 1) {
        ab += __shfl_down_sync(0xffffffffu, ab, d);
        em += __shfl_down_sync(0xffffffffu, em, d);
        tm += __shfl_down_sync(0xffffffffu, tm, d);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sv.diag[0], ab);
        atomicAdd(&sv.diag[1], em);
        atomicAdd(&sv.diag[2], tm);
    }
}

// ------------------------------------------------------------------ launchers
#define NX_LIST(X) X(8) X(12) X(16) X(24) X(32) X(40) X(48) X(56) X(64)

bool conduction_nx_supported(int nx) {
#define NX_CASE(n) if (nx == n) return true;
    NX_LIST(NX_CASE)
#undef NX_CASE
    return false;
}

// some revolution has the paired sweep
static bool pairs_run(const Batch& b) { return b.cond_variant == 4 && !few_always(b); }

template <int MODE>
static int launch_rev_part(const Batch& b, int part, cudaStream_t st) {
    if (MODE == MODE_FAST && part == 0) k_prepare<<<1, kPrepThreads, 0, st>>>(b);
    // FAST + tensor cores: the conduction sweep keeps W current
    if (MODE == MODE_FAST && b.nq > 0 && part == 0) return cudaGetLastError() == cudaSuccess ? 0 : 2;
    if (MODE == MODE_FAST && b.nq > 0 && part == 1) return launch_spmm_tc(b, st);
    switch (part) {
        case 0: if (b.nw > 0) k_selfheat_w<MODE><<<b.nw, dim3(32, 8), 0, st>>>(b); break;
        case 1: {
            constexpr int W = kWide<typename Ar<MODE>::R>;
            if (b.nw > 0 && gather_wide(b.nw, W, b.sms)) k_selfheat_q<MODE, W><<<b.nw, 256, 0, st>>>(b);
            else if (b.nw > 0) k_selfheat_q<MODE, 1><<<b.nw, 1024, 0, st>>>(b);
            break;
        }
        case 2:
            if (MODE != MODE_FAST) return launch_conduction_split(b, st);
            switch (b.nx) {
#define NX_CASE(N)                                                                       \
    case N:                                                                               \
        if (b.cond_variant >= 3) k_conduction<N, 3><<<b.nfb, 128, 0, st>>>(b);            \
        else if (b.cond_variant == 2) k_conduction<N, 2><<<b.nfb, 128, 0, st>>>(b);       \
        else k_conduction<N, 1><<<b.nfb, 128, 0, st>>>(b);                                \
        if (pairs_run(b)) k_conduction_pairs<N><<<b.nfb, 64, 0, st>>>(b);                 \
        break;
                NX_LIST(NX_CASE)
#undef NX_CASE
                default: return 1;
            }
            return launch_conduction_few(b, st);
        case 3: k_converge<<<b.nfb, 128, 0, st>>>(b); break;
        default: return 1;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_revolution_part(const Batch& b, int part, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    switch (b.mode) {
        case MODE_REF: return launch_rev_part<MODE_REF>(b, part, st);
        case MODE_FP64: return launch_rev_part<MODE_FP64>(b, part, st);
        case MODE_FAST: return launch_rev_part<MODE_FAST>(b, part, st);
    }
    return 1;
}

int kernels_per_revolution(const Batch& b) {
    const bool tc = b.mode == MODE_FAST && b.nq > 0;
    // k_spmm_tc (+ k_spmm_rem), or W + Q
    const int selfheat = tc ? 1 + (b.rem_nmb > 0 ? 1 : 0) : (b.nw > 0 ? 2 : 0);
    // k_prepare, k_conduction, k_conduction_few (+ k_conduction_pairs)
    const int conduction = b.mode == MODE_FAST ? (pairs_run(b) ? 4 : 3) : 1;
    return selfheat + conduction + 1;                    // + k_converge
}

int launch_revolution(const Batch& b, stream_t st) {
    for (int part = 0; part < kRevolutionParts; ++part) {
        const int rc = launch_revolution_part(b, part, st);
        if (rc) return rc;
    }
    return 0;
}

// the steps are split between blocks until there are two a SM: a block that
// stores all of them takes 32 us a call at 1,280 facets x 720 steps, against
// 25 us split; with four or eight a SM 5,440 facets take 39 and 53 us, with two 38
int launch_initial(const DevSolve& s, const PowTab& pq, int sms, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    const int g = (s.nf + kInitFacets - 1) / kInitFacets;
    const dim3 grid((unsigned)g, (unsigned)std::max(1, std::min((s.ntau + 31) / 32, 2 * sms / g)));
    switch (s.mode) {
        case MODE_REF: k_initial<MODE_REF><<<grid, 256, 0, st>>>(s, pq); break;
        case MODE_FP64: k_initial<MODE_FP64><<<grid, 256, 0, st>>>(s, pq); break;
        default: k_initial<MODE_FAST><<<grid, 256, 0, st>>>(s, pq); break;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// Progress of every solve of a batch for one read-back: its control word,
// status word and the convergence counts of its last `window` revolutions
// (record of 5 + window ints per solve)
__global__ void k_progress(Batch b, int window, int* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.n) return;
    const DevSolve& s = b.tab[i];
    int* o = out + (size_t)i * (5 + window);
    const Ctl c = *s.ctl;
    o[0] = c.rev;
    o[1] = c.active;
    o[2] = c.converged;
    o[3] = c.numconv;
    o[4] = *s.status;
    for (int j = 0; j < window; ++j) {
        const int r = c.rev - window + j;
        o[5 + j] = (r >= 0 && r < s.revcap) ? s.counts[r] : 0;
    }
}

int launch_progress(const Batch& b, int window, int* out, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    k_progress<<<(b.n + 127) / 128, 128, 0, st>>>(b, window, out);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_energy_balance(const DevSolve& s, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    const int g = (s.nf + 127) / 128;
    if (s.mode == MODE_FP64) k_energy<MODE_FP64><<<g, 128, 0, st>>>(s);
    else k_energy<MODE_REF><<<g, 128, 0, st>>>(s);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace atpm
