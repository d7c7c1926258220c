// Depth-column sweep with each facet's column split over the lanes of a warp
// (inertiadifference, 3905/Thermal/NominalPole/main.cpp:1473-1557).
//
// A facet's 720 or so steps are one dependent chain, so with a thread per
// facet a small shape leaves the GPU idle: 6,280 facets are 49 blocks, and a
// step costs a column of NX updates in series with the Newton solve.  Here L
// lanes share a facet: lane l holds nodes l K .. l K + K - 1 (K = NX / L, at
// least 3, so that lane 0 has nodes 0, 1 and 2 and the boundary solve waits on
// no shuffle), the two edge nodes are shuffled once per step, and every node's
// update is the thread-per-facet sweep's operation sequence, so all forms
// give the same bits.  The bottom node is a copy of node NX-1 after every
// step, so node NX-1 reads itself for it and the bottom is written at the end.
// Forcing, flux and the previous temperature of L steps at a time are
// prefetched by the lanes (lane j: step s0 + j) through a cp.async ring two
// blocks ahead; the step's result collects in the lane of that step, and the
// block's outputs are stored once per block.
//
// CTAs are one warp, so the few warps of a small shape spread over every SM.
// What bounds a small shape is a step's latency: at 1,280 facets, NX 56, a
// FAST step takes 0.14 us of which the two Newton iterations' dependent
// operations are about half (ncu: 70 instructions a step, 3.3 cycles each, one
// warp per scheduler); with one warp per facet and nodes 0-3 on every lane it
// took 0.20 us, with one thread per facet 0.36 us.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "atpm_column.cuh"
#include "atpm_internal.h"

namespace atpm {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kRing = 4;  // blocks of L steps in the prefetch ring

template <class R>
__device__ __forceinline__ void cp_async_word(R* dst, const R* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(sizeof(R))
                 : "memory");
}
__device__ __forceinline__ void ring_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ring_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// one FTCS update in each precision's own order
template <int MODE>
__device__ __forceinline__ typename Ar<MODE>::R ftcs(typename Ar<MODE>::R r, typename Ar<MODE>::R up,
                                                     typename Ar<MODE>::R dn, typename Ar<MODE>::R t) {
    using A = Ar<MODE>;
    using R = typename A::R;
    if constexpr (MODE == MODE_FAST) return ftcs_node(r, up, dn, t);
    else return A::add(t, A::mul(r, A::add(A::sub(up, A::mul(R(2), t)), dn)));
}

// the powers of a Newton step; the exception lookups only where `own`
template <int MODE>
__device__ __forceinline__ void powers(const Batch& b, typename Ar<MODE>::R t, bool own, int* st,
                                       typename Ar<MODE>::R& t4, typename Ar<MODE>::R& t3) {
    if constexpr (MODE == MODE_REF) {
        // lanes without a boundary node carry some interior temperature
        // through the same instructions; a fixed value keeps them out of the
        // lookups
        const float x = own ? t : 1.0f;
        t4 = libm_pow4(b.p4, x, st);
        t3 = libm_pow3(b.p3, x, st);
    } else {
        t4 = Pw<MODE>::p4(b.p4, t, st);
        t3 = Pw<MODE>::p3(b.p3, t, st);
    }
}

template <int MODE, int NX, int L>
struct Column {
    static constexpr int K = (NX + L - 1) / L;          // nodes per lane
    static constexpr int LN = (NX - 1) / K, KN = (NX - 1) % K;  // lane and slot of node NX-1
};

// one warp's staging: the prefetch ring and the surface temperatures of the
// block being swept
template <class R>
struct Stage {
    R ring[kRing][3][32];
    R out[2][32];
};

// the revolution of facet f on this group of L lanes; a group that is not
// `live` runs along and stores nothing.  A step's chain is node 1, then the
// Newton solve; everything else is kept off it: the step's absorbed flux is
// shuffled one step ahead, the edge nodes of the next step as soon as they are
// known, and the result leaves through shared memory.
template <int MODE, int NX, int L>
__device__ __forceinline__ void column_split(const DevSolve& sv, const Batch& b, int f, bool live,
                                             Stage<typename Ar<MODE>::R>& sm) {
    using A = Ar<MODE>;
    using R = typename A::R;
    using C = Column<MODE, NX, L>;
    constexpr int K = C::K;
    constexpr bool FAST = MODE == MODE_FAST;
    static_assert(L == 1 || K >= 3, "lane 0 holds nodes 0, 1 and 2");
    const int nf = sv.nf, ntau = sv.ntau;
    const int wl = threadIdx.x & 31, lane = wl & (L - 1);
    const bool head = lane == 0, own = head && live, last = lane == C::LN;
    Sc<MODE> c;
    c.load(sv);
    c.body(sv, f);
    R* temp = static_cast<R*>(sv.temp);
    const R* E = static_cast<const R*>(sv.E);
    const R* Q = static_cast<const R*>(sv.Q);
    R* S0 = static_cast<R*>(sv.stemp0);
    R* S1 = static_cast<R*>(sv.stemp1);
    const R Tref = FAST ? temp[(size_t)NX * nf + f] : R(0);
    R T[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int n = lane * K + k;
        const R t = n < NX ? temp[(size_t)n * nf + f] : R(0);
        T[k] = FAST ? (n < NX ? A::sub(t, Tref) : R(0)) : t;
    }
    bool hot = false;
    int flags = 0;
    const int cap = sv.newton_cap;
    WOut wout;
    if constexpr (FAST) wout.open(sv, f);
    const bool first = FAST || R(1) >= c.tacc10;  // the reference starts its loop with a change of 1 K
    auto fetch = [&](int s0, int slot) {
        const int s = s0 + lane;
        if (s < ntau) {
            const size_t o = (size_t)s * nf + f;
            cp_async_word(&sm.ring[slot][0][wl], E + o);
            cp_async_word(&sm.ring[slot][1][wl], Q + o);
            cp_async_word(&sm.ring[slot][2][wl], static_cast<const R*>(S1) + o);
        }
        ring_commit();
    };
    // lane j: the absorbed flux and the previous temperature of step s0 + j
    auto take = [&](int slot, R& absorbed, R& old) {
        const R e = sm.ring[slot][0][wl], q = sm.ring[slot][1][wl];
        if constexpr (FAST) absorbed = __fmaf_rn(c.oma, e, q);
        else absorbed = A::add(A::mul(c.oma, e), q);
        old = sm.ring[slot][2][wl];
    };
    int slot = 0;
    fetch(0, 0);
    fetch(L, 1);
    fetch(2 * L, 2);
    R ca, old, na, nold;
    ring_wait<2>();
    take(0, ca, old);
    R a = L > 1 ? __shfl_sync(FULL, ca, 0, L) : ca;
    R surf = FAST ? A::add(Tref, T[0]) : R(0);  // the surface temperature the next solve starts from
    R left = L > 1 ? __shfl_up_sync(FULL, T[K - 1], 1, L) : R(0);
    R right = L > 1 ? __shfl_down_sync(FULL, T[0], 1, L) : R(0);
    for (int s0 = 0, par = 0; s0 < ntau; s0 += L, par ^= 1) {
        fetch(s0 + 3 * L, (slot + 3) & (kRing - 1));
        slot = (slot + 1) & (kRing - 1);
        ring_wait<2>();
        take(slot, na, nold);  // the next block's
        const int nstep = min(L, ntau - s0);
// FAST: 4 steps in one body (fewer loop instructions, longer stretches to
// schedule); REFERENCE's steps are long enough that it loses by them (1.19 ->
// 1.40 ms a revolution at 6,280 facets)
#pragma unroll(FAST ? 4 : 1)
        for (int j = 0; j < nstep; ++j) {
            const R t0 = T[0];
            const R t1n = ftcs<MODE>(c.r, C::KN == 1 && last ? T[1] : T[2], t0, T[1]);
            // the boundary solve (only lane 0's counts)
            R th, DT;
            if constexpr (FAST) {
                th = newton_at(t0, surf, t1n, a, c.m1, c.es, c.es4, DT);
            } else {
                R p4, p3;
                powers<MODE>(b, t0, own, sv.status, p4, p3);
                const R sbc = A::sub(A::add(a, A::mul(c.m1, A::sub(t1n, t0))), A::mul(c.es, p4));
                const R sbcd = A::add(c.m1, A::mul(c.es4, p3));
                const R x = A::add(t0, A::div(sbc, sbcd));
                DT = first ? A::fabs_(A::sub(x, t0)) : R(0);
                th = first ? x : t0;
            }
            // the other nodes, from old values
            R tm = T[1];
            T[1] = t1n;
            const R edge = ftcs<MODE>(c.r, C::KN == 0 && last ? t0 : tm, left, t0);
#pragma unroll
            for (int k = 2; k < K; ++k) {
                const R tk = T[k];
                R up = k + 1 < K ? T[k + 1] : right;
                if (k == C::KN) up = last ? tk : up;  // node NX-1 reads itself for the bottom
                T[k] = ftcs<MODE>(c.r, up, tm, tk);
                tm = tk;
            }
            if constexpr (L > 1) {  // the next step's edges
                left = __shfl_up_sync(FULL, T[K - 1], 1, L);
                right = __shfl_down_sync(FULL, edge, 1, L);
            }
            const R an = L > 1 ? __shfl_sync(FULL, j + 1 < L ? ca : na, (j + 1) & (L - 1), L) : na;
            if constexpr (FAST) {
                float d2;
                const float t2 = newton_fast(th, Tref, t1n, a, c.m1, c.es, c.es4, d2);
                const bool two = DT >= c.tacc10;
                th = two ? t2 : th;
                DT = two && own ? d2 : 0.0f;
            } else if (!own) {
                DT = R(0);
            }
            int it = FAST ? 2 : 1;
            while (DT >= c.tacc10) {
                if (it >= cap) { flags |= ST_NEWTON_CAP; break; }
                if constexpr (FAST) {
                    th = newton_fast(th, Tref, t1n, a, c.m1, c.es, c.es4, DT);
                } else {
                    R p4, p3;
                    powers<MODE>(b, th, true, sv.status, p4, p3);
                    const R sbc = A::sub(A::add(a, A::mul(c.m1, A::sub(t1n, th))), A::mul(c.es, p4));
                    const R sbcd = A::add(c.m1, A::mul(c.es4, p3));
                    const R x = A::add(th, A::div(sbc, sbcd));
                    DT = A::fabs_(A::sub(x, th));
                    th = x;
                }
                ++it;
            }
            T[0] = head ? th : edge;
            a = an;
            surf = FAST ? A::add(Tref, th) : th;
            if (head) sm.out[par][wl + j] = surf;
        }
        if constexpr (L > 1) __syncwarp();
        if (live && lane < nstep) {
            const R ts = sm.out[par][wl];
            const int s = s0 + lane;
            const size_t o = (size_t)s * nf + f;
            S0[o] = old;
            S1[o] = ts;
            if constexpr (FAST) {
                if (wout.tiles) wout.store(s, ts);
            } else {
                if (!isfinite(ts)) flags |= ST_NONFINITE;
            }
            hot = hot || A::fabs_(A::sub(ts, old)) >= c.tacc;
        }
        ca = na;
        old = nold;
    }
    ring_wait<0>();
    if (!live) hot = false;
    const unsigned any = __ballot_sync(FULL, hot);
    if (!live) return;
    if constexpr (FAST) {
        if (head && !isfinite(A::add(T[0], Tref))) flags |= ST_NONFINITE;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int n = lane * K + k;
        if (n < NX) temp[(size_t)n * nf + f] = FAST ? A::add(Tref, T[k]) : T[k];
    }
    if (last) temp[(size_t)NX * nf + f] = FAST ? A::add(Tref, T[C::KN]) : T[C::KN];
    if (head) sv.hot[f] = (any >> (wl & ~(L - 1))) & (L == 32 ? FULL : (1u << L) - 1u) ? 1 : 0;
    if (flags) atomicOr(sv.status, flags);
}

// instequilibrium (main.cpp:1563-1612): no depth and no chain between steps;
// the group's lanes take every L-th step
template <int MODE, int L>
__device__ __forceinline__ void equilibrium_split(const DevSolve& sv, const Batch& b, int f, bool live) {
    using A = Ar<MODE>;
    using R = typename A::R;
    const int nf = sv.nf, ntau = sv.ntau;
    const int wl = threadIdx.x & 31, lane = wl & (L - 1);
    Sc<MODE> c;
    c.load(sv);
    const R* E = static_cast<const R*>(sv.E);
    const R* Q = static_cast<const R*>(sv.Q);
    R* S0 = static_cast<R*>(sv.stemp0);
    R* S1 = static_cast<R*>(sv.stemp1);
    bool hot = false;
    if (live)
        for (int s = lane; s < ntau; s += L) {
            const size_t o = (size_t)s * nf + f;
            const R old = S1[o];
            S0[o] = old;
            const R x = A::div(A::add(A::mul(c.oma, E[o]), Q[o]), c.es);
            R tn;
            if constexpr (MODE == MODE_FP64) tn = sqrt(sqrt(x));
            else tn = libm_qroot(b.pq, x, sv.status);  // powf(x, 0.25f)
            S1[o] = tn;
            hot = hot || (A::fabs_(A::sub(tn, old)) >= c.tacc);
        }
    const unsigned any = __ballot_sync(FULL, hot);
    if (live && lane == 0) sv.hot[f] = (any >> (wl & ~(L - 1))) & (L == 32 ? FULL : (1u << L) - 1u) ? 1 : 0;
}

// REFERENCE and FP64: every revolution; 4 L warps per 128-facet block of the
// map, 32 / L facets each
template <int MODE, int NX, int L>
__global__ void __launch_bounds__(32) k_conduction_split(Batch b) {
    using R = typename Ar<MODE>::R;
    constexpr int G = 32 / L, PER = 128 / G;
    const int2 fb = b.fmap[blockIdx.x / PER];
    const DevSolve& sv = b.tab[fb.x];
    if (!sv.ctl->active) return;
    __shared__ Stage<R> sm;
    const int f = fb.y + (blockIdx.x % PER) * G + (threadIdx.x & 31) / L;
    const bool inst = (MODE == MODE_FP64) ? (sv.ti_d == 0.0) : (sv.ti == 0.0f);
    const bool live = f < sv.nf && (inst || !(sv.freeze && sv.conv[f]));
    if (!__any_sync(FULL, live)) return;
    const int fc = min(f, sv.nf - 1);
    if (inst) equilibrium_split<MODE, L>(sv, b, fc, live);
    else column_split<MODE, NX, L>(sv, b, fc, live, sm);
}

// FAST: the facets k_prepare counted, as warps of 32 / L facets of one solve
// each (the active-facet list where one is kept for this revolution, else the
// facet range)
template <int NX, int L>
__device__ __forceinline__ void fast_warps(const Batch& b, int total, Stage<float>& sm) {
    constexpr int G = 32 / L;
    const int lane = threadIdx.x & 31;
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        // the solve whose warps include w: the last one starting at or before it
        int si = 0, start = 0;
        for (int i0 = 0; i0 < b.n; i0 += 32) {
            const int off = i0 + lane < b.n ? b.tab[i0 + lane].act_cnt[ACT_START] : total;
            const unsigned m = __ballot_sync(FULL, off <= w);
            if (!m) break;
            const int top = 31 - __clz(m);
            si = i0 + top;
            start = __shfl_sync(FULL, off, top);
            if (top < 31) break;
        }
        const DevSolve& sv = b.tab[si];
        const int rev = sv.ctl->rev;
        const bool listed = active_listed(sv, rev);
        const int n = listed ? sv.act_cnt[rev & 1] : sv.nf;
        const int k = (w - start) * G + lane / L;
        int f = min(k, n - 1);
        if (listed) f = sv.act_list[(size_t)(rev & 1) * sv.nf + f];
        const bool live = k < n && !(sv.freeze && sv.conv[f]);
        if (!__any_sync(FULL, live)) continue;
        column_split<MODE_FAST, NX, L>(sv, b, f, live, sm);
    }
}

template <int NX>
__global__ void __launch_bounds__(32) k_conduction_few(Batch b) {
    const int* d = b.tab[0].act_cnt;
    const int lanes = d[ACT_LANES], total = d[ACT_WARPS];
    if (lanes == 0) return;  // the thread-per-facet kernels run this revolution
    __shared__ Stage<float> sm;
    constexpr int L4 = split_lanes(NX, kFewLanes), L16 = split_lanes(NX, kFewestLanes);
    if (lanes == L16) fast_warps<NX, L16>(b, total, sm);
    else fast_warps<NX, L4>(b, total, sm);
}

template <int MODE, int NX>
void launch_nx(const Batch& b, int lanes, cudaStream_t st) {
    constexpr int L4 = split_lanes(NX, 4), L16 = split_lanes(NX, 16);
    if (lanes >= 16 && L16 > L4) k_conduction_split<MODE, NX, L16><<<b.nfb * 4 * L16, 32, 0, st>>>(b);
    else if (lanes >= 4) k_conduction_split<MODE, NX, L4><<<b.nfb * 4 * L4, 32, 0, st>>>(b);
    else k_conduction_split<MODE, NX, 1><<<b.nfb * 4, 32, 0, st>>>(b);
}

}  // namespace

#define SPLIT_NX(X) X(8) X(12) X(16) X(24) X(32) X(40) X(48) X(56) X(64)

int launch_conduction_split(const Batch& b, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    const int warps = 4 * b.nfb;  // with a thread per facet
    // Lanes per facet by the warps a thread per facet would give (ms per
    // revolution with 1 / 4 / 16 lanes, self-heating included; the line lies
    // where the next count stops winning).  REFERENCE: 0.99 / 0.78 / 0.74 at
    // 1,280 facets (NX 56, 720 steps), 2.21 / 1.99 / 1.97 at 9,280 (NX 48,
    // 600 steps), 3.56 / 3.40 / 4.08 at 16,960 (NX 56, 720 steps), 16.1 / 16.2
    // / 17.2 at 32,000 (NX 48, 500 steps).  FP64, bound by its 1/64-rate pipe,
    // where every lane group repeats the boundary solve: 2.68 / 1.30 / 1.04 at
    // 980 facets (NX 32, 360 steps), 8.55 / 3.98 / 4.12 at 1,800 (NX 56, 700
    // steps), 3.35 / 2.19 / 3.03 at 5,780 (NX 32, 400 steps), 2.68 / 3.23 /
    // 4.50 at 11,520 (NX 32, 300 steps).  One thread per facet in 128-thread
    // CTAs took 2.68, 4.54, 6.26 and 18.1 ms (REFERENCE, the sizes above) and
    // 3.03, 9.65, 3.73 and 2.98 ms (FP64).
    const bool f64 = b.mode == MODE_FP64;
    const int most16 = f64 ? b.sms / 4 : 2 * b.sms, most4 = f64 ? 2 * b.sms : 4 * b.sms;
    const int lanes = warps <= most16 ? 16 : warps <= most4 ? 4 : 1;
    switch (b.nx) {
#define NX_CASE(n)                                                       \
    case n:                                                              \
        if (b.mode == MODE_FP64) launch_nx<MODE_FP64, n>(b, lanes, st);  \
        else launch_nx<MODE_REF, n>(b, lanes, st);                       \
        break;
        SPLIT_NX(NX_CASE)
#undef NX_CASE
        default: return 1;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// FAST: runs the revolutions that k_prepare gives it, returns at once in the
// others
int launch_conduction_few(const Batch& b, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    const int grid = (int)std::min<long long>(16ll * b.sms, 64ll * b.nfb);
    switch (b.nx) {
#define NX_CASE(n) case n: k_conduction_few<n><<<grid, 32, 0, st>>>(b); break;
        SPLIT_NX(NX_CASE)
#undef NX_CASE
        default: return 1;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace atpm
