// Scattered-sunlight kernels (reference singlescattering / multiplescattering,
// 3905/Thermal/NominalPole/main.cpp:1321-1433).
//
//   k_lit_cosine, k_single_rows
//                     E[f][s] = S cos_f shadow_f + sum_k vf_k S A cos_g shadow_g
//                     over rows of cos x shadow (atpm_gather.cuh)
//   k_single_scatter  the same without the rows, where there is no memory for
//                     them and for the no-allocation entry point: warp = 32
//                     steps of one facet
//   k_multi_gs        the reference's per-step Gauss-Seidel sweep in facet
//                     order (values of facets before f in this sweep, after f
//                     from the last sweep) until every |change| <= accuracy;
//                     one warp per step, lanes fetch 32 list entries at once
//                     and the two partial sums are accumulated in list order
//                     (unsorted lists, lists that chain facet to facet, very
//                     large shapes, and the no-allocation entry point)
//   k_multi_levels    the same sweeps with every facet whose lower neighbours
//                     are done swept together
//   k_multi_jacobi    FAST precision: Jacobi sweeps of every facet and step at
//                     once (rows as the single scattering), iterated to the
//                     same accuracy; the fixed point is the reference's, the
//                     iterates are not
//   k_forcing_t       [nf][ntau] -> [ntau][nf] for the conduction sweep
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <utility>

#include "../../include/atpm.h"
#include "atpm_gather.cuh"
#include "atpm_internal.h"

namespace atpm {

template <int MODE> struct Sa;
template <> struct Sa<MODE_REF> {
    using R = float;
    static __device__ __forceinline__ R add(R a, R b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ R sub(R a, R b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ R mul(R a, R b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ R div(R a, R b) { return __fdiv_rn(a, b); }
};
template <> struct Sa<MODE_FP64> {
    using R = double;
    static __device__ __forceinline__ R add(R a, R b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ R sub(R a, R b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ R mul(R a, R b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ R div(R a, R b) { return __ddiv_rn(a, b); }
};
template <> struct Sa<MODE_FAST> {
    using R = float;
    static __device__ __forceinline__ R add(R a, R b) { return a + b; }
    static __device__ __forceinline__ R sub(R a, R b) { return a - b; }
    static __device__ __forceinline__ R mul(R a, R b) { return a * b; }
    static __device__ __forceinline__ R div(R a, R b) { return a / b; }
};

template <int MODE>
__global__ void __launch_bounds__(256) k_single_scatter(DevSolve sv) {
    using A = Sa<MODE>;
    using R = typename A::R;
    const int nf = sv.nf, ntau = sv.ntau;
    const int f = blockIdx.y * blockDim.y + threadIdx.y;
    const int s = blockIdx.x * 32 + threadIdx.x;
    if (f >= nf) return;
    const R* cs = static_cast<const R*>(sv.cosil);
    const R solar = (MODE == MODE_FP64) ? (R)sv.solar_d : (R)sv.solar;
    const R alb = (MODE == MODE_FP64) ? (R)sv.alb_d : (R)sv.alb;
    const bool ok = s < ntau;
    const int sc = ok ? s : 0;
    R e = A::mul(A::mul(solar, cs[(size_t)f * ntau + sc]), (R)sv.shadow[(size_t)f * ntau + sc]);
    const int k1 = sv.dep_ptr[f + 1];
    for (int k = sv.dep_ptr[f]; k < k1; ++k) {
        const int g = __ldg(&sv.dep_idx[k]);
        const R v = (R)__ldg(&sv.dep_vf[k]);
        const size_t o = (size_t)g * ntau + sc;
        e = A::add(e, A::mul(A::mul(A::mul(A::mul(v, solar), alb), cs[o]), (R)sv.shadow[o]));
    }
    if (ok) static_cast<R*>(sv.Efm)[(size_t)f * ntau + s] = e;
}

// cos x shadow of every facet and step in rows of gather_ld(ntau) (the flag is 0
// or 1: multiplying by it first or last gives the same bits)
template <class R>
__global__ void __launch_bounds__(256) k_lit_cosine(DevSolve sv, R* p) {
    const int ld = gather_ld(sv.ntau);
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)sv.nf * ld) return;
    const int f = (int)(i / ld), s = (int)(i % ld);
    const size_t o = (size_t)f * sv.ntau + s;
    p[i] = s < sv.ntau ? static_cast<const R*>(sv.cosil)[o] * (R)sv.shadow[o] : R(0);
}

// stores a lane's steps s .. s + N - 1 of a [nf][ntau] row
template <class R, int N>
__device__ __forceinline__ void put_row(R* row, int ntau, int s, const R (&x)[N]) {
    if (ntau % N == 0) {
        Steps<R, N>::put(row + s, x);
        return;
    }
#pragma unroll
    for (int u = 0; u < N; ++u)
        if (s + u < ntau) row[s + u] = x[u];
}

// single scattering over the rows of k_lit_cosine: k_single_scatter's sums in
// the same order, from one gathered array.  next: FAST multiple scattering's
// first iterate, albedo x this (or null).  21,760 facets, 5.8 M entries, 720
// steps: 3.05 -> 1.3 ms.  The last facets go first: a binary's secondary comes
// last and has its longest rows.
template <int MODE, int N>
__global__ void __launch_bounds__(256) k_single_rows(DevSolve sv, const typename Sa<MODE>::R* lit,
                                                     typename Sa<MODE>::R* next) {
    // FAST rounds product and sum apart, as the form without rows does (there the
    // flag is the sum's factor): a forcing one ulp off moves the revolution in
    // which a facet counts as converged
    using A = Sa<MODE == MODE_FP64 ? MODE_FP64 : MODE_REF>;
    using R = typename A::R;
    const int f = (gridDim.y - 1 - blockIdx.y) * blockDim.y + threadIdx.y;
    if (f >= sv.nf) return;  // warp-uniform
    const int ld = gather_ld(sv.ntau), s = (blockIdx.x * 32 + threadIdx.x) * N;
    const bool ok = s < sv.ntau;
    const R* rows = lit + (ok ? s : 0);
    const R solar = (MODE == MODE_FP64) ? (R)sv.solar_d : (R)sv.solar;
    const R alb = (MODE == MODE_FP64) ? (R)sv.alb_d : (R)sv.alb;
    R own[N], e[N];
    Steps<R, N>::get(rows + (size_t)f * ld, own);
#pragma unroll
    for (int u = 0; u < N; ++u) e[u] = A::mul(solar, own[u]);
    gather<R, N>(sv.dep_idx, sv.dep_vf, sv.dep_ptr[f], sv.dep_ptr[f + 1], rows, ld,
                 [&](float v) { return A::mul(A::mul((R)v, solar), alb); },
                 [&](int, R c, const R(&x)[N]) {
#pragma unroll
                     for (int u = 0; u < N; ++u) e[u] = A::add(e[u], A::mul(c, x[u]));
                 });
    if (!ok) return;
    put_row(static_cast<R*>(sv.Efm) + (size_t)f * sv.ntau, sv.ntau, s, e);
    if (!next) return;
#pragma unroll
    for (int u = 0; u < N; ++u) e[u] = A::mul(alb, e[u]);
    Steps<R, N>::put(next + (size_t)f * ld + s, e);
}

// Gauss-Seidel multiple scattering, one warp per step.  `work` holds three
// [ntau][nf] arrays: solar power, previous sweep, current sweep.
template <int MODE>
__global__ void __launch_bounds__(32) k_multi_gs(DevSolve sv, void* work, int cap) {
    using A = Sa<MODE>;
    using R = typename A::R;
    const int nf = sv.nf, ntau = sv.ntau;
    const int s = blockIdx.x;
    const int lane = threadIdx.x;
    if (s >= ntau) return;
    R* sp = static_cast<R*>(work) + (size_t)s * nf;
    R* po = sp + (size_t)ntau * nf;
    R* pn = po + (size_t)ntau * nf;
    const R* cs = static_cast<const R*>(sv.cosil);
    R* Efm = static_cast<R*>(sv.Efm);
    const R solar = (MODE == MODE_FP64) ? (R)sv.solar_d : (R)sv.solar;
    const R alb = (MODE == MODE_FP64) ? (R)sv.alb_d : (R)sv.alb;
    const R acc = (MODE == MODE_FP64) ? (R)sv.sacc_d : (R)sv.sacc;
    for (int c = lane; c < nf; c += 32) {
        const size_t o = (size_t)c * ntau + s;
        sp[c] = A::mul(A::mul(solar, cs[o]), (R)sv.shadow[o]);
        po[c] = A::mul(alb, Efm[o]);
    }
    __syncwarp();
    bool more = true;
    int it = 0;
    while (more) {
        if (it == cap) {
            if (lane == 0) atomicOr(sv.status, ST_SCATTER_CAP);
            break;
        }
        for (int c = 0; c < nf; ++c) {
            const int d0 = sv.dep_ptr[c], d1 = sv.dep_ptr[c + 1];
            R val;
            if (d1 == d0) {
                val = po[c];
            } else {
                R after = R(0), before = R(0);
                for (int base = d0; base < d1; base += 32) {
                    const int k = base + lane;
                    R term = R(0);
                    int isafter = 0;
                    if (k < d1) {
                        const int g = __ldg(&sv.dep_idx[k]);
                        const R v = (R)__ldg(&sv.dep_vf[k]);
                        isafter = g > c;
                        term = A::mul(v, isafter ? po[g] : pn[g]);
                    }
                    const int n = min(32, d1 - base);
                    for (int j = 0; j < n; ++j) {
                        const R tj = __shfl_sync(0xffffffffu, term, j);
                        const int aj = __shfl_sync(0xffffffffu, isafter, j);
                        if (aj) after = A::add(after, tj);
                        else before = A::add(before, tj);
                    }
                }
                val = A::mul(alb, A::add(A::add(sp[c], after), before));
            }
            if (lane == 0) pn[c] = val;
            __syncwarp();
        }
        int test = 0;
        for (int c = lane; c < nf; c += 32) {
            const R d = A::sub(pn[c], po[c]);
            if ((d < R(0) ? -d : d) > acc) test = 1;
            po[c] = pn[c];
        }
        more = __any_sync(0xffffffffu, test) != 0;
        __syncwarp();
        ++it;
    }
    for (int c = lane; c < nf; c += 32) Efm[(size_t)c * ntau + s] = A::div(pn[c], alb);
}

// The same Gauss-Seidel sweeps in level order.  A facet needs this sweep's
// values of the lower facets it sees and the last sweep's of the higher ones,
// so facets whose lower neighbours are done can go together: the plan sorts
// them by level (one more than the highest level among the lower neighbours)
// and a CTA sweeps STEPS steps, STEPS lanes a facet, its values in shared
// memory.  Every facet's two sums run in list order as above (ascending lists:
// the lower neighbours are a row's first entries), so the results are the
// facet-by-facet kernel's bits.  Per sweep:
//   pre[c] = sp[c] + after[c] of every facet, from the last sweep's values
//   level by level, p[c] = alb (pre[c] + before[c]) in place
// A step stops at its own convergence; its lanes then keep their values.
// The facet-by-facet kernel was one warp per step with a chain of nf dependent
// sums: 26.7 ms for 5,440 facets and 720 steps (geometry, scattering and
// read-back 31.3 ms), against about 2 ms here (6.7 ms); bound by the list
// entries' loads and, where relief makes long level chains, by a barrier a
// level.
template <int MODE, int STEPS>
__global__ void __launch_bounds__(1024) k_multi_levels(DevSolve sv, GsPlan plan, void* work, int cap) {
    using A = Sa<MODE>;
    using R = typename A::R;
    extern __shared__ __align__(16) unsigned char dyn[];
    R* p = reinterpret_cast<R*>(dyn);  // [nf][STEPS]
    __shared__ int more[STEPS];
    constexpr int GROUPS = 1024 / STEPS;
    const int nf = sv.nf, ntau = sv.ntau;
    const int k = threadIdx.x % STEPS, grp = threadIdx.x / STEPS;
    const int s = blockIdx.x * STEPS + k;
    const bool valid = s < ntau;
    const int sc = valid ? s : ntau - 1;
    R* pre = static_cast<R*>(work) + (size_t)blockIdx.x * nf * STEPS;
    const R* cs = static_cast<const R*>(sv.cosil);
    R* Efm = static_cast<R*>(sv.Efm);
    const R solar = (MODE == MODE_FP64) ? (R)sv.solar_d : (R)sv.solar;
    const R alb = (MODE == MODE_FP64) ? (R)sv.alb_d : (R)sv.alb;
    const R acc = (MODE == MODE_FP64) ? (R)sv.sacc_d : (R)sv.sacc;
    // sum of entries [e0, e1) in order
    auto row = [&](int e0, int e1) {
        R t = R(0);
#pragma unroll 4
        for (int e = e0; e < e1; ++e)
            t = A::add(t, A::mul((R)__ldg(&sv.dep_vf[e]), p[__ldg(&sv.dep_idx[e]) * STEPS + k]));
        return t;
    };
    for (int c = grp; c < nf; c += GROUPS) p[c * STEPS + k] = A::mul(alb, Efm[(size_t)c * ntau + sc]);
    bool active = valid;
    __syncthreads();
    for (int it = 0;; ++it) {
        if (it == cap) {
            if (threadIdx.x == 0) atomicOr(sv.status, ST_SCATTER_CAP);
            break;
        }
        if (threadIdx.x < STEPS) more[threadIdx.x] = 0;
        for (int c = grp; c < nf; c += GROUPS) {
            const int m = plan.mid[c], e1 = sv.dep_ptr[c + 1];
            if (sv.dep_ptr[c] == e1) continue;
            const size_t o = (size_t)c * ntau + sc;
            const R sp = A::mul(A::mul(solar, cs[o]), (R)sv.shadow[o]);
            pre[(size_t)c * STEPS + k] = A::add(sp, row(m, e1));
        }
        __syncthreads();
        bool moved = false;
        int lo = 0;
        for (int l = 0; l < plan.levels; ++l) {
            const int hi = plan.off[l + 1];
            for (int q = lo + grp; q < hi; q += GROUPS) {
                const int4 r = plan.rows[q];  // facet, its lower neighbours' entries
                const R x = pre[(size_t)r.x * STEPS + k];
                const R val = A::mul(alb, A::add(x, row(r.y, r.z)));
                R* d = &p[r.x * STEPS + k];
                const R diff = A::sub(val, *d);
                moved = moved || (diff < R(0) ? -diff : diff) > acc;
                if (active) *d = val;
            }
            lo = hi;
            __syncthreads();
        }
        if (active && moved) more[k] = 1;
        __syncthreads();
        active = active && more[k] != 0;
        if (!__syncthreads_or(active)) break;
    }
    if (valid)
        for (int c = grp; c < nf; c += GROUPS) Efm[(size_t)c * ntau + s] = A::div(p[c * STEPS + k], alb);
}

// one Jacobi sweep: pn = alb (sp + sum_k v_k po[g_k]) for every (facet, step),
// rows of gather_ld(ntau); *more = 1 if some |pn - po| > accuracy.  sp = solar x
// the lit cosine; the list's sum is two fused partial sums over every other entry.
template <int N>
__global__ void __launch_bounds__(256) k_multi_jacobi(DevSolve sv, const float* lit, const float* po, float* pn,
                                                      int* more) {
    const int f = (gridDim.y - 1 - blockIdx.y) * blockDim.y + threadIdx.y;
    if (f >= sv.nf) return;  // warp-uniform
    const int ld = gather_ld(sv.ntau), s = (blockIdx.x * 32 + threadIdx.x) * N;
    const bool ok = s < sv.ntau;
    const size_t at = ok ? s : 0;
    float a0[N] = {}, a1[N] = {}, old[N], sp[N];
    gather<float, N>(sv.dep_idx, sv.dep_vf, sv.dep_ptr[f], sv.dep_ptr[f + 1], po + at, ld, [](float v) { return v; },
                  [&](int i, float c, const float(&x)[N]) {
#pragma unroll
                      for (int u = 0; u < N; ++u) {
                          if (i & 1) a1[u] = __fmaf_rn(c, x[u], a1[u]);
                          else a0[u] = __fmaf_rn(c, x[u], a0[u]);
                      }
                  });
    if (!ok) return;
    const size_t o = (size_t)f * ld + at;
    Steps<float, N>::get(po + o, old);
    Steps<float, N>::get(lit + o, sp);
    bool moved = false;
    float v[N];
#pragma unroll
    for (int u = 0; u < N; ++u) {
        v[u] = sv.alb * __fadd_rn(__fmul_rn(sv.solar, sp[u]), a0[u] + a1[u]);  // the sunlight is a rounded term
        moved = moved || (s + u < sv.ntau && fabsf(v[u] - old[u]) > sv.sacc);
    }
    Steps<float, N>::put(pn + o, v);
    if (moved) *more = 1;
}

__global__ void k_status_or(int* status, int bits) { atomicOr(status, bits); }

__global__ void __launch_bounds__(256) k_multi_jacobi_out(DevSolve sv, const float* p) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)sv.nf * sv.ntau) return;
    const int f = (int)(i / sv.ntau), s = (int)(i % sv.ntau);
    static_cast<float*>(sv.Efm)[i] = p[(size_t)f * gather_ld(sv.ntau) + s] / sv.alb;
}

// [nf][ntau] -> [ntau][nf]
template <class R>
__global__ void __launch_bounds__(256) k_forcing_t(const R* src, R* dst, int nf, int ntau) {
    __shared__ R sm[32][33];
    const int f0 = blockIdx.y * 32, s0 = blockIdx.x * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int f = f0 + j, s = s0 + threadIdx.x;
        sm[j][threadIdx.x] = (f < nf && s < ntau) ? src[(size_t)f * ntau + s] : R(0);
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int s = s0 + j, f = f0 + threadIdx.x;
        if (f < nf && s < ntau) dst[(size_t)s * nf + f] = sm[threadIdx.x][j];
    }
}

// [rows][cols] -> [cols][rows] with a type conversion, 32 x 32 tiles
template <class Ri, class Ro>
__global__ void __launch_bounds__(256) k_transpose(const Ri* src, Ro* dst, size_t rows, size_t cols) {
    __shared__ Ri sm[32][33];
    const size_t r0 = (size_t)blockIdx.y * 32, c0 = (size_t)blockIdx.x * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const size_t r = r0 + j, c = c0 + threadIdx.x;
        sm[j][threadIdx.x] = (r < rows && c < cols) ? src[r * cols + c] : Ri(0);
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const size_t c = c0 + j, r = r0 + threadIdx.x;
        if (r < rows && c < cols) dst[c * rows + r] = (Ro)sm[threadIdx.x][j];
    }
}

// flags [nf][ntau] as the 32-bit words of the host interface, four at a time
__global__ void __launch_bounds__(256) k_widen_flags(const uint8_t* src, int32_t* dst, size_t n) {
    const size_t i = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (i + 4 <= n) {
        const uchar4 v = *reinterpret_cast<const uchar4*>(src + i);
        *reinterpret_cast<int4*>(dst + i) = make_int4(v.x, v.y, v.z, v.w);
    } else {
        for (size_t j = i; j < n; ++j) dst[j] = src[j];
    }
}

template <class R>
__global__ void k_set_forcing(DevSolve sv, const int32_t* shadow, const float* illum) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)sv.nf * sv.ntau;
    if (i >= n) return;
    sv.shadow[i] = shadow[i] ? 1 : 0;
    static_cast<R*>(sv.Efm)[i] = (R)illum[i];
}

// ------------------------------------------------------------------ launchers
namespace {
size_t rows_words(const DevSolve& s) { return (size_t)s.nf * gather_ld(s.ntau); }

dim3 rows_grid(const DevSolve& s, int steps) { return dim3((s.ntau + 32 * steps - 1) / (32 * steps), (s.nf + 7) / 8); }

bool wide_rows(const DevSolve& s, int wide) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return true;
    return gather_wide((long long)((s.nf + 31) / 32) * ((s.ntau + 31) / 32), wide, sms);
}

template <int MODE>
void launch_single(const DevSolve& s, void* work, bool multiple, cudaStream_t st) {
    using R = typename Sa<MODE>::R;
    R* lit = static_cast<R*>(work);
    if (!lit) {
        k_single_scatter<MODE><<<dim3((s.ntau + 31) / 32, (s.nf + 7) / 8), dim3(32, 8), 0, st>>>(s);
        return;
    }
    const size_t n = rows_words(s);
    R* next = MODE == MODE_FAST && multiple ? lit + n : nullptr;
    const dim3 blk(32, 8);
    k_lit_cosine<R><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s, lit);
    if (wide_rows(s, kWide<R>)) k_single_rows<MODE, kWide<R>><<<rows_grid(s, kWide<R>), blk, 0, st>>>(s, lit, next);
    else k_single_rows<MODE, 1><<<rows_grid(s, 1), blk, 0, st>>>(s, lit, next);
}
}  // namespace

// work: scattering_work_bytes, kept for launch_multiple_scattering (null for single
// scattering alone where there is no room for it)
int launch_single_scattering(const DevSolve& s, void* work, bool multiple, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    switch (s.mode) {
        case MODE_REF: launch_single<MODE_REF>(s, work, multiple, st); break;
        case MODE_FP64: launch_single<MODE_FP64>(s, work, multiple, st); break;
        default: launch_single<MODE_FAST>(s, work, multiple, st); break;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

size_t scattering_work_bytes(const DevSolve& s, bool multiple) {
    const size_t rs = (s.mode == MODE_FP64) ? 8 : 4;
    // the lit cosines; then FAST's two iterates, or the Gauss-Seidel sweeps'
    // three arrays or one of whole 8-step chunks (k_multi_levels), over them
    const size_t rows = rows_words(s) * rs;
    if (!multiple) return rows;
    if (s.mode == MODE_FAST) return 3 * rows + 256;
    return std::max(rows, std::max<size_t>(3 * (size_t)s.ntau, (size_t)s.ntau + 8) * s.nf * rs) + 256;
}

namespace {
// FAST: Jacobi sweeps until no (facet, step) changes by more than the
// accuracy; one 4-byte read-back per sweep
int multiple_scattering_jacobi(const DevSolve& s, void* work, cudaStream_t st, int cap) {
    const size_t n = rows_words(s);
    const float* lit = static_cast<float*>(work);
    float* pa = static_cast<float*>(work) + n;  // the first iterate (k_single_rows)
    float* pb = pa + n;
    int* more = reinterpret_cast<int*>(pb + n);
    const dim3 blk(32, 8);
    const bool wide = wide_rows(s, kWide<float>);
    for (int it = 0;; ++it) {
        if (it == cap) {
            k_status_or<<<1, 1, 0, st>>>(s.status, ST_SCATTER_CAP);
            break;
        }
        cudaMemsetAsync(more, 0, 4, st);
        if (wide) k_multi_jacobi<4><<<rows_grid(s, 4), blk, 0, st>>>(s, lit, pa, pb, more);
        else k_multi_jacobi<1><<<rows_grid(s, 1), blk, 0, st>>>(s, lit, pa, pb, more);
        int m = 0;
        if (cudaMemcpyAsync(&m, more, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess) return 2;
        if (cudaStreamSynchronize(st) != cudaSuccess) return 2;
        std::swap(pa, pb);
        if (!m) break;
    }
    k_multi_jacobi_out<<<(unsigned)(((size_t)s.nf * s.ntau + 255) / 256), 256, 0, st>>>(s, pa);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
}  // namespace

namespace {
// -1: not launched, the facet-by-facet kernel is faster
template <int MODE, int STEPS>
int launch_levels(const DevSolve& s, const GsPlan& plan, void* work, cudaStream_t st, int cap) {
    const auto kernel = k_multi_levels<MODE, STEPS>;
    const size_t smem = (size_t)s.nf * STEPS * sizeof(typename Sa<MODE>::R);
    // the limit belongs to the function, not to the launch: every thread sets the
    // same one, or a small shape's would refuse a large one's launch
    int dev = 0, sms = 0, per = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGsSharedBytes) != cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 1024, smem) != cudaSuccess || per < 1)
        return 2;
    // A level costs a barrier in every wave of CTAs, a facet of the other kernel a
    // warp's turn, and they cost about the same: lists that chain facet to facet go
    // facet by facet.  ms by levels and by facets, 720 steps, 2 neighbours either
    // side of a facet: 5,440 facets (one wave) 9.9 and 8.6 in 5,440 levels, 6.0 and
    // 8.6 in 2,720; 12,000 (two waves) 37 and 20 in 12,000, 22 and 20 in 6,000;
    // 20,480 (three) 98 and 36 in 20,480, 53 and 36 in 10,240; 16 neighbours,
    // 20,480 facets 54 and 53 in 6,826, 36 and 54 in 5,120.
    const long long grid = (s.ntau + STEPS - 1) / STEPS, waves = (grid + (long long)sms * per - 1) / ((long long)sms * per);
    if (6 * waves * plan.levels > 5ll * plan.listed) return -1;
    kernel<<<(unsigned)grid, 1024, smem, st>>>(s, plan, work, cap);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
// as many steps a CTA (lanes a facet) as their values fit shared memory
template <int MODE>
int launch_gauss_seidel(const DevSolve& s, const GsPlan& plan, void* work, cudaStream_t st, int cap) {
    const size_t most = kGsSharedBytes / sizeof(typename Sa<MODE>::R) / (size_t)s.nf;
    int rc = -1;
    if (plan.rows && most >= 8) rc = launch_levels<MODE, 8>(s, plan, work, st, cap);
    else if (plan.rows && most >= 4) rc = launch_levels<MODE, 4>(s, plan, work, st, cap);
    else if (plan.rows && most >= 2) rc = launch_levels<MODE, 2>(s, plan, work, st, cap);
    else if (plan.rows && most >= 1) rc = launch_levels<MODE, 1>(s, plan, work, st, cap);
    if (rc >= 0) return rc;
    k_multi_gs<MODE><<<s.ntau, 32, 0, st>>>(s, work, cap);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
}  // namespace

int launch_multiple_scattering(const DevSolve& s, const GsPlan& plan, void* work, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    const int cap = 1000;  // the reference iterates unbounded; real cases need < 50 sweeps
    if (s.mode == MODE_FAST) return multiple_scattering_jacobi(s, work, st, cap);
    if (s.mode == MODE_FP64) return launch_gauss_seidel<MODE_FP64>(s, plan, work, st, cap);
    return launch_gauss_seidel<MODE_REF>(s, plan, work, st, cap);
}

int launch_forcing_transpose(const DevSolve& s, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    dim3 blk(32, 8), grd((s.ntau + 31) / 32, (s.nf + 31) / 32);
    if (s.mode == MODE_FP64)
        k_forcing_t<double><<<grd, blk, 0, st>>>(static_cast<const double*>(s.Efm), static_cast<double*>(s.E), s.nf, s.ntau);
    else
        k_forcing_t<float><<<grd, blk, 0, st>>>(static_cast<const float*>(s.Efm), static_cast<float*>(s.E), s.nf, s.ntau);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_transpose(const void* src, int src_bytes, void* dst, int dst_bytes, size_t rows, size_t cols,
                     stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    dim3 blk(32, 8), grd((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32));
    if (src_bytes == 4 && dst_bytes == 4)
        k_transpose<float, float><<<grd, blk, 0, st>>>(static_cast<const float*>(src), static_cast<float*>(dst), rows, cols);
    else if (src_bytes == 8 && dst_bytes == 8)
        k_transpose<double, double><<<grd, blk, 0, st>>>(static_cast<const double*>(src), static_cast<double*>(dst), rows, cols);
    else if (src_bytes == 4 && dst_bytes == 8)
        k_transpose<float, double><<<grd, blk, 0, st>>>(static_cast<const float*>(src), static_cast<double*>(dst), rows, cols);
    else if (src_bytes == 8 && dst_bytes == 4)
        k_transpose<double, float><<<grd, blk, 0, st>>>(static_cast<const double*>(src), static_cast<float*>(dst), rows, cols);
    else
        return 1;
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_widen_flags(const uint8_t* src, int32_t* dst, size_t n, stream_t stv) {
    k_widen_flags<<<(unsigned)((n / 4 + 256) / 256), 256, 0, static_cast<cudaStream_t>(stv)>>>(src, dst, n);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_set_forcing(const DevSolve& s, const int32_t* shadow_d, const float* illum_d, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    const size_t n = (size_t)s.nf * s.ntau;
    const int g = (int)((n + 255) / 256);
    if (s.mode == MODE_FP64) k_set_forcing<double><<<g, 256, 0, st>>>(s, shadow_d, illum_d);
    else k_set_forcing<float><<<g, 256, 0, st>>>(s, shadow_d, illum_d);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}


// --------------------------------------------------------- no-allocation variant
// Scattered sunlight over caller-owned device buffers for callers that cannot
// allocate device memory themselves or through this library: code running
// where cudaMalloc is unavailable or forbidden (inside a framework that owns
// every device allocation through its own pool, or a host loop that must not
// trigger allocator synchronisation).  The Gauss-Seidel work arrays live in a
// fixed file-scope device array instead of a per-call allocation.
//
//  * Limit: nf * ntau <= ATPM_NOALLOC_MAX_CELLS (2^20 cells, 12 MiB of
//    scratch); larger problems are rejected with ATPM_E_UNSUPPORTED.  Every
//    GPU that loads the library reserves this array until the process exits.
//  * The first call on a device looks up the array's device address with
//    cudaGetSymbolAddress, with that device current; make that first call
//    before any stream capture on the device.
//  * All calls share the one array: calls whose work overlaps on the GPU
//    (different streams, or different host threads) race and corrupt each
//    other's results.  Serialise them.
//  * The array keeps the previous call's contents; every cell a call reads is
//    written by that call first (the status word is cleared by each call).
namespace {
constexpr size_t kNoAllocMaxCells = size_t(1) << 20;
constexpr size_t kNoAllocStatusSlot = 3 * kNoAllocMaxCells;  // one int after the three arrays
constexpr int kNoAllocMaxFacets = 8 * 65535;  // grid.y of the single-scattering launch is nf / 8
static __device__ __align__(256) float g_noalloc_scratch[3 * kNoAllocMaxCells + 64];

std::mutex g_noalloc_mu;
void* g_noalloc_addr[256] = {};  // per-device address of g_noalloc_scratch

int noalloc_scratch(void** out, int* device, char* err, size_t errlen) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        std::snprintf(err, errlen, "cudaGetDevice: %s", cudaGetErrorString(e));
        return 1;
    }
    if (dev < 0 || dev >= 256) {
        std::snprintf(err, errlen, "device ordinal %d out of range", dev);
        return 1;
    }
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            std::snprintf(err, errlen, "cudaGetSymbolAddress(scratch): %s", cudaGetErrorString(e));
            return 1;
        }
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    *device = dev;
    return 0;
}
}  // namespace

void set_last_error(const char* msg);

}  // namespace atpm

extern "C" ATPM_API atpm_status atpm_scattering_noalloc(
    int32_t nf, int32_t ntau, const int32_t* dep_ptr, const int32_t* dep_idx, const float* dep_vf,
    const float* cosillum, const uint8_t* shadow, float solar, float albedo, float scattering_accuracy,
    int32_t multiple, float* illumination, int32_t* status, void* stream) {
    using namespace atpm;
    char err[256];
    if (nf < 1 || ntau < 1 || !dep_ptr || !dep_idx || !dep_vf || !cosillum || !shadow || !illumination) {
        set_last_error("scattering_noalloc: bad arguments (every array, dep_idx and dep_vf included, must be a "
                       "device pointer)");
        return ATPM_E_INVALID;
    }
    if (multiple && !status) {
        set_last_error("scattering_noalloc: multiple scattering needs a status word (the Gauss-Seidel cap is "
                       "reported there)");
        return ATPM_E_INVALID;
    }
    if (nf > kNoAllocMaxFacets) {
        std::snprintf(err, sizeof err, "scattering_noalloc: nf = %d exceeds %d facets (launch grid limit)", nf,
                      kNoAllocMaxFacets);
        set_last_error(err);
        return ATPM_E_UNSUPPORTED;
    }
    if ((size_t)nf * (size_t)ntau > kNoAllocMaxCells) {
        std::snprintf(err, sizeof err,
                      "scattering_noalloc: nf*ntau = %lld exceeds the fixed scratch of %lld cells; "
                      "use atpm_scattering",
                      (long long)nf * ntau, (long long)kNoAllocMaxCells);
        set_last_error(err);
        return ATPM_E_UNSUPPORTED;
    }
    void* scratch = nullptr;
    int dev = 0;
    if (noalloc_scratch(&scratch, &dev, err, sizeof err)) {
        set_last_error(err);
        return ATPM_E_CUDA;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int* st_word = status ? status : reinterpret_cast<int*>(static_cast<float*>(scratch) + kNoAllocStatusSlot);
    if (!status) {
        cudaError_t e = cudaMemsetAsync(st_word, 0, sizeof(int), st);
        if (e != cudaSuccess) {
            std::snprintf(err, sizeof err, "scattering_noalloc: %s", cudaGetErrorString(e));
            set_last_error(err);
            return ATPM_E_CUDA;
        }
    }
    DevSolve sv{};
    sv.nf = nf;
    sv.ntau = ntau;
    sv.mode = MODE_REF;
    sv.dep_ptr = dep_ptr;
    sv.dep_idx = dep_idx;
    sv.dep_vf = dep_vf;
    sv.nnz = 0;
    sv.shadow = const_cast<uint8_t*>(shadow);
    sv.cosil = const_cast<float*>(cosillum);
    sv.Efm = illumination;
    sv.status = st_word;
    sv.solar = solar;
    sv.alb = albedo;
    sv.sacc = scattering_accuracy;
    dim3 blk(32, 8), grd((ntau + 31) / 32, (nf + 7) / 8);
    k_single_scatter<MODE_REF><<<grd, blk, 0, st>>>(sv);
    if (multiple) k_multi_gs<MODE_REF><<<ntau, 32, 0, st>>>(sv, scratch, 1000);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        std::snprintf(err, sizeof err, "scattering_noalloc launch: %s", cudaGetErrorString(e));
        set_last_error(err);
        return ATPM_E_CUDA;
    }
    return ATPM_OK;
}
