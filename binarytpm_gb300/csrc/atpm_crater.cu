// Crater (surface roughness) module: the kernels of the reference's Thermal
// GPU module (3905/Thermal/NominalPole/GPU_code.cu:152-594), rebuilt for
// GB300 with runtime sizes.
//
// Every facet carries a hemispherical crater of nsf (= 100) sub-facets.  The
// reference launches one kernel per time step (2 x NTAU launches and
// synchronisations per revolution, GPU_code.cu:982-998).  Here:
//
//   k_crater_shadow      sfcpartialshadow (152-210): 10x10 sub-points of each
//                        sub-facet against the analytic crater rim, every
//                        (facet, step) in one launch
//   k_crater_scatter     roughness_single/multiple_scattering (216-304):
//                        one block per batch of a facet's steps, the 100x100
//                        crater view-factor matrix staged in shared memory
//   k_crater_revolution  finite_difference + boundary_condition (377-490)
//                        for a whole revolution in ONE launch: a block owns a
//                        facet, a thread owns a sub-facet's depth column in
//                        registers; the crater self-heating sum reads the
//                        other sub-facets' previous-revolution temperatures
//                        through shared memory
//   k_crater_equilibrium roughness_inst_equilibrium (496-548)
//   k_crater_converged   converged (554-594)
//
// REFERENCE precision evaluates every float expression in the GPU module's
// operand order without contraction, with this host's libm powf for x^4 and
// x^0.25 (the exception tables of atpm_powtab.cpp); it is bit-identical to
// the CPU restatement of the module the reference driver links for GPU-free
// runs.  FAST precision contracts and reorders.
#include <cuda_runtime.h>

#include "atpm_crater_rim.cuh"
#include "atpm_internal.h"

namespace atpm {

namespace {

__device__ __forceinline__ float cpow4_exact(const PowTab& t, float x, int* st) {
    // x^4 corrected to this host's libm powf (atpm_powtab.cpp)
    return libm_pow4(t, x, st);
}

template <int MODE>
__device__ __forceinline__ float cpow4(const PowTab& t, float x, int* st) {
    if constexpr (MODE == MODE_REF) return cpow4_exact(t, x, st);
    else { const float x2 = x * x; return x2 * x2; }
}

}  // namespace

// sfcpartialshadow: a block takes kRimDirs consecutive (facet, step) Sun
// directions at a time, a thread one sub-facet in all of them.  A sub-facet
// that is dark already has nothing to lose and is skipped.  Bound by
// instruction issue; one direction at a time, with its square root for every
// point, 160 facets x 360 steps took 665 us in REFERENCE, now 298; 200 x 720 in
// FAST 1,105 and 660.
template <int MODE>
__global__ void __launch_bounds__(128) k_crater_shadow(CraterDev c) {
    using A = Ca<MODE>;
    __shared__ RimShared r;
    __shared__ float dir[2][kRimDirs][3];  // direction and slope
    __shared__ int lit[2][kRimDirs];
    const int nsf = c.nsf, j = threadIdx.x;
    const long long n = (long long)c.nf * c.ntau;
    rim_open<MODE>(r, c);
    Rim<MODE> rim;
    if (j < nsf) rim.load(c, r, j);
    int turn = 0;
    for (long long fs0 = (long long)blockIdx.x * kRimDirs; fs0 < n; fs0 += (long long)gridDim.x * kRimDirs, turn ^= 1) {
        if (threadIdx.x < kRimDirs) {
            const long long fs = fs0 + threadIdx.x;
            const bool use = fs < n && c.shadow[fs] == 1;
            lit[turn][threadIdx.x] = use;
            if (use) {
                const float* iv = c.illumvec + 3 * fs;
                // sun vector normalised by its x-y length (GPU_code.cu:177-181)
                const float s = A::sqrt_(A::add(A::mul(iv[0], iv[0]), A::mul(iv[1], iv[1])));
                const float sv0 = A::div(iv[0], s), sv1 = A::div(iv[1], s), sv2 = A::div(iv[2], s);
                dir[turn][threadIdx.x][0] = sv0;
                dir[turn][threadIdx.x][1] = sv1;
                dir[turn][threadIdx.x][2] = A::div(fabsf(sv2), A::sqrt_(A::add(A::mul(sv0, sv0), A::mul(sv1, sv1))));
            }
        }
        __syncthreads();  // the other turn's directions are overwritten only after the next one
        if (j >= nsf) continue;
        float sh[kRimDirs], w0[kRimDirs], w1[kRimDirs], a[kRimDirs];
        bool any = false;
#pragma unroll
        for (int d = 0; d < kRimDirs; ++d) {
            const bool use = lit[turn][d];
            sh[d] = use ? c.sfc_shadow[(fs0 + d) * nsf + j] : 0.0f;
            any = any || sh[d] != 0.0f;
            w0[d] = use ? dir[turn][d][0] : 0.0f;
            w1[d] = use ? dir[turn][d][1] : 0.0f;
            a[d] = use ? dir[turn][d][2] : 1.0f;
        }
        if (!any) continue;
        int m[kRimDirs];
        rim.count(r, w0, w1, a, m);
#pragma unroll
        for (int d = 0; d < kRimDirs; ++d)
            if (sh[d] != 0.0f)
                c.sfc_shadow[(fs0 + d) * nsf + j] = sh[d] == 1.0f ? r.left[m[d]] : rim_take<MODE>(sh[d], m[d]);
    }
}

// single (multiple == 0) or single + Jacobi multiple scattering of kScatSteps
// steps of a facet per block iteration: a view factor is read once for all of
// them, and two barriers an iteration serve them all.  A step that has
// converged keeps its values while the others go on.  Bound by shared-memory
// reads; one step at a time 160 facets x 360 steps took 495 us in REFERENCE, now
// 307; 200 x 720 in FAST 1,164 and 607.
constexpr int kScatSteps = 4;

template <int MODE>
__global__ void __launch_bounds__(128) k_crater_scatter(CraterDev c, float solar, float acc, int multiple, int cap) {
    using A = Ca<MODE>;
    extern __shared__ __align__(16) float sm[];
    const int nsf = c.nsf;
    float4* vals = reinterpret_cast<float4*>(sm);  // nsf: illumination, then the last iterate, of the four steps
    float* Vs = sm + 4 * nsf;                      // nsf * nsf
    __shared__ int more[2];
    for (int k = threadIdx.x; k < nsf * nsf; k += blockDim.x) Vs[k] = c.V[k];
    if (threadIdx.x < 2) more[threadIdx.x] = 0;
    const int per = (c.ntau + kScatSteps - 1) / kScatSteps;
    const long long n = (long long)c.nf * per;
    const int j = threadIdx.x;
    for (long long g = blockIdx.x; g < n; g += gridDim.x) {
        const int f = (int)(g / per), s0 = (int)(g % per) * kScatSteps, ns = min(kScatSteps, c.ntau - s0);
        const float alb = c.albedo[f];
        const size_t o = ((size_t)f * c.ntau + s0) * nsf + j;
        float power[kScatSteps], tot[kScatSteps], w[kScatSteps];
#pragma unroll
        for (int d = 0; d < kScatSteps; ++d) {
            power[d] = tot[d] = 0.0f;
            if (j < nsf && d < ns) {
                const size_t od = o + (size_t)d * nsf;
                const float sh = c.sfc_shadow[od], ia = c.illumangle[od], gi = c.RGI[od];
                tot[d] = A::add(A::mul(A::mul(solar, sh), ia), gi);
                power[d] = A::add(A::mul(A::mul(solar, ia), sh), gi);
            }
        }
        __syncthreads();  // the last steps' values are read
        if (j < nsf) vals[j] = make_float4(tot[0], tot[1], tot[2], tot[3]);
        __syncthreads();
        auto terms = [&](int i, float v) {
            const float4 x = vals[i];
            w[0] = A::mul(v, x.x);
            w[1] = A::mul(v, x.y);
            w[2] = A::mul(v, x.z);
            w[3] = A::mul(v, x.w);
        };
        if (j < nsf) {
#pragma unroll 4
            for (int i = 0; i < nsf; ++i) {
                terms(i, A::mul(Vs[i * nsf + j], alb));
#pragma unroll
                for (int d = 0; d < kScatSteps; ++d) tot[d] = A::add(tot[d], w[d]);
            }
#pragma unroll
            for (int d = 0; d < kScatSteps; ++d)
                if (tot[d] <= 0.0f) tot[d] = 0.0f;
        }
        if (multiple) {
            float old[kScatSteps], next[kScatSteps] = {};
            __syncthreads();
#pragma unroll
            for (int d = 0; d < kScatSteps; ++d) old[d] = A::mul(alb, tot[d]);
            if (j < nsf) vals[j] = make_float4(old[0], old[1], old[2], old[3]);
            __syncthreads();
            int going = (1 << ns) - 1;  // uniform: steps that have not converged
            for (int it = 0; it < cap; ++it) {
                float sum[kScatSteps] = {};
                if (j < nsf) {
#pragma unroll 4
                    for (int i = 0; i < nsf; ++i) {
                        terms(i, Vs[i * nsf + j]);
#pragma unroll
                        for (int d = 0; d < kScatSteps; ++d) sum[d] = A::add(sum[d], w[d]);
                    }
                }
                __syncthreads();  // the iterate and the last flags are read
                int moved = 0;
                if (j < nsf) {
#pragma unroll
                    for (int d = 0; d < kScatSteps; ++d)
                        if ((going >> d) & 1) {
                            next[d] = A::mul(alb, A::add(power[d], sum[d]));
                            if (fabsf(A::sub(next[d], old[d])) > acc) moved |= 1 << d;
                            old[d] = next[d];
                        }
                    vals[j] = make_float4(old[0], old[1], old[2], old[3]);
                }
                moved = __reduce_or_sync(0xffffffffu, moved);
                if ((threadIdx.x & 31) == 0 && moved) atomicOr(&more[it & 1], moved);
                if (threadIdx.x == 0) more[(it + 1) & 1] = 0;
                __syncthreads();
                going = more[it & 1];
                if (!going) break;
                if (it + 1 == cap && threadIdx.x == 0) atomicOr(c.status, ST_SCATTER_CAP);
            }
#pragma unroll
            for (int d = 0; d < kScatSteps; ++d) tot[d] = A::div(next[d], alb);
            __syncthreads();
            if (threadIdx.x < 2) more[threadIdx.x] = 0;  // the next steps begin with the flags of iteration 0
        }
        if (j < nsf)
#pragma unroll
            for (int d = 0; d < kScatSteps; ++d)
                if (d < ns) c.RI[o + (size_t)d * nsf] = tot[d];
    }
}

// steps whose crater sums are formed together
constexpr int kBatch = 8;

// acc[k] += V[i][j] x w[i][k] over i = i0, i0 + step, ... < n, in order, on the
// packed FP32 instructions (two steps an instruction), each lane rounded as the
// scalar operations
template <int MODE>
__device__ __forceinline__ void add_view(float2 (&acc)[kBatch / 2], const float* V, const float* w, int nsf, int j,
                                         int i0, int step, int n) {
#pragma unroll 5
    for (int i = i0; i < n; i += step) {
        const float v = __ldg(V + i * nsf + j);
        const float4 lo = *reinterpret_cast<const float4*>(w + i * kBatch);
        const float4 hi = *reinterpret_cast<const float4*>(w + i * kBatch + 4);
        const float2 x[kBatch / 2] = {make_float2(lo.x, lo.y), make_float2(lo.z, lo.w), make_float2(hi.x, hi.y),
                                      make_float2(hi.z, hi.w)};
        const float2 vv = make_float2(v, v);
#pragma unroll
        for (int k = 0; k < kBatch / 2; ++k) {
            if constexpr (MODE == MODE_REF) {
                // scalar additions: ptxas may fuse a packed product and sum
                const float2 q = __fmul2_rn(x[k], vv);
                acc[k] = make_float2(__fadd_rn(acc[k].x, q.x), __fadd_rn(acc[k].y, q.y));
            } else {
                acc[k] = __ffma2_rn(x[k], vv, acc[k]);
            }
        }
    }
}

__device__ __forceinline__ void copy_word(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// one revolution of finite_difference + boundary_condition for every step:
// block = one facet, thread j = sub-facet j (its depth column in registers).
// The crater's mutual heating of a step needs only the previous revolution's
// temperatures, so it is summed for kBatch steps at a time: a view factor then
// serves kBatch multiply-adds and the steps between two barriers (one a batch)
// are independent per thread.  The next batch's forcing arrives by cp.async
// while this batch's steps run.  The view factors are read through L1, which
// all CTAs of an SM share: shared memory then leaves room for as many CTAs as
// the registers do.
//
// A facet's revolution is long, so a last wave of few facets would cost as
// much as a full one.  With more facets than resident CTAs the steps are
// therefore dealt out in kSegments pieces (take_piece): a CTA takes the next
// (segment, facet) ticket, and the facet's column waits in memory between its
// segments.  A segment's predecessor was taken a whole grid of tickets
// earlier by a CTA that is running or done, so the wait for it always ends
// (it is bounded all the same).
//
// With one step at a time and the matrix in shared memory the kernel was bound
// by shared memory (125 reads for 100 multiply-adds a step) and, in REFERENCE
// precision, by the one chain of 100 additions.  Now it is bound by instruction
// issue (470 a sub-facet step) and, for few facets, by a step's latency.  ms a
// revolution, before and after (720 steps): FAST, NX 48: 0.92 and 0.56 at 152
// facets, 1.50 and 1.03 at 608, 1.78 and 1.15 at 640 (1.85 without the
// segments), 2.92 and 2.07 at 1,216; REFERENCE, NX 48, 200 facets: 1.76 and
// 0.88.
constexpr int kSegments = 8;
constexpr long long kPieceWait = 2000000000LL;  // clock cycles (about a second)

// the next piece of work: facet and first step in f, s0; false when none is
// left.  Uniform over the block.  `work`: [nf] segments done, then the ticket.
__device__ __forceinline__ bool take_piece(const CraterDev& c, int* work, int segs, int len, int& f, int& s0,
                                           int& piece) {
    __shared__ int next;
    for (;;) {
        __syncthreads();  // the last piece is done with shared memory
        if (threadIdx.x == 0) {
            int t = atomicAdd(&work[c.nf], 1);
            if (t >= segs * c.nf) t = -1;
            else if (t >= c.nf && t / c.nf * len < c.ntau && !c.conv[t % c.nf]) {
                const volatile int* done = &work[t % c.nf];
                const long long begin = clock64();
                while (*done < t / c.nf) {
                    __nanosleep(200);
                    if (clock64() - begin > kPieceWait) {
                        atomicOr(c.status, ST_TC_TIMEOUT);
                        t = -1;
                        break;
                    }
                }
                __threadfence();
            }
            next = t;
        }
        __syncthreads();
        const int t = next;
        if (t < 0) return false;
        f = t % c.nf;
        piece = t / c.nf;
        s0 = piece * len;
        if (!c.conv[f] && s0 < c.ntau) return true;
    }
}

// RESIDENT: CTAs an SM holds (the register allocator's bound): 4, or 2 where no
// SM gets more than two facets (200 facets, NX 56: 0.73 against 0.85 ms)
template <int MODE, int NX, int RESIDENT>
__global__ void __launch_bounds__(128, RESIDENT)
    k_crater_revolution(CraterDev c, PowTab p4, float es, float es4, float m0, float dz, float tacc, float tacc2,
                        int* work, int segs) {
    using A = Ca<MODE>;
    __shared__ float stage[2][3][kBatch][128];               // previous temperature, heating, illumination -> flux
    __shared__ __align__(16) float W[2][128 * kBatch];       // eps sigma T_prev^4 of the batch's steps
    const int nsf = c.nsf, ntau = c.ntau;
    const int len = (ntau + segs * kBatch - 1) / (segs * kBatch) * kBatch;  // steps of a segment
    int f = blockIdx.x, first = 0, piece = 0;
    while (segs > 1 ? take_piece(c, work, segs, len, f, first, piece) : piece++ == 0 && !c.conv[f]) {
        const int end = min(ntau, first + len);
        const int j = threadIdx.x;
        const bool act = j < nsf;
        const float alb = c.albedo[f];
        // the facet body's revolutions per model period scale the time step and
        // the skin factor (175706/Run-04/thermal_GPU.cu:448-450, 539); with none
        // given the expressions are the synchronous module's (GPU_code.cu:392-393)
        const float w2pi = c.numrevs ? A::mul(A::mul(2.0f, c.PI), c.numrevs[f]) : A::mul(2.0f, c.PI);
        const float m0f = c.numrevs ? A::div(A::div(w2pi, (float)ntau), A::mul(dz, dz)) : m0;
        const float m1 = A::div(A::mul(c.ti[f], A::sqrt_(A::div(w2pi, c.rot_period))), dz);
        const float esw = A::mul(c.ir_abs, es);  // IR_ABS * EPSSIGMA (thermal_GPU.cu:521): es when ir_abs = 1
        const float oma = A::sub(1.0f, alb);
        float T[NX + 1];
        float* tp = c.temp + (size_t)f * (NX + 1) * nsf;
#pragma unroll
        for (int i = 0; i <= NX; ++i) T[i] = act ? __ldcg(tp + (size_t)i * nsf + j) : 0.0f;
        bool hot = false;
        int flags = 0;
        const size_t base = (size_t)f * ntau * nsf + j;
        const float* V = c.V;
        // a thread copies and reads its own words only
        auto fetch = [&](int s0, int buf) {
            if (act)
                for (int k = 0; k < kBatch && s0 + k < end; ++k) {
                    const size_t o = base + (size_t)(s0 + k) * nsf;
                    copy_word(&stage[buf][0][k][j], c.stemp1 + o);
                    copy_word(&stage[buf][1][k][j], c.RGH + o);
                    copy_word(&stage[buf][2][k][j], c.RI + o);
                }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        fetch(first, 0);
        for (int s0 = first, buf = 0; s0 < end; s0 += kBatch, buf ^= 1) {
            const int cnt = min(kBatch, end - s0);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (act) {
                float w[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; ++k)
                    w[k] = k < cnt ? A::mul(esw, cpow4<MODE>(p4, stage[buf][0][k][j], c.status)) : 0.0f;
                float4* d = reinterpret_cast<float4*>(&W[buf][j * kBatch]);
                d[0] = make_float4(w[0], w[1], w[2], w[3]);
                d[1] = make_float4(w[4], w[5], w[6], w[7]);
            }
            fetch(s0 + kBatch, buf ^ 1);
            __syncthreads();
            if (!act) continue;
            {
                // incident flux of boundary_condition (GPU_code.cu:418-490): the
                // module's order in REFERENCE precision, four partial sums in FAST
                const float* w = W[buf];
                float2 inc[kBatch / 2];
#pragma unroll
                for (int k = 0; k < kBatch / 2; ++k)
                    inc[k] = make_float2(stage[buf][1][2 * k][j], stage[buf][1][2 * k + 1][j]);
                if constexpr (MODE == MODE_REF) {
                    add_view<MODE>(inc, V, w, nsf, j, 0, 1, nsf);
                } else {
                    const int n4 = nsf & ~3;
                    const float2 zero = make_float2(0.0f, 0.0f);
                    float2 x[kBatch / 2], y[kBatch / 2], z[kBatch / 2];
#pragma unroll
                    for (int k = 0; k < kBatch / 2; ++k) x[k] = y[k] = zero;
                    add_view<MODE>(x, V, w, nsf, j, 0, 4, n4);
                    add_view<MODE>(x, V, w, nsf, j, n4, 1, nsf);
                    add_view<MODE>(y, V, w, nsf, j, 1, 4, n4);
#pragma unroll
                    for (int k = 0; k < kBatch / 2; ++k) {
                        x[k] = __fadd2_rn(x[k], y[k]);
                        y[k] = z[k] = zero;
                    }
                    add_view<MODE>(y, V, w, nsf, j, 2, 4, n4);
                    add_view<MODE>(z, V, w, nsf, j, 3, 4, n4);
#pragma unroll
                    for (int k = 0; k < kBatch / 2; ++k)
                        inc[k] = __fadd2_rn(inc[k], __fadd2_rn(x[k], __fadd2_rn(y[k], z[k])));
                }
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    const float in = (k & 1) ? inc[k / 2].y : inc[k / 2].x;
                    stage[buf][2][k][j] = A::add(A::mul(oma, stage[buf][2][k][j]), in);
                }
            }
            size_t o = base + (size_t)s0 * nsf;
#pragma unroll 2
            for (int k = 0; k < cnt; ++k, o += nsf) {
                const float old = stage[buf][0][k][j], m2 = stage[buf][2][k][j];
                // finite_difference (GPU_code.cu:377-412)
                float t0 = T[0];
#pragma unroll
                for (int i = 1; i < NX; ++i) {
                    const float t1 = T[i];
                    T[i] = A::add(t1, A::mul(m0f, A::add(A::sub(T[i + 1], A::mul(2.0f, t1)), t0)));
                    t0 = t1;
                }
                T[NX] = T[NX - 1];
                c.stemp0[o] = old;
                float TR0 = T[0], TR1 = T[0], DT = 1.0f;
                int it = 0;
                while (DT >= tacc2) {
                    if (it == 200) { flags |= ST_NEWTON_CAP; break; }
                    const float t3 = A::mul(A::mul(A::mul(es, TR0), TR0), TR0);
                    const float sbc = A::sub(A::add(m2, A::mul(m1, A::sub(T[1], TR0))), A::mul(t3, TR0));
                    const float sbcd = A::add(m1, A::mul(A::mul(A::mul(es4, TR0), TR0), TR0));
                    TR1 = A::add(TR0, A::div(sbc, sbcd));
                    DT = fabsf(A::sub(TR1, TR0));
                    TR0 = TR1;
                    ++it;
                }
                T[0] = TR1;
                c.stemp1[o] = TR1;
                hot = hot || (fabsf(A::sub(old, TR1)) >= tacc);
                if (!isfinite(TR1)) flags |= ST_NONFINITE;
            }
        }
        if (act) {
#pragma unroll
            for (int i = 0; i <= NX; ++i) tp[(size_t)i * nsf + j] = T[i];
        }
        if (flags) atomicOr(c.status, flags);
        const int any = __syncthreads_or(hot);
        if (threadIdx.x == 0) {
            if (any || first == 0) c.hot[f] = any ? 1 : 0;
            if (segs > 1) {
                __threadfence();  // the block's column and flags before the count
                *static_cast<volatile int*>(&work[f]) = piece + 1;
            }
        }
    }
}

// roughness_inst_equilibrium (GPU_code.cu:496-548)
template <int MODE>
__global__ void __launch_bounds__(128) k_crater_equilibrium(CraterDev c, PowTab p4, PowTab pq, float es) {
    using A = Ca<MODE>;
    extern __shared__ float sm[];
    const int nsf = c.nsf, ntau = c.ntau, f = blockIdx.x;
    if (c.conv[f]) return;
    float* Vs = sm;
    float* W = Vs + nsf * nsf;
    for (int k = threadIdx.x; k < nsf * nsf; k += blockDim.x) Vs[k] = c.V[k];
    const int j = threadIdx.x;
    const bool act = j < nsf;
    const float oma = A::sub(1.0f, c.albedo[f]);
    const float esw = A::mul(c.ir_abs, es);
    for (int s = 0; s < ntau; ++s) {
        const size_t o = (size_t)f * ntau * nsf + (size_t)s * nsf + j;
        if (act) {
            const float old = c.stemp1[o];
            c.stemp0[o] = old;
            W[j] = A::mul(esw, cpow4<MODE>(p4, old, c.status));
        }
        __syncthreads();
        if (act) {
            float inc = c.RGH[o];
            for (int i = 0; i != nsf; ++i) inc = A::add(inc, A::mul(W[i], Vs[i * nsf + j]));
            const float x = A::div(A::add(A::mul(oma, c.RI[o]), inc), es);
            c.stemp1[o] = (MODE == MODE_REF) ? libm_qroot(pq, x, c.status) : dev_qroot(x);
        }
        __syncthreads();
    }
}

// converged (GPU_code.cu:554-594); a facet still changing shows it in the first
// few steps, so the block stops at the first kConvSpan values per thread that
// hold a change (640 facets of 100 sub-facets, 720 steps, none converged: 313
// -> 44 us)
constexpr int kConvSpan = 8;
__global__ void __launch_bounds__(128) k_crater_converged(CraterDev c, float tacc) {
    const int f = blockIdx.x;
    if (c.conv[f]) return;
    const size_t n = (size_t)c.ntau * c.nsf, base = (size_t)f * n;
    int bad = 0;
    for (size_t k0 = 0; k0 < n && !bad; k0 += (size_t)kConvSpan * blockDim.x) {
#pragma unroll
        for (int u = 0; u < kConvSpan; ++u) {
            const size_t k = k0 + (size_t)u * blockDim.x + threadIdx.x;
            if (k < n && fabsf(c.stemp0[base + k] - c.stemp1[base + k]) >= tacc) bad = 1;
        }
        bad = __syncthreads_or(bad);
    }
    if (threadIdx.x == 0) c.conv[f] = bad ? 0 : 1;
}

// first initialisation pass: per sub-facet mean of (1-A) RI + RGH (GPU_code.cu:341-345)
__global__ void k_crater_init_mean(CraterDev c, float* out, int with_self, const float* selfh) {
    const int f = blockIdx.x, j = threadIdx.x;
    if (j >= c.nsf) return;
    const float alb = c.albedo[f];
    const float inv = __fdiv_rn(1.0f, (float)c.ntau);
    const float sh = with_self ? selfh[(size_t)f * c.nsf + j] : 0.0f;
    float t = 0.0f;
#pragma unroll 8
    for (int s = 0; s < c.ntau; ++s) {
        const size_t o = (size_t)f * c.ntau * c.nsf + (size_t)s * c.nsf + j;
        float x = __fadd_rn(__fmul_rn(__fsub_rn(1.0f, alb), c.RI[o]), c.RGH[o]);
        if (with_self) x = __fadd_rn(x, sh);
        t = __fadd_rn(t, __fmul_rn(inv, x));
    }
    out[(size_t)f * c.nsf + j] = t;
}

// crater self-heating of the first initialisation temperatures (GPU_code.cu:351-354)
__global__ void k_crater_init_self(CraterDev c, PowTab p4, float es, const float* t0, float* out) {
    extern __shared__ float sm[];
    const int f = blockIdx.x, j = threadIdx.x, nsf = c.nsf;
    float* w = sm;
    if (j < nsf) w[j] = __fmul_rn(__fmul_rn(c.ir_abs, es), cpow4_exact(p4, t0[(size_t)f * nsf + j], c.status));
    __syncthreads();
    if (j >= nsf) return;
    float sh = 0.0f;
    for (int i = 0; i != nsf; ++i) sh = __fadd_rn(sh, __fmul_rn(w[i], c.V[i * nsf + j]));
    out[(size_t)f * nsf + j] = sh;
}

// t = (t / (eps sigma))^0.25 of the initialisation (GPU_code.cu:346, 362)
template <int MODE>
__global__ void k_crater_root(CraterDev c, PowTab pq, float es, float* t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.nf * c.nsf) return;
    const float x = __fdiv_rn(t[i], es);
    t[i] = (MODE == MODE_REF) ? libm_qroot(pq, x, c.status) : dev_qroot(x);
}

__global__ void k_crater_fill(CraterDev c, const float* t) {
    const int f = blockIdx.x, j = threadIdx.x;
    if (j >= c.nsf) return;
    const float v = t[(size_t)f * c.nsf + j];
    for (int i = 0; i <= c.nx; ++i) c.temp[((size_t)f * (c.nx + 1) + i) * c.nsf + j] = v;
    for (int s = 0; s < c.ntau; ++s) {
        const size_t o = (size_t)f * c.ntau * c.nsf + (size_t)s * c.nsf + j;
        c.stemp0[o] = v;
        c.stemp1[o] = v;
    }
}

// ------------------------------------------------------------------ launchers
#define CRATER_NX_LIST(X) X(8) X(12) X(16) X(24) X(32) X(40) X(48) X(56) X(64)

namespace {
template <int MODE, int NX>
int launch_crater_revolution(const CraterDev& c, const PowTab& p4, const float* a, int* work, cudaStream_t st) {
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_crater_revolution<MODE, NX, 4>, 128, 0) != cudaSuccess)
        return 2;
    const int resident = sms * per;
    const int segs = c.nf > resident ? kSegments : 1;
    if (segs > 1 && cudaMemsetAsync(work, 0, ((size_t)c.nf + 1) * sizeof(int), st) != cudaSuccess) return 2;
    if (c.nf <= 2 * sms)
        k_crater_revolution<MODE, NX, 2><<<c.nf, 128, 0, st>>>(c, p4, a[0], a[1], a[2], a[3], a[4], a[5], work, segs);
    else
        k_crater_revolution<MODE, NX, 4><<<segs > 1 ? resident : c.nf, 128, 0, st>>>(c, p4, a[0], a[1], a[2], a[3],
                                                                                    a[4], a[5], work, segs);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
}  // namespace

int crater_launch(int what, const CraterDev& c, const PowTab& p4, const PowTab& pq, const float* fargs, void* p0,
                  void* p1, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    const size_t smv = (size_t)c.nsf * c.nsf * 4;
    // dynamic shared memory of the largest crater (128 sub-facets): the limit belongs
    // to a function, not to a launch, so every thread sets the same one
    constexpr int kSharedLimit = (128 * 128 + kScatSteps * 128) * 4;
    const int grid_fs = 152 * 8;
    switch (what) {
        case 0:  // partial shadow
        {
            // one wave, as every block sets its sub-points up
            int dev = 0, sms = 0, per = 0;
            const void* k = c.mode == MODE_FAST ? (const void*)k_crater_shadow<MODE_FAST> : (const void*)k_crater_shadow<MODE_REF>;
            if (cudaGetDevice(&dev) != cudaSuccess ||
                cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, 128, 0) != cudaSuccess)
                return 2;
            if (c.mode == MODE_FAST) k_crater_shadow<MODE_FAST><<<sms * per, 128, 0, st>>>(c);
            else k_crater_shadow<MODE_REF><<<sms * per, 128, 0, st>>>(c);
            break;
        }
        case 1: {  // scattering: fargs = {solar, acc, multiple}
            const size_t sm = smv + (size_t)kScatSteps * c.nsf * 4;
            cudaFuncSetAttribute(k_crater_scatter<MODE_REF>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedLimit);
            cudaFuncSetAttribute(k_crater_scatter<MODE_FAST>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedLimit);
            if (c.mode == MODE_FAST)
                k_crater_scatter<MODE_FAST><<<grid_fs, 128, sm, st>>>(c, fargs[0], fargs[1], (int)fargs[2], 10000);
            else
                k_crater_scatter<MODE_REF><<<grid_fs, 128, sm, st>>>(c, fargs[0], fargs[1], (int)fargs[2], 10000);
            break;
        }
        case 2:  // revolution: fargs = {es, es4, m0, dz, tacc, tacc2}, p0 = [nf + 1] work words
#define NX_CASE(n)                                                                                              \
    case n:                                                                                                     \
        return c.mode == MODE_FAST ? launch_crater_revolution<MODE_FAST, n>(c, p4, fargs, static_cast<int*>(p0), st) \
                                   : launch_crater_revolution<MODE_REF, n>(c, p4, fargs, static_cast<int*>(p0), st);
            switch (c.nx) {
                CRATER_NX_LIST(NX_CASE)
                default: return 1;
            }
#undef NX_CASE
        case 3: {  // equilibrium: fargs = {es}
            const size_t sm = smv + c.nsf * 4;
            cudaFuncSetAttribute(k_crater_equilibrium<MODE_REF>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedLimit);
            cudaFuncSetAttribute(k_crater_equilibrium<MODE_FAST>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedLimit);
            if (c.mode == MODE_FAST) k_crater_equilibrium<MODE_FAST><<<c.nf, 128, sm, st>>>(c, p4, pq, fargs[0]);
            else k_crater_equilibrium<MODE_REF><<<c.nf, 128, sm, st>>>(c, p4, pq, fargs[0]);
            break;
        }
        case 4:  // converged: fargs = {tacc}
            k_crater_converged<<<c.nf, 128, 0, st>>>(c, fargs[0]);
            break;
        case 5:  // init mean (pass 1 when p1 == null, pass 2 with self-heating p1)
            k_crater_init_mean<<<c.nf, 128, 0, st>>>(c, static_cast<float*>(p0), p1 ? 1 : 0,
                                                     static_cast<const float*>(p1));
            break;
        case 6:  // init self-heating: fargs = {es}; p0 = t0, p1 = out
            k_crater_init_self<<<c.nf, 128, c.nsf * 4, st>>>(c, p4, fargs[0], static_cast<const float*>(p0),
                                                             static_cast<float*>(p1));
            break;
        case 7:  // fill
            k_crater_fill<<<c.nf, 128, 0, st>>>(c, static_cast<const float*>(p0));
            break;
        case 8: {  // fourth root in place: fargs = {es}; p0 = t
            const int g = (c.nf * c.nsf + 127) / 128;
            if (c.mode == MODE_FAST) k_crater_root<MODE_FAST><<<g, 128, 0, st>>>(c, pq, fargs[0], static_cast<float*>(p0));
            else k_crater_root<MODE_REF><<<g, 128, 0, st>>>(c, pq, fargs[0], static_cast<float*>(p0));
            break;
        }
        default:
            return 1;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

bool crater_nx_supported(int nx) {
#define NX_CASE(n) if (nx == n) return true;
    CRATER_NX_LIST(NX_CASE)
#undef NX_CASE
    return false;
}

}  // namespace atpm
