// Disk-integrated thermal flux seen by an observer, in FP64 on the device:
// the smooth-surface sum of the reference's Observe stage
// (observe, 3905/Observe/NominalPole/wise_main.cpp:662-730, geometry
// 555-645).  For every step s and wavelength l:
//
//   F[s][l] = sum over facets f visible at s of
//             B_l(T_f[s]) * eps * A_f * cos(e_f[s]) / d_f[s]^2
//
// with B the Planck radiance (the stage's constants), e the angle between
// the facet normal and the direction to the observer, d the facet's distance
// to the observer, A_f the facet area as the stage leaves it (computed at the
// last step of its geometry loop).
//
//   k_flux_vertices every vertex at every step (host-libm rotation table, pole
//                   matrix), once instead of for each facet around it
//   k_flux_area     the facets' areas
//   k_flux_flags    the caller's visibility words, transposed to bytes
//   k_flux_partial  one thread per (facet, step): weight and Planck terms; a
//                   fixed-order sum over each 256-facet block
//   k_flux_sum      sums the block partials of every (step, wavelength) in
//                   block order: the result does not depend on scheduling
//
// All of it is FP64, on a part whose FP64 rate is 1/64 of FP32, so FP64
// operations are what it costs.  The positions are the stage's, operand by
// operand (its body lies 1e11 m away from an origin while its shape keeps its
// own units, so their rounding shows in the normals and, for an observer near the
// body, in the view vector); from them on, cosines come from one reciprocal square
// root instead of a facet frame, acos and cos, and a wavelength costs one exp and
// one reciprocal: 13.0 -> 4.1 ms for 21,760 facets, 720 steps and three
// wavelengths.  A cosine within kSure of 0 or 1 is formed by the stage's own
// sequence (stage_view): there its rounding decides whether a facet or sub-facet
// counts.
//
// The rough-surface sum (observe, wise_main.cpp:695-727) replaces each
// facet's own term by its crater's: the sub-facets with a visible fraction
// toward the observer > 0 add B(T_sub) eps a_sub vis cos(e_sub) / d^2, and
// the facet's total enters scaled by A_f over the crater's projected area.
#include <cuda_runtime.h>

#include "atpm_internal.h"

namespace atpm {

namespace {

constexpr int kFluxThreads = 256;

template <class R>
__device__ __forceinline__ double temp_at(const DevSolve& s, int f, int step) {
    return (double)static_cast<const R*>(s.stemp1)[(size_t)step * s.nf + f];
}

__global__ void __launch_bounds__(256) k_flux_vertices(DevSolve s, FluxArgs a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)s.nv * a.ns) return;
    const int step = a.s0 + (int)(i / s.nv), v = (int)(i % s.nv);
    const double* e = s.vert + 3 * v;
    const double* rt = (v < a.vsplit) ? a.rot : a.rot2;
    const double c = rt[2 * step], sn = rt[2 * step + 1];
    double rq[3];
    rq[0] = __dsub_rn(__dmul_rn(e[0], c), __dmul_rn(e[1], sn));
    rq[1] = __dadd_rn(__dmul_rn(e[0], sn), __dmul_rn(e[1], c));
    rq[2] = e[2];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        a.hp[3 * i + k] =
            __dadd_rn(a.car[k], __dadd_rn(__dadd_rn(__dmul_rn(a.tm[3 * k], rq[0]), __dmul_rn(a.tm[3 * k + 1], rq[1])),
                                          __dmul_rn(a.tm[3 * k + 2], rq[2])));
}

// a facet's corners at a step, its first edge and its normal (not scaled)
struct Facet {
    double sum[3], edge[3], n[3];
    __device__ __forceinline__ Facet(const DevSolve& s, const FluxArgs& a, int f, int step) {
        const double* hp = a.hp + (size_t)(step - a.s0) * s.nv * 3;
        const int* fv = s.fac + 3 * f;
        const double *h0 = hp + 3 * (size_t)fv[0], *h1 = hp + 3 * (size_t)fv[1], *h2 = hp + 3 * (size_t)fv[2];
        double nc1[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double x = __ldg(h0 + k), y = __ldg(h1 + k), z = __ldg(h2 + k);
            sum[k] = __dadd_rn(__dadd_rn(x, y), z);
            edge[k] = __dsub_rn(y, x);
            nc1[k] = __dsub_rn(z, x);
        }
        n[0] = __dsub_rn(__dmul_rn(edge[1], nc1[2]), __dmul_rn(edge[2], nc1[1]));
        n[1] = __dsub_rn(__dmul_rn(edge[2], nc1[0]), __dmul_rn(edge[0], nc1[2]));
        n[2] = __dsub_rn(__dmul_rn(edge[0], nc1[1]), __dmul_rn(edge[1], nc1[0]));
    }
};

__device__ __forceinline__ double dot3(const double* a, const double* b) {
    return __dadd_rn(__dadd_rn(__dmul_rn(a[0], b[0]), __dmul_rn(a[1], b[1])), __dmul_rn(a[2], b[2]));
}

// area as the stage leaves it: from the last step of its geometry loop
__global__ void __launch_bounds__(256) k_flux_area(DevSolve s, FluxArgs a) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= s.nf) return;
    const Facet t(s, a, f, s.ntau - 1);
    a.area[f] = __ddiv_rn(__dsqrt_rn(dot3(t.n, t.n)), 2.0);
}

// [nf][steps] words -> [steps][nf] bytes
__global__ void __launch_bounds__(256) k_flux_flags(const int32_t* src, uint8_t* dst, int nf, int ntau) {
    __shared__ uint8_t t[32][33];
    const int f0 = blockIdx.y * 32, s0 = blockIdx.x * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int f = f0 + j, s = s0 + threadIdx.x;
        if (f < nf && s < ntau) t[j][threadIdx.x] = src[(size_t)f * ntau + s] ? 1 : 0;
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int s = s0 + j, f = f0 + threadIdx.x;
        if (f < nf && s < ntau) dst[(size_t)s * nf + f] = t[threadIdx.x][j];
    }
}

// what the cosines here and the stage's may differ by (each a few operations of
// 2^-53 on terms of at most 1), with room to spare
constexpr double kSure = 1e-14;

__device__ __forceinline__ int exponent(double x) { return __double2hiint(x) >> 20 & 0x7ff; }

// x / 3 correctly rounded: the product with the rounded 1/3, corrected by its exact
// residual (P. Markstein, IBM J. Res. Dev. 34, 1990), on a part where a division
// takes some ten FP64 operations
__device__ __forceinline__ double third(double x) {
    const double q = __dmul_rn(x, 1.0 / 3.0);
    return __fma_rn(__fma_rn(-3.0, q, x), 1.0 / 3.0, q);
}

// the stage's own view of a facet in its operand order (wise_main.cpp:555-645):
// the view vector in the facet's frame (rows x^, y, n) and its length; returns the
// angle to the normal, NaN where the cosine rounds above 1
__device__ __noinline__ double stage_view(const DevSolve& s, const FluxArgs& a, int f, int step, double (&v)[3],
                                          double& d) {
    const Facet t(s, a, f, step);
    const double nn = __dsqrt_rn(dot3(t.n, t.n)), xx = __dsqrt_rn(dot3(t.edge, t.edge));
    double n[3], x[3], ov[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        n[k] = __ddiv_rn(t.n[k], nn);
        x[k] = __ddiv_rn(t.edge[k], xx);
        ov[k] = __dsub_rn(__ddiv_rn(t.sum[k], 3.0), a.obs[k]);
    }
    const double y[3] = {__dsub_rn(__dmul_rn(n[1], x[2]), __dmul_rn(n[2], x[1])),
                         __dsub_rn(__dmul_rn(n[2], x[0]), __dmul_rn(n[0], x[2])),
                         __dsub_rn(__dmul_rn(n[0], x[1]), __dmul_rn(n[1], x[0]))};
    v[0] = -dot3(x, ov);
    v[1] = -dot3(y, ov);
    v[2] = -dot3(n, ov);
    d = __dsqrt_rn(dot3(v, v));
    return acos(__ddiv_rn(v[2], __dsqrt_rn(dot3(ov, ov))));
}
constexpr double kRight = 3.141592653589793 / 2.0;

// (2hc^2 / lambda^5) * (1 / (exp(hc / (lambda k T)) - 1)), 0 where that is NaN
__device__ __forceinline__ double planck(const FluxArgs& a, int l, double inv_t) {
    const double b = a.b1[l] / (exp(a.hl[l] * inv_t) - 1.0);
    return b == b ? b : 0.0;
}

template <class R, bool ROUGH>
__global__ void __launch_bounds__(kFluxThreads) k_flux_partial(DevSolve s, FluxArgs a) {
    constexpr int kWarps = kFluxThreads / 32;
    __shared__ double red[kMaxFluxWavelengths][kWarps];
    // rough: each facet's unit view vector in its frame and its weight
    __shared__ double view[ROUGH ? kFluxThreads : 1][4];
    const int step = a.s0 + blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f = blockIdx.x * kFluxThreads + threadIdx.x;
    double term[kMaxFluxWavelengths];
#pragma unroll
    for (int l = 0; l < kMaxFluxWavelengths; ++l) term[l] = 0.0;
    double weight = 0.0;
    if (f < s.nf && (!a.visible || a.visible[(size_t)blockIdx.y * s.nf + f])) {
        const Facet t(s, a, f, step);
        double ov[3];  // from the facet to the observer
#pragma unroll
        for (int k = 0; k < 3; ++k) ov[k] = __dsub_rn(a.obs[k], a.close ? third(t.sum[k]) : t.sum[k] * (1.0 / 3.0));
        const double oo = dot3(ov, ov), nn = dot3(t.n, t.n), no = dot3(t.n, ov);
        // cosine toward the observer; |cosine| < kSure by the exponents
        const bool edge_on = 2 * exponent(no) < exponent(nn) + exponent(oo) - 88;
        double c = no > 0.0 ? no * rsqrt(nn * oo) : -1.0;
        bool seen = c > 0.0;
        if (edge_on || (__double2hiint(c) >= 0x3fefffff && c > 1.0 - kSure)) {
            double v[3], d;
            const double angle = stage_view(s, a, f, step, v, d);
            // NaN passes the stage's horizon test; its own term is then dropped,
            // a crater's terms have their own angles
            seen = !(angle > kRight) && (ROUGH || angle == angle);
            c = cos(angle);
        }
        if (seen) {
            weight = a.eps * a.area[f] / oo;
            if constexpr (!ROUGH) {
                weight *= c;
                const double inv_t = 1.0 / temp_at<R>(s, f, step);
#pragma unroll
                for (int l = 0; l < kMaxFluxWavelengths; ++l)
                    if (l < a.nwl) term[l] = planck(a, l, inv_t) * weight;
            } else {
                // the view vector in the facet's frame (rows x^, y, n)
                const double rx = rsqrt(dot3(t.edge, t.edge)), rn = rsqrt(nn), ro = rsqrt(oo);
                double x[3], n[3], u[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    x[k] = t.edge[k] * rx;
                    n[k] = t.n[k] * rn;
                    u[k] = ov[k] * ro;
                }
                const double y[3] = {n[1] * x[2] - n[2] * x[1], n[2] * x[0] - n[0] * x[2], n[0] * x[1] - n[1] * x[0]};
                view[threadIdx.x][0] = dot3(x, u);
                view[threadIdx.x][1] = dot3(y, u);
                view[threadIdx.x][2] = dot3(n, u);
                weight /= a.sub_total;
            }
        }
    }
    if constexpr (ROUGH) {
        // each facet's crater, a lane per sub-facet: every one with a visible
        // fraction > 0 at its own view angle (wise_main.cpp:515), the facet's
        // total scaled by its share of the crater's projected area
        // (wise_main.cpp:718)
        view[threadIdx.x][3] = weight;
        __syncwarp();
        // the warp's facets end to end, so that few sub-facets leave no lane idle
        int i = lane / a.nsf, j = lane % a.nsf;
        for (; i < 32; j += 32) {
            for (; j >= a.nsf; j -= a.nsf) ++i;
            if (i >= 32) break;
            const double* v = view[warp * 32 + i];
            if (v[3] == 0.0) continue;
            const int facet = blockIdx.x * kFluxThreads + warp * 32 + i;
            const size_t at = ((size_t)facet * s.ntau + step) * (size_t)a.nsf + j;
            const double vis = (double)a.sub_vis[at];
            const double* g = a.sub_geo + 4 * j;
            double c = v[0] * g[0] + v[1] * g[1] + v[2] * g[2];
            if (!(vis > 0.0)) continue;
            if (fabs(c) > 1.0 - kSure) {  // the stage's acos of a ratio above 1 is NaN: no term
                double w[3], d;
                stage_view(s, a, facet, step, w, d);
                c = __ddiv_rn(dot3(w, g), d);
            }
            if (!(fabs(c) <= 1.0)) continue;
            const double m = v[3] * g[3] * vis * c, inv_t = 1.0 / (double)a.sub_T[at];
#pragma unroll
            for (int l = 0; l < kMaxFluxWavelengths; ++l)
                if (l < a.nwl) term[l] += planck(a, l, inv_t) * m;
        }
    }
#pragma unroll
    for (int l = 0; l < kMaxFluxWavelengths; ++l) {
        if (l >= a.nwl) break;
        double t = term[l];
        for (int o = 16; o > 0; o >>= 1) t = __dadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
        if (lane == 0) red[l][warp] = t;
    }
    __syncthreads();
    if (threadIdx.x < a.nwl) {
        double t = red[threadIdx.x][0];
        for (int w = 1; w < kWarps; ++w) t = __dadd_rn(t, red[threadIdx.x][w]);
        a.partial[((size_t)step * gridDim.x + blockIdx.x) * a.nwl + threadIdx.x] = t;
    }
}

__global__ void k_flux_sum(FluxArgs a, int ntau, int nblk) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntau * a.nwl) return;
    const int step = i / a.nwl, l = i % a.nwl;
    double t = 0.0;
    for (int b = 0; b < nblk; ++b) t = __dadd_rn(t, a.partial[((size_t)step * nblk + b) * a.nwl + l]);
    a.out[i] = t;
}

}  // namespace

size_t flux_partial_bytes(const DevSolve& s, int nwl) {
    const size_t nblk = (size_t)(s.nf + kFluxThreads - 1) / kFluxThreads;
    return nblk * s.ntau * nwl * sizeof(double);
}

int launch_flux_steps(const DevSolve& s, const FluxArgs& a, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    if (a.nwl < 1 || a.nwl > kMaxFluxWavelengths) return 1;
    const dim3 grid((s.nf + kFluxThreads - 1) / kFluxThreads, a.ns);
    const long long nvt = (long long)s.nv * a.ns;
    k_flux_vertices<<<(unsigned)((nvt + 255) / 256), 256, 0, st>>>(s, a);
    if (a.s0 + a.ns == s.ntau) k_flux_area<<<(s.nf + 255) / 256, 256, 0, st>>>(s, a);
    if (a.visible)
        k_flux_flags<<<dim3((a.ns + 31) / 32, (s.nf + 31) / 32), dim3(32, 8), 0, st>>>(
            a.flags, const_cast<uint8_t*>(a.visible), s.nf, a.ns);
    if (a.sub_T) {
        if (s.mode == MODE_FP64) k_flux_partial<double, true><<<grid, kFluxThreads, 0, st>>>(s, a);
        else k_flux_partial<float, true><<<grid, kFluxThreads, 0, st>>>(s, a);
    } else {
        if (s.mode == MODE_FP64) k_flux_partial<double, false><<<grid, kFluxThreads, 0, st>>>(s, a);
        else k_flux_partial<float, false><<<grid, kFluxThreads, 0, st>>>(s, a);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_flux_sum(const DevSolve& s, const FluxArgs& a, stream_t stv) {
    const int nblk = (s.nf + kFluxThreads - 1) / kFluxThreads;
    k_flux_sum<<<(s.ntau * a.nwl + 127) / 128, 128, 0, static_cast<cudaStream_t>(stv)>>>(a, s.ntau, nblk);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace atpm
