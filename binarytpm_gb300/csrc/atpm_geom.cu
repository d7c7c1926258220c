// Geometry and shadowing in heliocentric FP64 (the reference's frame).
//
//   k_geom_vertices  rotation about the body z axis, pole transform and
//                    heliocentric offset of every vertex at every step
//                    (asteroidgeometry, 3905/Thermal/NominalPole/main.cpp:938-958),
//                    and its central projection for the culled drivers
//   k_geom_facets    Sun angle and self-shadow of every facet at every step
//                    (main.cpp:960-1030)
//   k_geom_arrays    midpoint, unit normal and distance, which only the plain
//                    drivers read from memory
//   k_shadow_dep     astshadow over the view-factor lists (main.cpp:1286-1315)
//   k_shadow_all     all-pairs astshadow of the Visibility stage
//                    (3905/Visibility/NominalPole/main.cpp:674-704)
//   shadowtest       astshadowtest (main.cpp:1187-1247)
//
// Culled drivers (same flags): every ray starts at the origin (the Sun, or the
// observer in the Visibility stage), so the test is two-dimensional in the
// central projection onto the plane normal to the body's direction: the ray's
// point lies inside facet h exactly when g's projected midpoint lies inside
// h's projected triangle.  Candidates go through a box test, the order of the
// two facets along the ray, and the projected triangle's edges, all in FP32; a
// point or an order within Proj::margin of a decision, far more than the
// rounding of both tests, is decided by the exact FP64 test from the vertex
// positions.  Nearly every decision is clear of it (GB300's FP64 rate is 1/64 of
// its FP32 rate).
//   k_window_box     each facet's box over every window of 32 steps
//   k_shadow_dep_cull the dependent-list driver: 32 entries' window boxes at a
//                    time, then the entries left, 32 steps at a time
//   k_grid_*         a uniform grid per step over the projected facets (each
//                    in every cell its box touches; cell size three
//                    quarters of the largest box), built by counting sort
//   k_shadow_grid    the all-pairs driver over the cell g lies in
//
// Every FP64 operation uses round-to-nearest intrinsics in the reference's
// operand order, with the rotation cos/sin and the pole matrix computed on the
// host by the same libm the reference uses, so positions, normals and shadow
// flags are bit-identical to the reference's.
//
// Layouts are facet-major over steps ([f][s][3]) so a warp that owns 32
// consecutive steps of one facet reads each neighbour's data as one
// contiguous segment.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "atpm_internal.h"

namespace atpm {

#define DADD __dadd_rn
#define DSUB __dsub_rn
#define DMUL __dmul_rn
#define DDIV __ddiv_rn

struct GeomArgs {
    DevSolve s;
    GeomWork g;
};

// the projection of k_geom_vertices: c the body's direction, e1 and e2 normal
// to it, coordinates in km at the body's distance
struct Proj {
    float c[3], e1[3], e2[3];
    float scale, inv; // distance of the body centre, and 1 over it
    float pad;        // box padding (km)
    float margin;     // beyond this from a decision FP32 decides (km)
    float lift;       // most a midpoint's distance exceeds the body's and its depth (km)
    float2* uv;       // [nv][ntau]
    float* w;         // [nv][ntau] depth behind the body centre along c
    unsigned* stats;  // [0] max |u|,|v| (float bits), [1] max box extent, [2] bad-projection flag, [3] max |w|,
                      // [4] max -w
    float4* wbox;     // [windows][nf] union of each facet's padded boxes over 32 steps (or null)
};

// the largest of the warp's values, every lane taking part, into *to
__device__ __forceinline__ void warp_max_to(unsigned* to, unsigned v) {
    const unsigned most = __reduce_max_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && most > __ldcg(to)) atomicMax(to, most);
}

__global__ void __launch_bounds__(256) k_geom_vertices(GeomArgs a, Proj p) {
    const int nv = a.s.nv, ntau = a.s.ntau;
    const long long n = (long long)nv * ntau, at = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = at < n ? at : n - 1;  // lanes beyond the end repeat the last vertex
    const int v = (int)(i / ntau), s = (int)(i % ntau);
    const double* e = a.s.vert + 3 * v;
    // a non-synchronous secondary turns at its own rate (its own table)
    const double* rt = (v < a.g.vsplit) ? a.g.rot : a.g.rot2;
    const double c = rt[2 * s], sn = rt[2 * s + 1];
    double rq[3];
    rq[0] = DSUB(DMUL(e[0], c), DMUL(e[1], sn));
    rq[1] = DADD(DMUL(e[0], sn), DMUL(e[1], c));
    rq[2] = e[2];
    double* hp = a.g.hp + ((size_t)v * ntau + s) * 3;
    float ef[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double ec = DADD(DADD(DMUL(a.g.tm[3 * k + 0], rq[0]), DMUL(a.g.tm[3 * k + 1], rq[1])),
                               DMUL(a.g.tm[3 * k + 2], rq[2]));
        hp[k] = DADD(a.g.car[k], ec);
        ef[k] = (float)ec;
    }
    if (!p.uv) return;
    // central projection of car + ec; car is along c, so only ec counts
    const float w = ef[0] * p.c[0] + ef[1] * p.c[1] + ef[2] * p.c[2];
    const float x = ef[0] * p.e1[0] + ef[1] * p.e1[1] + ef[2] * p.e1[2];
    const float y = ef[0] * p.e2[0] + ef[1] * p.e2[1] + ef[2] * p.e2[2];
    const float d = p.scale + w;
    if (!(d > 0.5f * sqrtf(d * d + x * x + y * y))) atomicOr(&p.stats[2], 1u);  // the projection is not used
    const float m = 1.0f / (1.0f + w / p.scale), u = x * m, t = y * m;
    p.uv[i] = make_float2(u, t);
    p.w[i] = w;
    warp_max_to(&p.stats[0], __float_as_uint(fmaxf(fabsf(u), fabsf(t))));
    warp_max_to(&p.stats[3], __float_as_uint(fabsf(w)));
    warp_max_to(&p.stats[4], __float_as_uint(fmaxf(-w, 0.0f)));
}

// a facet's midpoint, unit normal and the midpoint's distance at one step, in
// the reference's operand order
__device__ __forceinline__ void facet_frame(const double* h0, const double* h1, const double* h2, double* hm, double* n,
                                            double* dist) {
    double nc0[3], nc1[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        hm[k] = DDIV(DADD(DADD(h0[k], h1[k]), h2[k]), 3.0);
        nc0[k] = DSUB(h1[k], h0[k]);
        nc1[k] = DSUB(h2[k], h0[k]);
    }
    *dist = __dsqrt_rn(DADD(DADD(DMUL(hm[0], hm[0]), DMUL(hm[1], hm[1])), DMUL(hm[2], hm[2])));
    n[0] = DSUB(DMUL(nc0[1], nc1[2]), DMUL(nc0[2], nc1[1]));
    n[1] = DSUB(DMUL(nc0[2], nc1[0]), DMUL(nc0[0], nc1[2]));
    n[2] = DSUB(DMUL(nc0[0], nc1[1]), DMUL(nc0[1], nc1[0]));
    const double nn = __dsqrt_rn(DADD(DADD(DMUL(n[0], n[0]), DMUL(n[1], n[1])), DMUL(n[2], n[2])));
    n[0] = DDIV(n[0], nn);
    n[1] = DDIV(n[1], nn);
    n[2] = DDIV(n[2], nn);
}

__device__ __forceinline__ const double* vertex(const double* hp, const int* fac, int ntau, int f, int k, int s) {
    return hp + ((size_t)fac[3 * f + k] * ntau + s) * 3;
}

// the cosine of the Sun angle before acos, in the reference's operand order
__device__ __noinline__ double sun_cosine(const double* hp, const int* fac, int ntau, int f, int s) {
    double hm[3], n[3], t;
    facet_frame(vertex(hp, fac, ntau, f, 0, s), vertex(hp, fac, ntau, f, 1, s), vertex(hp, fac, ntau, f, 2, s), hm, n, &t);
    const double iv2 = -DADD(DADD(DMUL(n[0], hm[0]), DMUL(n[1], hm[1])), DMUL(n[2], hm[2]));
    return DDIV(iv2, t);
}

// Sun angle and self-shadow.  FAST keeps the cosine itself, dark where it is
// negative; REFERENCE keeps (float)cos(acos(cosine)), dark where the angle is
// above pi/2 (both the same but for the last bits of a double).  The divisions,
// square roots and transcendentals of that are most of the kernel on a part
// whose FP64 rate is 1/64 of FP32, and the flag and a float need few of the
// double's bits: the cosine is first formed with one reciprocal square root,
// within 1e-15 of the exact sequence (each sums a handful of terms of at most
// 1 rounded to 53 bits), and only where kSure does not settle the float or the
// sign does the exact sequence run.  21,760 facets x 720 steps, FAST: 3.1 ms (with
// midpoints and normals written) -> 1.2; FP64 keeps the exact sequence.
constexpr double kSure = 1e-14;

template <int MODE>
__global__ void __launch_bounds__(256) k_geom_facets(GeomArgs a) {
    const int nf = a.s.nf, ntau = a.s.ntau;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nf * ntau) return;
    const int f = (int)(i / ntau), s = (int)(i % ntau);
    const size_t o = (size_t)f * ntau + s;
    if constexpr (MODE != MODE_FP64) {
        const double* h0 = vertex(a.g.hp, a.s.fac, ntau, f, 0, s);
        const double* h1 = vertex(a.g.hp, a.s.fac, ntau, f, 1, s);
        const double* h2 = vertex(a.g.hp, a.s.fac, ntau, f, 2, s);
        double m[3], x[3], y[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            m[k] = (h0[k] + h1[k]) + h2[k];
            x[k] = h1[k] - h0[k];
            y[k] = h2[k] - h0[k];
        }
        const double n0 = DSUB(DMUL(x[1], y[2]), DMUL(x[2], y[1]));
        const double n1 = DSUB(DMUL(x[2], y[0]), DMUL(x[0], y[2]));
        const double n2 = DSUB(DMUL(x[0], y[1]), DMUL(x[1], y[0]));
        const double nn = n0 * n0 + n1 * n1 + n2 * n2, mm = m[0] * m[0] + m[1] * m[1] + m[2] * m[2];
        const double ci = -(n0 * m[0] + n1 * m[1] + n2 * m[2]) * rsqrt(nn * mm);
        const float lo = (float)(ci - kSure), hi = (float)(ci + kSure);
        if (lo == hi && (lo > 0.0f || hi < 0.0f) && fabs(ci) < 1.0 - kSure) {  // false for NaN
            static_cast<float*>(a.s.cosil)[o] = lo;
            a.s.shadow[o] = lo > 0.0f ? 1 : 0;
            return;
        }
    }
    const double ci = sun_cosine(a.g.hp, a.s.fac, ntau, f, s);
    if constexpr (MODE == MODE_FAST) {
        static_cast<float*>(a.s.cosil)[o] = (float)ci;
        a.s.shadow[o] = ci < 0.0 ? 0 : 1;
    } else {
        const double ia = acos(ci);
        if (MODE == MODE_FP64) static_cast<double*>(a.s.cosil)[o] = cos(ia);
        else static_cast<float*>(a.s.cosil)[o] = (float)cos(ia);
        a.s.shadow[o] = (ia > (3.141592653589793 / 2.0)) ? 0 : 1;
    }
}

__global__ void __launch_bounds__(256) k_geom_arrays(GeomArgs a) {
    const int nf = a.s.nf, ntau = a.s.ntau;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nf * ntau) return;
    const int f = (int)(i / ntau), s = (int)(i % ntau);
    double hm[3], n[3];
    facet_frame(vertex(a.g.hp, a.s.fac, ntau, f, 0, s), vertex(a.g.hp, a.s.fac, ntau, f, 1, s),
                vertex(a.g.hp, a.s.fac, ntau, f, 2, s), hm, n, &a.g.dist[i]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a.g.hm[3 * i + k] = hm[k];
        a.g.nrm[3 * i + k] = n[k];
    }
}

// astshadowtest: 0 when the triangle V0 V1 V2 (midpoint Hm, normal Hn) blocks
// the ray from the Sun (origin) to Gm
__device__ __forceinline__ int shadowtest(const double* Gm, const double* Hm, const double* Hn, const double* V0,
                                          const double* V1, const double* V2) {
    const double tc2 = DADD(DADD(DMUL(Gm[0], Hn[0]), DMUL(Gm[1], Hn[1])), DMUL(Gm[2], Hn[2]));
    const double tc1 = DADD(DADD(DMUL(Hm[0], Hn[0]), DMUL(Hm[1], Hn[1])), DMUL(Hm[2], Hn[2]));
    const double t = DDIV(tc1, tc2);
    double x[3], n1[3], n2[3], n3[3], x1[3], x2[3], x3[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        x[k] = DMUL(t, Gm[k]);
        n1[k] = DSUB(V1[k], V0[k]);
        n2[k] = DSUB(V0[k], V2[k]);
        n3[k] = DSUB(V2[k], V1[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        x1[k] = DSUB(x[k], V0[k]);
        x3[k] = DSUB(x[k], V1[k]);
        x2[k] = DSUB(x[k], V2[k]);
    }
    double t1[3], t2[3], t3[3];
    t1[0] = DSUB(DMUL(n1[1], x1[2]), DMUL(n1[2], x1[1]));
    t1[1] = DSUB(DMUL(n1[2], x1[0]), DMUL(n1[0], x1[2]));
    t1[2] = DSUB(DMUL(n1[0], x1[1]), DMUL(n1[1], x1[0]));
    t2[0] = DSUB(DMUL(n2[1], x2[2]), DMUL(n2[2], x2[1]));
    t2[1] = DSUB(DMUL(n2[2], x2[0]), DMUL(n2[0], x2[2]));
    t2[2] = DSUB(DMUL(n2[0], x2[1]), DMUL(n2[1], x2[0]));
    t3[0] = DSUB(DMUL(n3[1], x3[2]), DMUL(n3[2], x3[1]));
    t3[1] = DSUB(DMUL(n3[2], x3[0]), DMUL(n3[0], x3[2]));
    t3[2] = DSUB(DMUL(n3[0], x3[1]), DMUL(n3[1], x3[0]));
    const double c1 = DADD(DADD(DMUL(t1[0], Hn[0]), DMUL(t1[1], Hn[1])), DMUL(t1[2], Hn[2]));
    const double c2 = DADD(DADD(DMUL(t2[0], Hn[0]), DMUL(t2[1], Hn[1])), DMUL(t2[2], Hn[2]));
    const double c3 = DADD(DADD(DMUL(t3[0], Hn[0]), DMUL(t3[1], Hn[1])), DMUL(t3[2], Hn[2]));
    return (c1 >= 0.0 && c2 >= 0.0 && c3 >= 0.0) ? 0 : 1;
}

// the plain drivers' test, from the arrays
__device__ __forceinline__ int dev_shadowtest(const GeomArgs& a, int g, int h, int s) {
    const int ntau = a.s.ntau;
    return shadowtest(a.g.hm + ((size_t)g * ntau + s) * 3, a.g.hm + ((size_t)h * ntau + s) * 3,
                      a.g.nrm + ((size_t)h * ntau + s) * 3, vertex(a.g.hp, a.s.fac, ntau, h, 0, s),
                      vertex(a.g.hp, a.s.fac, ntau, h, 1, s), vertex(a.g.hp, a.s.fac, ntau, h, 2, s));
}

// the same test, and the sign of |g| - |h|, from the vertex positions
__device__ __noinline__ int exact_test(const double* hp, const int* fac, int ntau, int g, int h, int s) {
    double Gm[3], Hm[3], n[3], t;
    facet_frame(vertex(hp, fac, ntau, g, 0, s), vertex(hp, fac, ntau, g, 1, s), vertex(hp, fac, ntau, g, 2, s), Gm, n, &t);
    const double *V0 = vertex(hp, fac, ntau, h, 0, s), *V1 = vertex(hp, fac, ntau, h, 1, s),
                 *V2 = vertex(hp, fac, ntau, h, 2, s);
    facet_frame(V0, V1, V2, Hm, n, &t);
    return shadowtest(Gm, Hm, n, V0, V1, V2);
}

__device__ __noinline__ int exact_order(const double* hp, const int* fac, int ntau, int g, int h, int s) {
    double m[3], n[3], dg, dh;
    facet_frame(vertex(hp, fac, ntau, g, 0, s), vertex(hp, fac, ntau, g, 1, s), vertex(hp, fac, ntau, g, 2, s), m, n, &dg);
    facet_frame(vertex(hp, fac, ntau, h, 0, s), vertex(hp, fac, ntau, h, 1, s), vertex(hp, fac, ntau, h, 2, s), m, n, &dh);
    return dg > dh ? 1 : dh > dg ? -1 : 0;
}

// dependent-list shadowing; warp = 32 consecutive steps of one facet
__global__ void __launch_bounds__(256) k_shadow_dep(GeomArgs a) {
    const int nf = a.s.nf, ntau = a.s.ntau;
    const int g = blockIdx.y * blockDim.y + threadIdx.y;
    const int s = blockIdx.x * 32 + threadIdx.x;
    if (g >= nf) return;
    const int d0 = a.s.dep_ptr[g], d1 = a.s.dep_ptr[g + 1];
    if (d0 == d1) return;
    const bool valid = s < ntau;
    const size_t o = (size_t)g * ntau + (valid ? s : 0);
    bool lit = valid && a.s.shadow[o] == 1;
    const double gd = a.g.dist[o];
    for (int k = d0; k < d1; ++k) {
        if (!__any_sync(0xffffffffu, lit)) break;
        const int h = __ldg(&a.s.dep_idx[k]);
        if (lit) {
            const double hd = a.g.dist[(size_t)h * ntau + s];
            if (gd > hd && dev_shadowtest(a, g, h, s) == 0) lit = false;
        }
    }
    if (valid && !lit) a.s.shadow[o] = 0;
}

// all pairs: facet g is tested against every h with |h| < |g| (the reference
// loops g < h and tests whichever of the two is farther from the Sun; the
// outcome per facet is the same AND over occluders)
__global__ void __launch_bounds__(256) k_shadow_all(GeomArgs a) {
    const int nf = a.s.nf, ntau = a.s.ntau;
    const int g = blockIdx.y * blockDim.y + threadIdx.y;
    const int s = blockIdx.x * 32 + threadIdx.x;
    if (g >= nf) return;
    const bool valid = s < ntau;
    const size_t o = (size_t)g * ntau + (valid ? s : 0);
    bool lit = valid && a.s.shadow[o] == 1;
    const double gd = a.g.dist[o];
    for (int h = 0; h < nf; ++h) {
        if (!__any_sync(0xffffffffu, lit)) break;
        if (h == g) continue;
        if (lit) {
            const double hd = a.g.dist[(size_t)h * ntau + s];
            // pair (min,max): reference tests the farther facet when strictly
            // farther; for equal distances the higher index is tested
            const bool g_tested = (g < h) ? (gd > hd) : !(hd > gd);
            if (g_tested && dev_shadowtest(a, g, h, s) == 0) lit = false;
        }
    }
    if (valid && !lit) a.s.shadow[o] = 0;
}

// ------------------------------------------------------------- culled drivers
// a projected facet: its corners and their depths
struct Tri {
    float2 q0, q1, q2;
    float w0, w1, w2;
};
// a facet's midpoint: its projection, and its distance from the origin less the
// body's
struct Mid {
    float2 q;
    float r;
};

__device__ __forceinline__ Tri load_tri(const GeomArgs& a, const Proj& p, int f, int s) {
    const int* fv = a.s.fac + 3 * f;
    const size_t i0 = (size_t)fv[0] * a.s.ntau + s, i1 = (size_t)fv[1] * a.s.ntau + s, i2 = (size_t)fv[2] * a.s.ntau + s;
    return {p.uv[i0], p.uv[i1], p.uv[i2], p.w[i0], p.w[i1], p.w[i2]};
}

// With corners at depths w_i the midpoint projects to the mean of theirs weighted
// by scale + w_i, and lies (scale + w) sqrt(1 + t) from the origin, t the square of
// its projection over scale.  Both hold at any distance: plain means and the depth
// itself leave them by the square of the body's size over the distance, which an
// observer close by would need a margin of whole facets for.
__device__ __forceinline__ Mid middle(const Proj& p, const Tri& t) {
    const float p0 = 1.0f + t.w0 * p.inv, p1 = 1.0f + t.w1 * p.inv, p2 = 1.0f + t.w2 * p.inv;
    const float m = __fdividef(1.0f, p0 + p1 + p2), w = (t.w0 + t.w1 + t.w2) * (1.0f / 3.0f);
    const float x = (t.q0.x * p0 + t.q1.x * p1 + t.q2.x * p2) * m, y = (t.q0.y * p0 + t.q1.y * p1 + t.q2.y * p2) * m;
    const float u = x * p.inv, v = y * p.inv, sq = u * u + v * v;
    return {make_float2(x, y), w + (p.scale + w) * __fdividef(sq, 1.0f + sqrtf(1.0f + sq))};
}

__device__ __forceinline__ float4 tri_box(const Tri& t, float pad) {
    return make_float4(fminf(t.q0.x, fminf(t.q1.x, t.q2.x)) - pad, fmaxf(t.q0.x, fmaxf(t.q1.x, t.q2.x)) + pad,
                       fminf(t.q0.y, fminf(t.q1.y, t.q2.y)) - pad, fmaxf(t.q0.y, fmaxf(t.q1.y, t.q2.y)) + pad);
}

__device__ __forceinline__ bool in_box(float2 q, float4 b) {
    return q.x >= b.x && q.x <= b.y && q.y >= b.z && q.y <= b.w;
}

// edge function of a -> b at q over the edge's length bound |dx| + |dy|
__device__ __forceinline__ float edge_of(float2 a, float2 b, float2 q, float sign, float margin, float& clear) {
    const float dx = b.x - a.x, dy = b.y - a.y;
    const float e = (dx * (q.y - a.y) - dy * (q.x - a.x)) * sign;
    clear = margin * (fabsf(dx) + fabsf(dy));
    return e;
}

// 1: q lies in the triangle, 0: it does not, 2: within the margin of an edge, or
// the triangle is no wider than the margin: its orientation, on which every edge's
// side rests, is then a matter of rounding (an edge-on facet ten times as long as
// its short edge would hide nothing)
__device__ __forceinline__ int locate(const Tri& t, float2 q, float margin) {
    const float ax = t.q1.x - t.q0.x, ay = t.q1.y - t.q0.y, bx = t.q2.x - t.q0.x, by = t.q2.y - t.q0.y;
    const float area = ax * by - ay * bx;
    if (fabsf(area) <= margin * (fabsf(ax) + fabsf(ay) + fabsf(bx) + fabsf(by))) return 2;
    const float sign = area < 0.0f ? -1.0f : 1.0f;
    float c0, c1, c2;
    const float e0 = edge_of(t.q0, t.q1, q, sign, margin, c0), e1 = edge_of(t.q1, t.q2, q, sign, margin, c1),
                e2 = edge_of(t.q2, t.q0, q, sign, margin, c2);
    if (e0 < -c0 || e1 < -c1 || e2 < -c2) return 0;
    return (e0 > c0 && e1 > c1 && e2 > c2) ? 1 : 2;
}

// whether g, at distance gr from the origin, is the one tested against h at hr: the
// farther, and on equal distances the higher index where `ties`
__device__ __forceinline__ bool behind(const GeomArgs& a, const Proj& p, int g, int h, int s, float gr, float hr,
                                       bool ties) {
    const float d = gr - hr;
    if (d > p.margin) return true;
    if (d < -p.margin) return false;
    const int o = exact_order(a.g.hp, a.s.fac, a.s.ntau, g, h, s);  // sign of |g| - |h|
    return o > 0 || (o == 0 && ties && g > h);
}

// each facet's padded box over every window of 32 steps (the union of its
// 32 per-step boxes): a warp of the dependent-list driver covers one window,
// and an occluder whose window box misses the box around the warp's lit
// points cannot pass any lane's per-step box test.  One warp per facet and
// window.
__global__ void __launch_bounds__(256) k_window_box(GeomArgs a, Proj p) {
    const int ntau = a.s.ntau;
    const int h = blockIdx.y * blockDim.y + threadIdx.y, s = blockIdx.x * 32 + threadIdx.x;
    if (h >= a.s.nf) return;
    float4 u = tri_box(load_tri(a, p, h, min(s, ntau - 1)), p.pad);
    for (int o = 16; o > 0; o >>= 1) {
        u.x = fminf(u.x, __shfl_xor_sync(0xffffffffu, u.x, o));
        u.y = fmaxf(u.y, __shfl_xor_sync(0xffffffffu, u.y, o));
        u.z = fminf(u.z, __shfl_xor_sync(0xffffffffu, u.z, o));
        u.w = fmaxf(u.w, __shfl_xor_sync(0xffffffffu, u.w, o));
    }
    if (threadIdx.x == 0) p.wbox[(size_t)blockIdx.x * a.s.nf + h] = u;
}

// adds a thread's triangle-test count to the launch's tally: one add per group
// of lanes leaving together, spread over 64 counters
__device__ __forceinline__ void count_tests(unsigned long long* ctr, unsigned n) {
    if (!ctr) return;
    const unsigned m = __activemask();
    const unsigned t = __reduce_add_sync(m, n);
    unsigned lane;
    asm("mov.u32 %0, %%laneid;" : "=r"(lane));
    if (lane == (unsigned)(__ffs(m) - 1) && t) atomicAdd(&ctr[blockIdx.x & 63], (unsigned long long)t);
}

// dependent-list shadowing: a warp takes 32 steps of one facet.  32 list
// entries at a time, a lane each, are held against the box around the warp's
// lit points; the entries left are tested one by one, a lane per step.  Taking
// every entry in turn was bound by the loop's instructions (7.2 ms
// for 21,760 facets, 5.8 M entries, 720 steps; 1.2 ms now).  Three CTAs an SM
// rather than the two its free choice of registers leaves: 0.200 against 0.217 ms
// for 5,840 facets and 360 steps.
__global__ void __launch_bounds__(256, 3) k_shadow_dep_cull(GeomArgs a, Proj p) {
    const int nf = a.s.nf, ntau = a.s.ntau;
    const int g = blockIdx.y * blockDim.y + threadIdx.y;
    const int lane = threadIdx.x, s = blockIdx.x * 32 + lane;
    if (g >= nf) return;
    const int d0 = a.s.dep_ptr[g], d1 = a.s.dep_ptr[g + 1];
    if (d0 == d1) return;
    const bool valid = s < ntau;
    const int sc = valid ? s : ntau - 1;
    const size_t o = (size_t)g * ntau + sc;
    bool lit = valid && a.s.shadow[o] == 1;
    const Mid mg = middle(p, load_tri(a, p, g, sc));
    const float2 q = mg.q;
    unsigned ntest = 0;
    // the box around this warp's lit points (empty when none is lit)
    float4 qb = lit ? make_float4(q.x, q.x, q.y, q.y) : make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);
    for (int o2 = 16; o2 > 0; o2 >>= 1) {
        qb.x = fminf(qb.x, __shfl_xor_sync(0xffffffffu, qb.x, o2));
        qb.y = fmaxf(qb.y, __shfl_xor_sync(0xffffffffu, qb.y, o2));
        qb.z = fminf(qb.z, __shfl_xor_sync(0xffffffffu, qb.z, o2));
        qb.w = fmaxf(qb.w, __shfl_xor_sync(0xffffffffu, qb.w, o2));
    }
    const float4* wb = p.wbox ? p.wbox + (size_t)blockIdx.x * nf : nullptr;  // this warp's step window
    for (int k0 = d0; k0 < d1; k0 += 32) {
        if (!__any_sync(0xffffffffu, lit)) break;
        const bool have = k0 + lane < d1;
        const int mine = have ? __ldg(&a.s.dep_idx[k0 + lane]) : 0;
        const float4 u = wb ? __ldg(wb + mine) : make_float4(-INFINITY, INFINITY, -INFINITY, INFINITY);
        unsigned left = __ballot_sync(0xffffffffu, have && !(u.x > qb.y || u.y < qb.x || u.z > qb.w || u.w < qb.z));
        for (; left; left &= left - 1) {
            const int h = __shfl_sync(0xffffffffu, mine, __ffs(left) - 1);
            if (!lit) continue;
            const Tri th = load_tri(a, p, h, s);
            if (!in_box(q, tri_box(th, p.pad))) continue;
            // h's distance is its mean depth and up to `lift`: the depth settles most
            const float d = mg.r - (th.w0 + th.w1 + th.w2) * (1.0f / 3.0f);
            if (d < -p.margin || (d <= p.margin + p.lift && !behind(a, p, g, h, s, mg.r, middle(p, th).r, false))) continue;
            ++ntest;
            int hit = locate(th, q, p.margin);
            if (hit == 2) hit = exact_test(a.g.hp, a.s.fac, ntau, g, h, s) == 0;
            if (hit) lit = false;
        }
    }
    if (valid && !lit) a.s.shadow[o] = 0;
    count_tests(a.g.tests, ntest);
}

struct GridArgs {
    int G;          // cells per side
    float cell;     // cell size (km): three quarters of the largest box
    float origin;   // grid spans [origin, origin + G * cell) on both axes
    int s0, ns;     // steps of this chunk
    int* start;     // [ns][G*G + 1] first entry of each cell
    int* cursor;    // [ns][G*G]
    float4* tri;    // [ns][nf][2] corners, midpoint distance, lit flag
    float2* mid;    // [ns][nf] midpoints
    int* who;       // [ns][kCover nf] facets by cell
};
constexpr int kCover = 9;  // a box of at most two cells' size touches at most 3 x 3 cells

__device__ __forceinline__ int cell_of(const GridArgs& gr, float x) {
    int c = (int)floorf((x - gr.origin) / gr.cell);
    return c < 0 ? 0 : (c >= gr.G ? gr.G - 1 : c);
}

__global__ void __launch_bounds__(256) k_grid_extent(GeomArgs a, Proj p) {
    const int ntau = a.s.ntau;
    const long long n = (long long)a.s.nf * ntau, at = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = at < n ? at : n - 1;  // lanes beyond the end repeat the last facet
    const float4 b = tri_box(load_tri(a, p, (int)(i / ntau), (int)(i % ntau)), p.pad);
    warp_max_to(&p.stats[1], __float_as_uint(fmaxf(b.y - b.x, b.w - b.z)));
}

// the cells a box touches, in turn
template <class F>
__device__ __forceinline__ void for_cells(const GridArgs& gr, const float4& b, F&& f) {
    const int x0 = cell_of(gr, b.x), x1 = cell_of(gr, b.y), y0 = cell_of(gr, b.z), y1 = cell_of(gr, b.w);
    for (int y = y0; y <= y1; ++y)
        for (int x = x0; x <= x1; ++x) f(y * gr.G + x);
}

// lanes take consecutive steps of a facet: the projected vertices load as
// segments and no two lanes count into the same step's grid
__global__ void __launch_bounds__(256) k_grid_count(GeomArgs a, Proj p, GridArgs gr) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.s.nf * gr.ns) return;
    const int f = (int)(i / gr.ns), k = (int)(i % gr.ns);
    int* st = gr.start + (size_t)k * (gr.G * gr.G + 1) + 1;
    for_cells(gr, tri_box(load_tri(a, p, f, gr.s0 + k), p.pad), [&](int c) { atomicAdd(&st[c], 1); });
}

// in-place inclusive scan of start[k][1..G*G] (so start[k][c] = first entry of
// cell c), a block per step, 8 cells a thread and pass
__global__ void __launch_bounds__(1024) k_grid_scan(GridArgs gr) {
    __shared__ int part[32];
    const int n = gr.G * gr.G, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* st = gr.start + (size_t)blockIdx.x * (n + 1) + 1;
    int* cu = gr.cursor + (size_t)blockIdx.x * n;
    int carry = 0;
    for (int base = 0; base < n; base += 8192) {
        const int j0 = base + 8 * threadIdx.x;
        int v[8], sum = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            v[u] = j0 + u < n ? st[j0 + u] : 0;
            sum += v[u];
        }
        int inc = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) part[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            int w = part[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += t;
            }
            part[lane] = w;
        }
        __syncthreads();
        int at = carry + inc - sum + (warp ? part[warp - 1] : 0);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (j0 + u < n) {
                cu[j0 + u] = at;
                at += v[u];
                st[j0 + u] = at;
            }
        carry += part[31];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) k_grid_fill(GeomArgs a, Proj p, GridArgs gr) {
    const int nf = a.s.nf, ntau = a.s.ntau;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nf * gr.ns) return;
    const int f = (int)(i / gr.ns), k = (int)(i % gr.ns), s = gr.s0 + k;
    const Tri t = load_tri(a, p, f, s);
    const Mid m = middle(p, t);
    float4* d = gr.tri + 2 * ((size_t)k * nf + f);
    d[0] = make_float4(t.q0.x, t.q0.y, t.q1.x, t.q1.y);
    d[1] = make_float4(t.q2.x, t.q2.y, m.r, a.s.shadow[(size_t)f * ntau + s] == 1 ? 1.0f : 0.0f);
    gr.mid[(size_t)k * nf + f] = m.q;
    const float4 b = tri_box(t, p.pad);
    int* cu = gr.cursor + (size_t)k * gr.G * gr.G;
    const size_t first = (size_t)k * kCover * nf;
    for_cells(gr, b, [&](int c) {
        gr.who[first + atomicAdd(&cu[c], 1)] = f;
    });
}

// corners (no depths) and the midpoint's distance
__device__ __forceinline__ Tri stored_tri(const float4* t, float* r) {
    const float4 x = __ldg(t), y = __ldg(t + 1);
    *r = y.z;
    return {make_float2(x.x, x.y), make_float2(x.z, x.w), make_float2(y.x, y.y)};
}

// all pairs over the grid: a facet's box is filed in every cell it touches, so
// the candidates of g are the entries of the cell its projected midpoint lies
// in.  Threads take consecutive facets of a step, which lie near each other and
// share cells.  Filing each facet once in cells as wide as the largest box and
// taking the 3 x 3 cells around g gave some 400 candidates a point, each
// gathering its vertices: 38.7 ms for 21,760 facets and 720 steps (with the
// grid 39.9) against 2.2 ms
// (with the grid 4.0).
__global__ void __launch_bounds__(256, 4) k_shadow_grid(GeomArgs a, Proj p, GridArgs gr) {
    const int nf = a.s.nf, ntau = a.s.ntau;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nf * gr.ns) return;
    const int k = (int)(i / nf), g = (int)(i % nf), s = gr.s0 + k;
    const float4* tri = gr.tri + 2 * (size_t)k * nf;
    const float4 own = __ldg(tri + 2 * (size_t)g + 1);
    if (own.w == 0.0f) return;  // dark already
    const float2 q = __ldg(gr.mid + (size_t)k * nf + g);
    const int* st = gr.start + (size_t)k * (gr.G * gr.G + 1) + cell_of(gr, q.y) * gr.G + cell_of(gr, q.x);
    const size_t first = (size_t)k * kCover * nf;
    const int* who = gr.who + first;
    unsigned ntest = 0;
    const int end = st[1];
    int next = st[0] < end ? __ldg(who + st[0]) : 0;
    for (int j = st[0]; j < end; ++j) {
        const int h = next;
        if (j + 1 < end) next = __ldg(who + j + 1);
        float hr;
        const Tri th = stored_tri(tri + 2 * (size_t)h, &hr);
        if (!in_box(q, tri_box(th, p.pad)) || h == g || !behind(a, p, g, h, s, own.z, hr, true)) continue;
        ++ntest;
        int hit = locate(th, q, p.margin);
        if (hit == 2) hit = exact_test(a.g.hp, a.s.fac, ntau, g, h, s) == 0;
        if (hit) {
            a.s.shadow[(size_t)g * ntau + s] = 0;
            break;
        }
    }
    count_tests(a.g.tests, ntest);
}

namespace {
// projection frame of the body direction; returns false when the body is
// too close to the origin for a central projection (the caller then runs
// the plain drivers)
bool make_frame(const GeomWork& g, Proj& p) {
    const double n = sqrt(g.car[0] * g.car[0] + g.car[1] * g.car[1] + g.car[2] * g.car[2]);
    if (!(n > 0.0)) return false;
    double c[3], e1[3], e2[3];
    for (int k = 0; k < 3; ++k) c[k] = g.car[k] / n;
    // e1: the coordinate axis least aligned with c, made orthogonal
    int ax = 0;
    for (int k = 1; k < 3; ++k)
        if (fabs(c[k]) < fabs(c[ax])) ax = k;
    double t[3] = {0, 0, 0};
    t[ax] = 1.0;
    const double dt = t[0] * c[0] + t[1] * c[1] + t[2] * c[2];
    for (int k = 0; k < 3; ++k) e1[k] = t[k] - dt * c[k];
    const double n1 = sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
    for (int k = 0; k < 3; ++k) e1[k] /= n1;
    e2[0] = c[1] * e1[2] - c[2] * e1[1];
    e2[1] = c[2] * e1[0] - c[0] * e1[2];
    e2[2] = c[0] * e1[1] - c[1] * e1[0];
    for (int k = 0; k < 3; ++k) {
        p.c[k] = (float)c[k];
        p.e1[k] = (float)e1[k];
        p.e2[k] = (float)e2[k];
    }
    p.scale = (float)n;
    p.inv = (float)(1.0 / n);
    p.uv = reinterpret_cast<float2*>(g.uv);
    p.w = g.depth;
    p.stats = g.stats;
    return p.uv != nullptr;
}

size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// Most cells of a step's grid.  Two small bodies far apart would have millions of
// empty ones to clear and scan, one block a step: with a cell for every three
// quarters of the largest box 2,560 facets x 720 steps took 94 ms at 40 km apart
// and 294 at 400; with the cells kept to a few a facet 3.2 and 4.4 (8 a facet 3.2
// and 4.2, but 0.81 against 0.71 at 2.5 km; 4 a facet 4.0 and 5.4).
size_t most_cells(size_t nf) { return 12 * nf + 4096; }
// a step of the all-pairs grid of n cells: entries, corners, midpoints; the cells
size_t grid_step_bytes(size_t nf, size_t n) {
    return nf * (kCover * sizeof(int) + 2 * sizeof(float4) + sizeof(float2)) + (2 * n + 1) * sizeof(int);
}
// What the grid may take at once, in chunks of steps: up to 1.5 GB (21,760 facets x
// 720 steps take 1.3 GB; in three chunks of 512 MB they take 1 % longer), one step
// at least.
size_t grid_budget(int nf, int ntau) {
    const size_t all = (size_t)ntau * grid_step_bytes(nf, most_cells(nf) / 3);
    return std::max(std::min<size_t>(all, 1536u << 20), grid_step_bytes(nf, most_cells(nf)));
}
}  // namespace

size_t shadow_scratch_bytes(int nf, int ntau, bool all_pairs) {
    return all_pairs ? grid_budget(nf, ntau) + 5 * 256 : al256((size_t)((ntau + 31) / 32) * nf * sizeof(float4));
}

// returns 0 when the culled driver ran, -1 when the caller should fall back
int launch_shadow_culled(const DevSolve& s, const GeomWork& g, bool all_pairs, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    GeomArgs a{s, g};
    Proj p{};
    if (!make_frame(g, p)) return -1;
    const long long nft = (long long)s.nf * s.ntau;
    unsigned stats[5] = {};
    auto read_stats = [&]() {
        return cudaMemcpyAsync(stats, p.stats, sizeof stats, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
               cudaStreamSynchronize(st) == cudaSuccess;
    };
    if (!read_stats()) return 2;
    if (stats[2]) return -1;  // a vertex too far off the body direction: no projection
    float umax, wmax, front;
    memcpy(&umax, &stats[0], 4);
    memcpy(&wmax, &stats[3], 4);
    memcpy(&front, &stats[4], 4);
    // What FP32 may not decide (km): some 16 ulps of the largest coordinate, as the
    // perspective enlarges them (scale over the nearest vertex's depth, and the
    // body's size over its distance, 1 for all but the closest observers), and a
    // good part of a metre per 1e11 km for the FP64 test's own rounding (1.5 mm at
    // 1 AU, where its positions have ulps of 0.03 mm).  The boxes are padded by a
    // centimetre besides.
    const float size = umax > wmax ? umax : wmax, wide = 1.0f + size / p.scale;
    p.margin = std::min(size, 2e-6f * size * wide * wide / (1.0f - front / p.scale)) + 1e-14f * p.scale;
    p.lift = size * wide * (size / p.scale);
    p.pad = 1e-5f + p.margin;
    int rc = 0;
    if (!all_pairs) {
        const int nw = (s.ntau + 31) / 32;
        void* wm = nullptr;
        const dim3 blk(32, 8), grd(nw, (s.nf + 7) / 8);
        if (cudaMallocAsync(&wm, (size_t)nw * s.nf * sizeof(float4), st) == cudaSuccess) {
            p.wbox = static_cast<float4*>(wm);
            k_window_box<<<grd, blk, 0, st>>>(a, p);
        } else {
            cudaGetLastError();  // without window boxes: the per-step tests alone (same flags)
        }
        k_shadow_dep_cull<<<grd, blk, 0, st>>>(a, p);
        if (wm) cudaFreeAsync(wm, st);
    } else {
        k_grid_extent<<<(unsigned)((nft + 255) / 256), 256, 0, st>>>(a, p);
        if (!read_stats()) return 2;
        float ext;
        memcpy(&ext, &stats[1], 4);
        GridArgs gr{};
        gr.cell = 0.75f * ext + 1e-6f;
        gr.origin = -(umax + 2.0f * p.pad) - gr.cell;
        const int most = (int)sqrt((double)most_cells(s.nf));
        long long G = (long long)ceilf(2.0f * -gr.origin / gr.cell) + 1;
        if (G > most) {  // coarser cells: a box touches fewer of them
            G = most;
            gr.cell = 2.0f * -gr.origin / (float)(most - 2);
        }
        gr.G = (int)G;
        const size_t n = (size_t)G * G, entries = (size_t)kCover * s.nf;
        const int sc = (int)std::max<size_t>(1, std::min<size_t>(s.ntau, grid_budget(s.nf, s.ntau) / grid_step_bytes(s.nf, n)));
        const size_t b_st = al256((size_t)sc * (n + 1) * 4), b_cu = al256((size_t)sc * n * 4),
                     b_tri = al256((size_t)sc * s.nf * 2 * sizeof(float4)), b_who = al256(sc * entries * 4),
                     b_mid = al256((size_t)sc * s.nf * sizeof(float2));
        void* gm = nullptr;
        if (cudaMallocAsync(&gm, b_st + b_cu + b_tri + b_who + b_mid, st) != cudaSuccess) return 2;
        char* t = static_cast<char*>(gm);
        gr.start = reinterpret_cast<int*>(t);
        gr.cursor = reinterpret_cast<int*>(t + b_st);
        gr.tri = reinterpret_cast<float4*>(t + b_st + b_cu);
        gr.who = reinterpret_cast<int*>(t + b_st + b_cu + b_tri);
        gr.mid = reinterpret_cast<float2*>(t + b_st + b_cu + b_tri + b_who);
        for (int s0 = 0; s0 < s.ntau && !rc; s0 += sc) {
            gr.s0 = s0;
            gr.ns = std::min(sc, s.ntau - s0);
            const unsigned m = (unsigned)(((long long)s.nf * gr.ns + 255) / 256);
            cudaMemsetAsync(gr.start, 0, (size_t)gr.ns * (n + 1) * 4, st);
            k_grid_count<<<m, 256, 0, st>>>(a, p, gr);
            k_grid_scan<<<gr.ns, 1024, 0, st>>>(gr);
            k_grid_fill<<<m, 256, 0, st>>>(a, p, gr);
            k_shadow_grid<<<m, 256, 0, st>>>(a, p, gr);
            if (cudaGetLastError() != cudaSuccess) rc = 2;
        }
        cudaFreeAsync(gm, st);
    }
    if (cudaGetLastError() != cudaSuccess) rc = 2;
    return rc;
}

// The Sun direction in every facet's local frame, the crater model's input
// (asteroidgeometry, 3905/Thermal/NominalPole/main.cpp:967-1030): frame rows
// = the first edge (unit), normal x edge, the unit normal; the vector is
// -frame . heliocentric midpoint, scaled to length 10^4 and rounded to float.
// The facet's final shadow flag (self-shadow and astshadow) goes beside it.
// Facets f0 .. f0 + nfc - 1; outputs [nfc][ntau][3] and [nfc][ntau].
__global__ void __launch_bounds__(256) k_crater_sun(GeomArgs a, int f0, int nfc, float* sun, int* shadow) {
    const int ntau = a.s.ntau;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nfc * ntau) return;
    const int fl = (int)(i / ntau), s = (int)(i % ntau), f = f0 + fl;
    const int* fv = a.s.fac + 3 * f;
    const double* h0 = a.g.hp + ((size_t)fv[0] * ntau + s) * 3;
    const double* h1 = a.g.hp + ((size_t)fv[1] * ntau + s) * 3;
    const double* h2 = a.g.hp + ((size_t)fv[2] * ntau + s) * 3;
    double hm[3], n[3], nc0[3], nc1[3], y[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        hm[k] = DDIV(DADD(DADD(h0[k], h1[k]), h2[k]), 3.0);
        nc0[k] = DSUB(h1[k], h0[k]);
        nc1[k] = DSUB(h2[k], h0[k]);
    }
    const double t = __dsqrt_rn(DADD(DADD(DMUL(hm[0], hm[0]), DMUL(hm[1], hm[1])), DMUL(hm[2], hm[2])));
    n[0] = DSUB(DMUL(nc0[1], nc1[2]), DMUL(nc0[2], nc1[1]));
    n[1] = DSUB(DMUL(nc0[2], nc1[0]), DMUL(nc0[0], nc1[2]));
    n[2] = DSUB(DMUL(nc0[0], nc1[1]), DMUL(nc0[1], nc1[0]));
    const double nn = __dsqrt_rn(DADD(DADD(DMUL(n[0], n[0]), DMUL(n[1], n[1])), DMUL(n[2], n[2])));
    const double x = __dsqrt_rn(DADD(DADD(DMUL(nc0[0], nc0[0]), DMUL(nc0[1], nc0[1])), DMUL(nc0[2], nc0[2])));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        n[k] = DDIV(n[k], nn);
        nc0[k] = DDIV(nc0[k], x);
    }
    y[0] = DSUB(DMUL(n[1], nc0[2]), DMUL(n[2], nc0[1]));
    y[1] = DSUB(DMUL(n[2], nc0[0]), DMUL(n[0], nc0[2]));
    y[2] = DSUB(DMUL(n[0], nc0[1]), DMUL(n[1], nc0[0]));
    const double* row[3] = {nc0, y, n};
    float* out = sun + ((size_t)fl * ntau + s) * 3;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double iv = -DADD(DADD(DMUL(row[k][0], hm[0]), DMUL(row[k][1], hm[1])), DMUL(row[k][2], hm[2]));
        out[k] = (float)DDIV(DMUL(10000.0, iv), t);
    }
    shadow[(size_t)fl * ntau + s] = a.s.shadow[(size_t)f * ntau + s];
}

int launch_crater_sun(const DevSolve& s, const GeomWork& g, int f0, int nfc, float* sun, int* shadow, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    GeomArgs a{s, g};
    const long long nvt = (long long)s.nv * s.ntau, nct = (long long)nfc * s.ntau;
    k_geom_vertices<<<(unsigned)((nvt + 255) / 256), 256, 0, st>>>(a, Proj{});
    k_crater_sun<<<(unsigned)((nct + 255) / 256), 256, 0, st>>>(a, f0, nfc, sun, shadow);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_geometry(const DevSolve& s, const GeomWork& g, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    GeomArgs a{s, g};
    const long long nvt = (long long)s.nv * s.ntau, nft = (long long)s.nf * s.ntau;
    Proj p{};
    if (!make_frame(g, p)) p.uv = nullptr;
    if (p.uv && cudaMemsetAsync(p.stats, 0, 5 * sizeof(unsigned), st) != cudaSuccess) return 2;
    k_geom_vertices<<<(unsigned)((nvt + 255) / 256), 256, 0, st>>>(a, p);
    if (s.mode == MODE_FP64) k_geom_facets<MODE_FP64><<<(unsigned)((nft + 255) / 256), 256, 0, st>>>(a);
    else if (s.mode == MODE_FAST) k_geom_facets<MODE_FAST><<<(unsigned)((nft + 255) / 256), 256, 0, st>>>(a);
    else k_geom_facets<MODE_REF><<<(unsigned)((nft + 255) / 256), 256, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_geometry_arrays(const DevSolve& s, const GeomWork& g, stream_t stv) {
    const long long nft = (long long)s.nf * s.ntau;
    k_geom_arrays<<<(unsigned)((nft + 255) / 256), 256, 0, static_cast<cudaStream_t>(stv)>>>(GeomArgs{s, g});
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_shadow_deplist(const DevSolve& s, const GeomWork& g, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    GeomArgs a{s, g};
    dim3 blk(32, 8), grd((s.ntau + 31) / 32, (s.nf + 7) / 8);
    k_shadow_dep<<<grd, blk, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_shadow_allpairs(const DevSolve& s, const GeomWork& g, stream_t stv) {
    cudaStream_t st = static_cast<cudaStream_t>(stv);
    GeomArgs a{s, g};
    dim3 blk(32, 8), grd((s.ntau + 31) / 32, (s.nf + 7) / 8);
    k_shadow_all<<<grd, blk, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace atpm
