// Facet-to-facet view factors (the reference's Shape_Selfheating stage,
// 3905/Shape_Selfheating/main.cpp).  FP32 throughout, like the reference,
// with round-to-nearest intrinsics in its operand order.
//
//   k_vf_count   per facet I: number of facets J with both normals facing
//                (thetai, thetaj <= pi/2 via acos, main.cpp:653-665)
//   k_vf_fill    the same screen, writing J in index order with
//                vf = cos(ti) cos(tj) A_J / (pi d^2) and the area-weighted
//                direction (main.cpp:700-735); an ordered block compaction
//                keeps the reference's list order
//   k_vf_hidden  occlusion culling (main.cpp:187-368): candidate Z of facet G
//                is dropped when another candidate S, nearer to Z than G,
//                intersects the segment; only pairs whose directions from G
//                come near enough go to the test
//   k_vf_keep_count, k_vf_compact  the lists that remain, in order
//   k_vf_refine  10x10 sub-triangle refinement of every pair with
//                vf >= 0.05 (main.cpp:374-622)
//   k_vf_photo   photon-momentum vectors (main.cpp:824-835)
//
// The facing test and cos(theta) go through the device's acosf/cosf, so a
// pair whose cos is within ~1e-7 of zero may be classified differently from
// the reference and view factors agree to float rounding (the reference
// writes them with 6 significant digits).
#include <cuda_runtime.h>

#include <cstdint>

namespace atpm {

#define FADD __fadd_rn
#define FSUB __fsub_rn
#define FMUL __fmul_rn
#define FDIV __fdiv_rn
#define FSQRT __fsqrt_rn

struct VfGeom {
    int nv, nf;
    const float* v;      // [nv][3]
    const int* fac;      // [nf][3]
    float* mid;          // [nf][3]
    float* nrm;          // [nf][3] un-normalised (v1-v0)x(v2-v0)
    float* area;         // [nf]
    float* nlen;         // [nf] |nrm|
};

__constant__ float c_PIF = 3.14159274101257324f;  // 4.0f*atan(1.0f) (main.cpp:8)

// initialise (main.cpp:750-811)
__global__ void k_vf_init(VfGeom g) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.nf) return;
    const float* a = g.v + 3 * g.fac[3 * c];
    const float* b = g.v + 3 * g.fac[3 * c + 1];
    const float* d = g.v + 3 * g.fac[3 * c + 2];
    float n0[3], n1[3], n[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        g.mid[3 * c + k] = FDIV(FADD(FADD(a[k], b[k]), d[k]), 3.0f);
        n0[k] = FSUB(b[k], a[k]);
        n1[k] = FSUB(d[k], a[k]);
    }
    n[0] = FSUB(FMUL(n0[1], n1[2]), FMUL(n0[2], n1[1]));
    n[1] = FSUB(FMUL(n0[2], n1[0]), FMUL(n0[0], n1[2]));
    n[2] = FSUB(FMUL(n0[0], n1[1]), FMUL(n0[1], n1[0]));
    const float l = FSQRT(FADD(FADD(FMUL(n[0], n[0]), FMUL(n[1], n[1])), FMUL(n[2], n[2])));
    g.area[c] = FDIV(l, 2.0f);
    g.nlen[c] = l;
#pragma unroll
    for (int k = 0; k < 3; ++k) g.nrm[3 * c + k] = n[k];
}

struct PairEval {
    bool facing;
    float vf, dir[3];
};

// main.cpp:700-735 for one (I, J)
__device__ __forceinline__ PairEval pair_eval(const VfGeom& g, int I, int J, bool want_vf) {
    PairEval r;
    float s[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) s[k] = FSUB(g.mid[3 * J + k], g.mid[3 * I + k]);
    const float d = FSQRT(FADD(FADD(FMUL(s[0], s[0]), FMUL(s[1], s[1])), FMUL(s[2], s[2])));
    const float ni = g.nlen[I], nj = g.nlen[J];
    const float* nI = g.nrm + 3 * I;
    const float* nJ = g.nrm + 3 * J;
    const float xi = FDIV(FADD(FADD(FMUL(nI[0], s[0]), FMUL(nI[1], s[1])), FMUL(nI[2], s[2])), FMUL(ni, d));
    const float xj = FDIV(FADD(FADD(FMUL(-nJ[0], s[0]), FMUL(-nJ[1], s[1])), FMUL(-nJ[2], s[2])), FMUL(nj, d));
    const float ti = acosf(xi), tj = acosf(xj);
    const float half = FDIV(c_PIF, 2.0f);
    r.facing = (ti <= half) && (tj <= half);
    if (r.facing && want_vf) {
        float vf = FDIV(FMUL(FMUL(cosf(ti), cosf(tj)), g.area[J]), FMUL(FMUL(c_PIF, d), d));
        if (vf < 0.0f) vf = 0.0f;
        r.vf = vf;
        const float aI = g.area[I];
#pragma unroll
        for (int k = 0; k < 3; ++k) r.dir[k] = FMUL(FMUL(aI, vf), FDIV(s[k], d));
    }
    return r;
}

__global__ void __launch_bounds__(256) k_vf_count(VfGeom g, int* count) {
    const int I = blockIdx.x;
    int c = 0;
    for (int J = threadIdx.x; J < g.nf; J += blockDim.x)
        if (J != I && pair_eval(g, I, J, false).facing) ++c;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    __shared__ int ws[8];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
        count[I] = t;
    }
}

// ordered fill: 256 candidates per round, ballot + warp prefix keeps J order
__global__ void __launch_bounds__(256) k_vf_fill(VfGeom g, const long long* ptr, int* idx, float* vf, float* dir) {
    const int I = blockIdx.x;
    __shared__ int woff[9];
    long long base = ptr[I];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int J0 = 0; J0 < g.nf; J0 += blockDim.x) {
        const int J = J0 + threadIdx.x;
        PairEval p;
        p.facing = false;
        if (J < g.nf && J != I) p = pair_eval(g, I, J, true);
        const unsigned m = __ballot_sync(0xffffffffu, p.facing);
        if (lane == 0) woff[w] = __popc(m);
        __syncthreads();
        if (threadIdx.x == 0) {
            int acc = 0;
            for (int k = 0; k < 8; ++k) { const int t = woff[k]; woff[k] = acc; acc += t; }
            woff[8] = acc;
        }
        __syncthreads();
        if (p.facing) {
            const long long o = base + woff[w] + __popc(m & ((1u << lane) - 1u));
            idx[o] = J;
            vf[o] = p.vf;
            dir[3 * o] = p.dir[0];
            dir[3 * o + 1] = p.dir[1];
            dir[3 * o + 2] = p.dir[2];
        }
        base += woff[8];
        __syncthreads();
    }
}

// one (Z, S) test of hidden (main.cpp:187-368) in its operand order: candidate
// S, nearer to Z than G is, intersects the segment's line beyond Z
__device__ __forceinline__ bool hides(const VfGeom& g, int G, int Z, int S) {
    if (S == G || S == Z) return false;
    const float *Gm = g.mid + 3 * G, *zm = g.mid + 3 * Z, *sm = g.mid + 3 * S, *nS = g.nrm + 3 * S;
    float gv[3], sv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        gv[k] = FSUB(Gm[k], zm[k]);
        sv[k] = FSUB(sm[k], zm[k]);
    }
    const float gl = FSQRT(FADD(FADD(FMUL(gv[0], gv[0]), FMUL(gv[1], gv[1])), FMUL(gv[2], gv[2])));
    const float sl = FSQRT(FADD(FADD(FMUL(sv[0], sv[0]), FMUL(sv[1], sv[1])), FMUL(sv[2], sv[2])));
    if (!(gl > sl)) return false;
    const float tc1 = FADD(FADD(FMUL(sv[0], nS[0]), FMUL(sv[1], nS[1])), FMUL(sv[2], nS[2]));
    const float tc2 = FADD(FADD(FMUL(gv[0], nS[0]), FMUL(gv[1], nS[1])), FMUL(gv[2], nS[2]));
    const float t = FDIV(tc1, tc2);
    if (!(t > 0.0f)) return false;
    const int* fv = g.fac + 3 * S;
    const float *V0 = g.v + 3 * fv[0], *V1 = g.v + 3 * fv[1], *V2 = g.v + 3 * fv[2];
    float x1[3], x2[3], x3[3], c1[3], c2[3], c3[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float x = FADD(FMUL(t, gv[k]), zm[k]);
        x1[k] = FSUB(x, V0[k]);
        x3[k] = FSUB(x, V1[k]);
        x2[k] = FSUB(x, V2[k]);
        c1[k] = FSUB(V1[k], V0[k]);   // normcalc1
        c2[k] = -FSUB(V2[k], V0[k]);  // normcalc2 = -(v2-v0)
        c3[k] = FSUB(V2[k], V1[k]);   // normcalc3
    }
    float t1[3], t2[3], t3[3];
    t1[0] = FSUB(FMUL(c1[1], x1[2]), FMUL(c1[2], x1[1]));
    t1[1] = FSUB(FMUL(c1[2], x1[0]), FMUL(c1[0], x1[2]));
    t1[2] = FSUB(FMUL(c1[0], x1[1]), FMUL(c1[1], x1[0]));
    t2[0] = FSUB(FMUL(c2[1], x2[2]), FMUL(c2[2], x2[1]));
    t2[1] = FSUB(FMUL(c2[2], x2[0]), FMUL(c2[0], x2[2]));
    t2[2] = FSUB(FMUL(c2[0], x2[1]), FMUL(c2[1], x2[0]));
    t3[0] = FSUB(FMUL(c3[1], x3[2]), FMUL(c3[2], x3[1]));
    t3[1] = FSUB(FMUL(c3[2], x3[0]), FMUL(c3[0], x3[2]));
    t3[2] = FSUB(FMUL(c3[0], x3[1]), FMUL(c3[1], x3[0]));
    const float q1 = FADD(FADD(FMUL(t1[0], nS[0]), FMUL(t1[1], nS[1])), FMUL(t1[2], nS[2]));
    const float q2 = FADD(FADD(FMUL(t2[0], nS[0]), FMUL(t2[1], nS[1])), FMUL(t2[2], nS[2]));
    const float q3 = FADD(FADD(FMUL(t3[0], nS[0]), FMUL(t3[1], nS[1])), FMUL(t3[2], nS[2]));
    return q1 >= 0.0f && q2 >= 0.0f && q3 >= 0.0f;
}

// Occlusion culling, one block per facet G.  Seen from G, S can only hide Z if
// the line G-Z passes S's midpoint within S's radius: |d_Z . d_S| of the unit
// directions is at least cos of S's angular radius (either way along the line,
// as the test does not bound the intersection to the segment).  That takes
// three multiply-adds a pair; the radius is widened by 1e-5 of the shape's size
// (the test's own rounding is some 1e-7 of it) and the cosine by 2e-6 (its rounding is 4e-7).  The pairs
// left are queued per warp and taken to the test 32 at a time.  Every pair
// through the test, its operands staged in shared memory, took 13.6 ms for 6,400
// facets (6.8e9 pairs) against 1.7 ms; now bound by the multiply-adds' issue.
constexpr int HID_CHUNK = 256;   // occluders staged at a time
constexpr int HID_Z = 4;         // candidates a thread holds
__global__ void __launch_bounds__(256) k_vf_hidden(VfGeom g, float size, const long long* ptr, const int* idx,
                                                   uint8_t* keep) {
    const int G = blockIdx.x;
    const long long p0 = ptr[G];
    const int D = (int)(ptr[G + 1] - p0);
    if (D == 0) return;
    __shared__ float4 cone[HID_CHUNK];
    __shared__ uint8_t hidden[HID_Z * 256];
    __shared__ int2 queue[8][64];  // {candidate within the block's span, occluder}
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int* list = idx + p0;
    const float gx = g.mid[3 * G], gy = g.mid[3 * G + 1], gz = g.mid[3 * G + 2];
    // unit direction from G to facet f's midpoint, and its distance
    auto toward = [&](int f, float& d) {
        const float x = g.mid[3 * f] - gx, y = g.mid[3 * f + 1] - gy, z = g.mid[3 * f + 2] - gz;
        d = sqrtf(x * x + y * y + z * z);
        const float r = 1.0f / d;
        return make_float3(x * r, y * r, z * r);
    };
    for (int z0 = 0; z0 < D; z0 += HID_Z * 256) {
        float3 dz[HID_Z];
#pragma unroll
        for (int u = 0; u < HID_Z; ++u) {
            const int zi = z0 + u * 256 + tid;
            float d;
            // beyond the list: a direction no cone holds
            dz[u] = zi < D ? toward(list[zi], d) : make_float3(0.0f, 0.0f, 0.0f);
            hidden[u * 256 + tid] = zi < D ? 0 : 1;
        }
        const int live = min(HID_Z, (D - z0 - warp * 32 + 255) / 256);  // spans holding one of this warp's candidates
        int queued = 0;
        auto drain = [&](int n) {  // the last n queued pairs, a lane each
            __syncwarp();
            if (lane < n) {
                const int2 q = queue[warp][queued - n + lane];
                if (!hidden[q.x] && hides(g, G, list[z0 + q.x], q.y)) hidden[q.x] = 1;
            }
            __syncwarp();
            queued -= n;
        };
        for (int s0 = 0; s0 < D; s0 += HID_CHUNK) {
            const int n = min(HID_CHUNK, D - s0);
            __syncthreads();
            if (tid < n) {
                const int S = list[s0 + tid];
                float d, r2 = 0.0f;
                const float3 u = toward(S, d);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float* V = g.v + 3 * g.fac[3 * S + k];
                    const float x = V[0] - g.mid[3 * S], y = V[1] - g.mid[3 * S + 1], z = V[2] - g.mid[3 * S + 2];
                    r2 = fmaxf(r2, x * x + y * y + z * z);
                }
                const float sine = (sqrtf(r2) + 1e-5f * size) / d;
                // not a number or no cone: every direction
                cone[tid] = make_float4(u.x, u.y, u.z, sine < 1.0f ? sqrtf(1.0f - sine * sine) - 2e-6f : -1.0f);
            }
            __syncthreads();
            if (live <= 0) continue;
            for (int j = 0; j < n; ++j) {
                const float4 c = cone[j];
#pragma unroll
                for (int u = 0; u < HID_Z; ++u) {
                    if (u >= live) break;
                    const float dot = dz[u].x * c.x + dz[u].y * c.y + dz[u].z * c.z;
                    // written so that a NaN passes
                    const unsigned m = __ballot_sync(0xffffffffu, !(fabsf(dot) < c.w));
                    if (m == 0) continue;
                    if ((m >> lane) & 1u)
                        queue[warp][queued + __popc(m & ((1u << lane) - 1u))] = make_int2(u * 256 + tid, list[s0 + j]);
                    queued += __popc(m);
                    if (queued >= 32) drain(32);
                }
            }
        }
        drain(queued);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < HID_Z; ++u) {
            const int zi = z0 + u * 256 + tid;
            if (zi < D) keep[p0 + zi] = hidden[u * 256 + tid] ? 0 : 1;
        }
    }
}

// the kept candidates of each row, in order: their number, then (rows scanned
// into optr) the entries themselves; a warp per row
__global__ void __launch_bounds__(256) k_vf_keep_count(int nf, const long long* ptr, const uint8_t* keep, int* count) {
    const int f = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (f >= nf) return;
    int n = 0;
    for (long long k = ptr[f] + lane; k < ptr[f + 1]; k += 32) n += keep[k];
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (lane == 0) count[f] = n;
}

__global__ void __launch_bounds__(256) k_vf_compact(int nf, const long long* ptr, const uint8_t* keep, const int* idx,
                                                    const float* vf, const float* dir, const long long* optr, int* oidx,
                                                    float* ovf, float* odir) {
    const int f = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (f >= nf) return;
    long long out = optr[f];
    const long long k1 = ptr[f + 1];
    for (long long k0 = ptr[f]; k0 < k1; k0 += 32) {
        const long long k = k0 + lane;
        const bool take = k < k1 && keep[k];
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (take) {
            const long long o = out + __popc(m & ((1u << lane) - 1u));
            oidx[o] = idx[k];
            ovf[o] = vf[k];
#pragma unroll
            for (int c = 0; c < 3; ++c) odir[3 * o + c] = dir[3 * k + c];
        }
        out += __popc(m);
    }
}

// photon-momentum vectors (main.cpp:824-835): each row's directions over the
// facet's area, summed in list order.  A warp per row: 32 entries are read and
// divided at a time, the next 32 on their way, and three lanes add the
// components up.  A thread per row and component, each with its own strided
// loads and divisions between the additions: 407 us for 6,400 facets with
// 1.7 M entries, now 25.
__global__ void __launch_bounds__(128) k_vf_photo(VfGeom g, const long long* ptr, const float* dir, float* photo) {
    __shared__ float over[4][96];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, f = blockIdx.x * 4 + warp;
    if (f >= g.nf) return;
    const long long p0 = 3 * ptr[f], p1 = 3 * ptr[f + 1];
    const float area = g.area[f];
    float* q = over[warp];
    float t = 0.0f, next[3];
    auto fetch = [&](long long p) {
#pragma unroll
        for (int u = 0; u < 3; ++u) next[u] = p + lane + 32 * u < p1 ? dir[p + lane + 32 * u] : 0.0f;
    };
    fetch(p0);
    for (long long p = p0; p < p1; p += 96) {
#pragma unroll
        for (int u = 0; u < 3; ++u) q[lane + 32 * u] = FDIV(next[u], area);
        __syncwarp();
        fetch(p + 96);
        if (lane < 3) {
            if (p + 96 <= p1) {
#pragma unroll
                for (int j = 0; j < 32; ++j) t = FADD(t, q[3 * j + lane]);
            } else {
                for (int j = lane; p + j < p1; j += 3) t = FADD(t, q[j]);
            }
        }
        __syncwarp();
    }
    if (lane < 3) photo[3 * f + lane] = t;
}

// 10x10 refinement (main.cpp:374-622) of pairs with vf >= 0.05.  One block
// per facet I; thread j < 100 owns sub-facet j of I.
__global__ void __launch_bounds__(128) k_vf_refine(VfGeom g, const long long* ptr, const int* idx, float* vf, float* dir) {
    const int I = blockIdx.x;
    const long long p0 = ptr[I], p1 = ptr[I + 1];
    constexpr int n = 10, SUBF = n * n, SUBV = (n + 1) * (n + 2) / 2;
    __shared__ float v1[SUBV][3], v2[SUBV][3];
    __shared__ int tf[SUBF][3];
    __shared__ float m1[SUBF][3], m2[SUBF][3];
    __shared__ float tot[SUBF], totv[SUBF][3];
    // sub-facet connectivity (identical for both triangles, main.cpp:486-543)
    if (threadIdx.x == 0) {
        int l = 0;
        for (int j = 1; j != n + 1; j++) {
            if (j != 1) {
                for (int k = 1; k != j; k++) {
                    tf[l][0] = ((j * (j - 1)) / 2) + k; tf[l][1] = ((j * (j - 1)) / 2) + k - 1; tf[l][2] = ((j * (j + 1)) / 2) + k - 1;
                    ++l;
                    tf[l][0] = ((j * (j + 1)) / 2) + k - 1; tf[l][1] = ((j * (j + 1)) / 2) + k; tf[l][2] = ((j * (j - 1)) / 2) + k;
                    ++l;
                }
            }
            tf[l][0] = (((j + 1) * (j + 2)) / 2) - 2; tf[l][1] = (((j + 1) * (j + 2)) / 2) - 1; tf[l][2] = ((j * (j + 1)) / 2) - 1;
            ++l;
        }
    }
    const float* nI = g.nrm + 3 * I;
    const float ni = g.nlen[I];
    const float aI = g.area[I];
    const float sub1 = FDIV(aI, (float)(n * n));
    const int* fI = g.fac + 3 * I;
    for (long long e = p0; e < p1; ++e) {
        if (!(vf[e] >= 0.05f)) continue;
        const int J = idx[e];
        const int* fJ = g.fac + 3 * J;
        const float* nJ = g.nrm + 3 * J;
        const float nj = g.nlen[J];
        const float sub2 = FDIV(g.area[J], (float)(n * n));
        __syncthreads();
        // sub-vertex tables (main.cpp:466-484)
        for (int t = threadIdx.x; t < SUBV; t += blockDim.x) {
            int l = 0, jj = 1, kk = 1;
            for (int j = 1; j != n + 2; j++)
                for (int k = 1; k != j + 1; k++) { if (l == t) { jj = j; kk = k; } ++l; }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float a1 = FDIV(FSUB(g.v[3 * fI[1] + c], g.v[3 * fI[0] + c]), (float)n);
                const float b1 = FDIV(FSUB(g.v[3 * fI[2] + c], g.v[3 * fI[0] + c]), (float)n);
                const float a2 = FDIV(FSUB(g.v[3 * fJ[1] + c], g.v[3 * fJ[0] + c]), (float)n);
                const float b2 = FDIV(FSUB(g.v[3 * fJ[2] + c], g.v[3 * fJ[0] + c]), (float)n);
                v1[t][c] = FSUB(FADD(g.v[3 * fI[2] + c], FMUL((float)(kk - 1), a1)), FMUL((float)(jj - 1), b1));
                v2[t][c] = FSUB(FADD(g.v[3 * fJ[2] + c], FMUL((float)(kk - 1), a2)), FMUL((float)(jj - 1), b2));
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < SUBF; t += blockDim.x)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                m1[t][c] = FDIV(FADD(FADD(v1[tf[t][0]][c], v1[tf[t][1]][c]), v1[tf[t][2]][c]), 3.0f);
                m2[t][c] = FDIV(FADD(FADD(v2[tf[t][0]][c], v2[tf[t][1]][c]), v2[tf[t][2]][c]), 3.0f);
            }
        __syncthreads();
        if (threadIdx.x < SUBF) {
            const int j = threadIdx.x;
            float T = 0.0f, TV[3] = {0.0f, 0.0f, 0.0f};
            for (int k = 0; k != SUBF; k++) {
                float s[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) s[c] = FSUB(m2[k][c], m1[j][c]);
                const float d = FSQRT(FADD(FADD(FMUL(s[0], s[0]), FMUL(s[1], s[1])), FMUL(s[2], s[2])));
                const float ci = FDIV(FADD(FADD(FMUL(nI[0], s[0]), FMUL(nI[1], s[1])), FMUL(nI[2], s[2])), FMUL(ni, d));
                const float cj = FDIV(FADD(FADD(FMUL(-nJ[0], s[0]), FMUL(-nJ[1], s[1])), FMUL(-nJ[2], s[2])), FMUL(nj, d));
                float v = FDIV(FMUL(FMUL(ci, cj), sub2), FMUL(FMUL(c_PIF, d), d));
                if (v < 0.0f) v = 0.0f;
                T = FADD(T, v);
#pragma unroll
                for (int c = 0; c < 3; ++c) TV[c] = FADD(TV[c], FMUL(v, FDIV(s[c], d)));
            }
            tot[j] = T;
#pragma unroll
            for (int c = 0; c < 3; ++c) totv[j][c] = TV[c];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            float ef = 0.0f, ev[3] = {0.0f, 0.0f, 0.0f};
            for (int j = 0; j != SUBF; j++) {
                ef = FADD(ef, FMUL(FDIV(sub1, aI), tot[j]));
#pragma unroll
                for (int c = 0; c < 3; ++c) ev[c] = FADD(ev[c], FMUL(sub1, totv[j][c]));
            }
            vf[e] = ef;
#pragma unroll
            for (int c = 0; c < 3; ++c) dir[3 * e + c] = ev[c];
        }
    }
}

// ------------------------------------------------------------------ launchers
struct VfBuffers {
    VfGeom g;
};

int vf_init(const VfGeom& g, cudaStream_t st) {
    k_vf_init<<<(g.nf + 127) / 128, 128, 0, st>>>(g);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
int vf_count(const VfGeom& g, int* count, cudaStream_t st) {
    k_vf_count<<<g.nf, 256, 0, st>>>(g, count);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
int vf_fill(const VfGeom& g, const long long* ptr, int* idx, float* vf, float* dir, cudaStream_t st) {
    k_vf_fill<<<g.nf, 256, 0, st>>>(g, ptr, idx, vf, dir);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
int vf_hidden(const VfGeom& g, float size, const long long* ptr, const int* idx, uint8_t* keep, int* kept,
              cudaStream_t st) {
    k_vf_hidden<<<g.nf, 256, 0, st>>>(g, size, ptr, idx, keep);
    k_vf_keep_count<<<(g.nf + 7) / 8, 256, 0, st>>>(g.nf, ptr, keep, kept);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
int vf_compact(const VfGeom& g, const long long* ptr, const uint8_t* keep, const int* idx, const float* vf,
               const float* dir, const long long* optr, int* oidx, float* ovf, float* odir, cudaStream_t st) {
    k_vf_compact<<<(g.nf + 7) / 8, 256, 0, st>>>(g.nf, ptr, keep, idx, vf, dir, optr, oidx, ovf, odir);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
int vf_photo(const VfGeom& g, const long long* ptr, const float* dir, float* photo, cudaStream_t st) {
    k_vf_photo<<<(g.nf + 3) / 4, 128, 0, st>>>(g, ptr, dir, photo);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
int vf_refine(const VfGeom& g, const long long* ptr, const int* idx, float* vf, float* dir, cudaStream_t st) {
    k_vf_refine<<<g.nf, 128, 0, st>>>(g, ptr, idx, vf, dir);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace atpm
