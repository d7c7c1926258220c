// Host side of the view-factor precompute (Shape_Selfheating,
// 3905/Shape_Selfheating/main.cpp:817-889): drives the kernels of
// atpm_viewfactor.cu.  Lists, view factors and vectors stay on the device until
// atpm_viewfactors_get copies them to the caller's arrays.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "../../include/atpm.h"

namespace atpm {
struct VfGeom {
    int nv, nf;
    const float* v;
    const int* fac;
    float* mid;
    float* nrm;
    float* area;
    float* nlen;
};
int vf_init(const VfGeom& g, cudaStream_t st);
int vf_count(const VfGeom& g, int* count, cudaStream_t st);
int vf_fill(const VfGeom& g, const long long* ptr, int* idx, float* vf, float* dir, cudaStream_t st);
int vf_hidden(const VfGeom& g, float size, const long long* ptr, const int* idx, uint8_t* keep, int* kept,
              cudaStream_t st);
int vf_compact(const VfGeom& g, const long long* ptr, const uint8_t* keep, const int* idx, const float* vf,
               const float* dir, const long long* optr, int* oidx, float* ovf, float* odir, cudaStream_t st);
int vf_refine(const VfGeom& g, const long long* ptr, const int* idx, float* vf, float* dir, cudaStream_t st);
int vf_photo(const VfGeom& g, const long long* ptr, const float* dir, float* photo, cudaStream_t st);
void set_last_error(const char* msg);
}  // namespace atpm

namespace {
// What a call leaves in the stream-ordered pool beyond what the pool held before
// is bounded: the candidates of a large shape take gigabytes, which the context's
// release threshold would keep from the rest of the process for good.
struct PoolGrowth {
    static constexpr uint64_t kKeep = 512ull << 20;
    cudaMemPool_t pool = nullptr;
    uint64_t before = 0;
    PoolGrowth() {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetMemPool(&pool, device) != cudaSuccess ||
            cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &before) != cudaSuccess)
            pool = nullptr;
    }
    ~PoolGrowth() {  // after the buffers' own destructors
        uint64_t now = 0;
        if (pool && cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &now) == cudaSuccess &&
            now > before + kKeep && cudaStreamSynchronize(0) == cudaSuccess)
            cudaMemPoolTrimTo(pool, before + kKeep);
    }
};
// device memory from the stream-ordered pool (kept by the context's release
// threshold from call to call), given back with its owner
struct DevBufs {
    std::vector<void*> p;
    cudaStream_t st = nullptr;
    ~DevBufs() {
        for (void* x : p) cudaFreeAsync(x, st);
    }
    template <class T> cudaError_t alloc(T** out, size_t n) {
        void* q = nullptr;
        cudaError_t e = cudaMallocAsync(&q, n ? n * sizeof(T) : 1, st);
        if (e == cudaSuccess) { p.push_back(q); *out = static_cast<T*>(q); }
        return e;
    }
};
// the device a result lives on is current within the scope
struct OnDevice {
    int before = -1;
    explicit OnDevice(int device) {
        if (cudaGetDevice(&before) != cudaSuccess) before = -1;
        if (before != device) cudaSetDevice(device);
    }
    ~OnDevice() {
        if (before >= 0) cudaSetDevice(before);
    }
};
atpm_status vfail(atpm_status s, const char* what, cudaError_t e) {
    char buf[256];
    cudaGetLastError();
    std::snprintf(buf, sizeof buf, "viewfactors: %s: %s", what, cudaGetErrorString(e));
    atpm::set_last_error(buf);
    return s;
}
}  // namespace

struct atpm_vf_result {
    int nf = 0, device = 0;
    std::vector<int32_t> ptr;
    DevBufs bufs;
    int* idx = nullptr;
    float *vf = nullptr, *dir = nullptr, *photo = nullptr;
};

extern "C" {

ATPM_API atpm_status atpm_viewfactors_compute(atpm_context* ctx, int32_t nv, int32_t nf, const float* vertices,
                                              const int32_t* facets, int32_t refine, atpm_vf_result** out,
                                              int64_t* nnz_out) {
    (void)ctx;
    if (!vertices || !facets || !out || nv < 3 || nf < 1) {
        atpm::set_last_error("viewfactors: bad arguments");
        return ATPM_E_INVALID;
    }
    for (int i = 0; i < 3 * nf; ++i)
        if (facets[i] < 0 || facets[i] >= nv) {
            atpm::set_last_error("viewfactors: facet vertex index out of range");
            return ATPM_E_INVALID;
        }
    float size = 0.0f;  // the largest coordinate: the scale of the positions' rounding
    for (int i = 0; i < 3 * nv; ++i) size = std::max(size, std::fabs(vertices[i]));
    cudaStream_t st = 0;
    PoolGrowth growth;
    DevBufs B;
    atpm::VfGeom g{};
    g.nv = nv;
    g.nf = nf;
    float* v = nullptr;
    int* fac = nullptr;
    cudaError_t e;
#define T(x, what) if ((e = (x)) != cudaSuccess) return vfail(ATPM_E_CUDA, what, e)
    T(B.alloc(&v, (size_t)nv * 3), "alloc");
    T(B.alloc(&fac, (size_t)nf * 3), "alloc");
    T(B.alloc(&g.mid, (size_t)nf * 3), "alloc");
    T(B.alloc(&g.nrm, (size_t)nf * 3), "alloc");
    T(B.alloc(&g.area, (size_t)nf), "alloc");
    T(B.alloc(&g.nlen, (size_t)nf), "alloc");
    T(cudaMemcpy(v, vertices, (size_t)nv * 12, cudaMemcpyHostToDevice), "upload");
    T(cudaMemcpy(fac, facets, (size_t)nf * 12, cudaMemcpyHostToDevice), "upload");
    g.v = v;
    g.fac = fac;
    if (atpm::vf_init(g, st)) return vfail(ATPM_E_CUDA, "init launch", cudaGetLastError());
    int* cnt = nullptr;
    long long* dptr = nullptr;
    T(B.alloc(&cnt, (size_t)nf), "alloc");
    T(B.alloc(&dptr, (size_t)nf + 1), "alloc");
    if (atpm::vf_count(g, cnt, st)) return vfail(ATPM_E_CUDA, "count launch", cudaGetLastError());
    std::vector<int> hc(nf);
    std::vector<long long> ptr(nf + 1, 0);
    T(cudaMemcpy(hc.data(), cnt, (size_t)nf * 4, cudaMemcpyDeviceToHost), "count");
    for (int i = 0; i < nf; ++i) ptr[i + 1] = ptr[i] + hc[i];
    const size_t tot = (size_t)ptr[nf];
    int* didx = nullptr;
    float *dvf = nullptr, *ddir = nullptr;
    uint8_t* keep = nullptr;
    T(B.alloc(&didx, tot), "alloc candidates");
    T(B.alloc(&dvf, tot), "alloc candidates");
    T(B.alloc(&ddir, 3 * tot), "alloc candidates");
    T(B.alloc(&keep, tot), "alloc candidates");
    T(cudaMemcpy(dptr, ptr.data(), (size_t)(nf + 1) * 8, cudaMemcpyHostToDevice), "upload");
    if (atpm::vf_fill(g, dptr, didx, dvf, ddir, st)) return vfail(ATPM_E_CUDA, "fill launch", cudaGetLastError());
    if (atpm::vf_hidden(g, size, dptr, didx, keep, cnt, st))
        return vfail(ATPM_E_CUDA, "hidden launch", cudaGetLastError());
    T(cudaMemcpy(hc.data(), cnt, (size_t)nf * 4, cudaMemcpyDeviceToHost), "kept count");
    auto* r = new atpm_vf_result();
    r->nf = nf;
    r->bufs.st = st;
    r->ptr.assign(nf + 1, 0);
    for (int i = 0; i < nf; ++i) r->ptr[i + 1] = r->ptr[i] + hc[i];
    const size_t n2 = (size_t)r->ptr[nf];
    std::vector<long long> p2(r->ptr.begin(), r->ptr.end());
    long long* optr = nullptr;
    e = cudaGetDevice(&r->device);
    if (e == cudaSuccess) e = B.alloc(&optr, (size_t)nf + 1);
    if (e == cudaSuccess) e = r->bufs.alloc(&r->idx, n2);
    if (e == cudaSuccess) e = r->bufs.alloc(&r->vf, n2);
    if (e == cudaSuccess) e = r->bufs.alloc(&r->dir, 3 * n2);
    if (e == cudaSuccess) e = r->bufs.alloc(&r->photo, 3 * (size_t)nf);
    if (e == cudaSuccess) e = cudaMemcpy(optr, p2.data(), (size_t)(nf + 1) * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && atpm::vf_compact(g, dptr, keep, didx, dvf, ddir, optr, r->idx, r->vf, r->dir, st))
        e = cudaGetLastError();
    if (e == cudaSuccess && refine && n2 > 0 && atpm::vf_refine(g, optr, r->idx, r->vf, r->dir, st))
        e = cudaGetLastError();
    if (e == cudaSuccess && atpm::vf_photo(g, optr, r->dir, r->photo, st)) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { delete r; return vfail(ATPM_E_CUDA, "lists", e); }
#undef T
    *out = r;
    if (nnz_out) *nnz_out = (int64_t)n2;
    return ATPM_OK;
}

ATPM_API atpm_status atpm_viewfactors_get(const atpm_vf_result* r, int32_t* dep_ptr, int32_t* dep_idx, float* dep_vf,
                                          float* dep_vec, float* photovectors) {
    if (!r) { atpm::set_last_error("viewfactors_get: null result"); return ATPM_E_INVALID; }
    OnDevice on(r->device);
    const size_t n = (size_t)r->ptr[r->nf];
    cudaError_t e = cudaSuccess;
    auto copy = [&](void* to, const void* from, size_t bytes) {
        if (to && bytes && e == cudaSuccess) e = cudaMemcpy(to, from, bytes, cudaMemcpyDeviceToHost);
    };
    if (dep_ptr) std::copy(r->ptr.begin(), r->ptr.end(), dep_ptr);
    copy(dep_idx, r->idx, n * 4);
    copy(dep_vf, r->vf, n * 4);
    copy(dep_vec, r->dir, n * 12);
    copy(photovectors, r->photo, (size_t)r->nf * 12);
    return e == cudaSuccess ? ATPM_OK : vfail(ATPM_E_CUDA, "download", e);
}

ATPM_API atpm_status atpm_viewfactors_free(atpm_vf_result* r) {
    if (!r) return ATPM_OK;
    OnDevice on(r->device);
    delete r;
    return ATPM_OK;
}
}
