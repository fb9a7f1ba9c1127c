// Source injection and receiver extraction (spacetime.cc:144-204), on the GPU.
//
// The reference runs its partitions in parallel (no grid point, resp. trace, is shared between
// two partitions: src/spacetime.jl:1087-1129) and each partition sequentially, so every grid
// cell (resp. trace sample) receives its contributions in partition order. Here the points are
// grouped by the cell they write (stable sort, which keeps that order) and one thread owns each
// group and accumulates it in order with separate IEEE multiply and add: the result is the
// reference's, bit for bit, whatever the grouping into partitions was.
//
// Drop-in entry points take host partition tables, as the reference does, and work for device,
// managed or host field/data arrays. The WFD_Points_* add-ons keep the grouped table resident
// on the device for the time loop.
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "wavefd_b200.h"
#include "wfd_alloc.h"
#include "wfd_points.h"
#include "wfd_prop.h"

namespace wfd {

namespace {

template <class T>
bool upload(Table<T> &t, cudaStream_t s) {
    const size_t ng = (size_t)t.ngroups, np = (size_t)t.npoints;
    if (wfd::dMallocAsync(&t.d_key, sizeof(long) * (ng + 1), s) != cudaSuccess) return false;
    if (wfd::dMallocAsync(&t.d_start, sizeof(long) * (ng + 1), s) != cudaSuccess) return false;
    if (wfd::dMallocAsync(&t.d_other, sizeof(long) * (np + 1), s) != cudaSuccess) return false;
    if (wfd::dMallocAsync(&t.d_c, sizeof(T) * (np + 1), s) != cudaSuccess) return false;
    if (ng) cudaMemcpyAsync(t.d_key, t.key.data(), sizeof(long) * ng, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(t.d_start, t.start.data(), sizeof(long) * (ng + 1), cudaMemcpyHostToDevice, s);
    if (np) cudaMemcpyAsync(t.d_other, t.other.data(), sizeof(long) * np, cudaMemcpyHostToDevice, s);
    if (np) cudaMemcpyAsync(t.d_c, t.c.data(), sizeof(T) * np, cudaMemcpyHostToDevice, s);
    return true;
}

template <class T>
void release(Table<T> &t, cudaStream_t s) {
    if (t.d_key) cudaFreeAsync(t.d_key, s);
    if (t.d_start) cudaFreeAsync(t.d_start, s);
    if (t.d_other) cudaFreeAsync(t.d_other, s);
    if (t.d_c) cudaFreeAsync(t.d_c, s);
    t.d_key = t.d_start = t.d_other = nullptr;
    t.d_c = nullptr;
}

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

// dst[key[g]] (+)= sum over the group of c * src[other * stride + off], in group order.
// With dst/src given as compact arrays (stride 0 / per-point values) the same kernel serves the
// staged drop-in path.
template <class T>
__global__ void k_scatter_groups(long ngroups, const long *__restrict__ key, const long *__restrict__ start,
                                 const long *__restrict__ other, const T *__restrict__ c, T *dst, long dst_stride,
                                 long dst_off, int dst_compact, const T *__restrict__ src, long src_stride,
                                 long src_off, int src_compact) {
    const long gi = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= ngroups) return;
    const long d = dst_compact ? gi : key[gi] * dst_stride + dst_off;
    T acc = dst[d];
    for (long j = start[gi]; j < start[gi + 1]; j++) {
        const T v = src_compact ? src[j] : src[other[j] * src_stride + src_off];
        acc = add_rn(acc, mul_rn(c[j], v));
    }
    dst[d] = acc;
}

// the device-table scatter with the time index read from device memory (graph-captured time loops):
// inject (by_receiver 0): field[key] += sum c * data[other*nt + it-1]; extract: data[key*nt + it-1]
// += sum c * field[other]; skipped when it is outside 1..nt
__global__ void k_scatter_groups_devit(long ngroups, const long *__restrict__ key, const long *__restrict__ start,
                                       const long *__restrict__ other, const float *__restrict__ c, int by_receiver,
                                       float *field, float *data, long nt, const long *__restrict__ d_it) {
    const long gi = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long it = *d_it;
    if (gi >= ngroups || it < 1 || it > nt) return;
    float *dst = by_receiver ? data + key[gi] * nt + (it - 1) : field + key[gi];
    float acc = *dst;
    for (long j = start[gi]; j < start[gi + 1]; j++) {
        const float v = by_receiver ? field[other[j]] : data[other[j] * nt + (it - 1)];
        acc = add_rn(acc, mul_rn(c[j], v));
    }
    *dst = acc;
}

// extraction at the device time index (as k_scatter_groups_devit, by receiver) followed by the
// index's advance: every block reads the index first, counts itself done, and the last block to
// finish writes index + 1 (and resets the count for the next launch); no block waits for another
__global__ void k_extract_tick(long ngroups, const long *__restrict__ key, const long *__restrict__ start,
                               const long *__restrict__ other, const float *__restrict__ c,
                               const float *__restrict__ field, float *data, long nt, long *d_it,
                               unsigned *done) {
    const long gi = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long it = *d_it;
    if (gi < ngroups && it >= 1 && it <= nt) {
        float *dst = data + key[gi] * nt + (it - 1);
        float acc = *dst;
        for (long j = start[gi]; j < start[gi + 1]; j++) acc = add_rn(acc, mul_rn(c[j], field[other[j]]));
        *dst = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(done, 1u) == gridDim.x - 1) {
            *d_it = it + 1;
            *done = 0u;
            __threadfence();
        }
    }
}

inline unsigned nb(long n) { return (unsigned)((n + 255) / 256); }

template <class T>
std::vector<PointsT<T>> flatten(void **partitions, size_t npartitions, const long *npoints) {
    std::vector<PointsT<T>> pts;
    size_t total = 0;
    for (size_t i = 0; i < npartitions; i++) total += (size_t)npoints[i];
    pts.reserve(total);
    for (size_t i = 0; i < npartitions; i++) {
        const PointsT<T> *p = reinterpret_cast<const PointsT<T> *>(partitions[i]);
        for (long j = 0; j < npoints[i]; j++) pts.push_back(p[j]);
    }
    return pts;
}

cudaStream_t st_stream() {
    static thread_local cudaStream_t s = nullptr;
    if (!s) cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    return s;
}

// Drop-in tables are kept between calls: a time loop calls injectdata/extractdata every step with
// the same partitions, and grouping, sorting and uploading 65,536 receivers every step would cost
// more than the step. An entry is reused when the caller's partitions hold the same points (iu, ir
// and the bits of c compared one by one, so a caller that rewrites its arrays in place gets a new
// table); up to kCacheEntries tables stay resident, least recently used evicted first. Each entry
// also keeps its device and pinned staging buffers. Calls are synchronous and serialised by the
// cache lock, as the reference's calls are synchronous.
constexpr int kCacheEntries = 8;

template <class T>
struct CachedTable {
    Table<T> t;
    int by_receiver = 0;
    std::vector<PointsT<T>> raw;       // the caller's points, partition by partition
    std::vector<long> counts;          // points per partition
    long longest = 0;                  // points of the largest group
    unsigned long long last_use = 0;
    T *d_src = nullptr;                    // device staging (points)
    T *h_dst = nullptr, *h_src = nullptr;  // pinned host staging (groups, points), mapped
};

// Host loops over the points of a drop-in call use up to the caller's thread count (the reference's
// nthreads argument) once they are long enough to pay for it.
constexpr long kParallelPoints = 8192;
// Values that the kernel reads from mapped pinned memory itself: up to kMappedPoints of them, and up to kMappedRun by one
// thread, which reads a group's one after another at 0.14 us each over the bus (0.03 from device memory, after a
// copy of 5 to 10 us). Extraction with host arrays, groups x points, us a call read so and copied: 1 x 32 34.5,
// 35.1; 1 x 64 39.4, 36.1; 64 x 64 57.7, 61.9; 1 x 128 48.1, 36.4; 8 x 512 120, 72; 1 x 4096 601, 153.
constexpr long kMappedPoints = 4096, kMappedRun = 64;

template <class T>
bool same_points(const CachedTable<T> &e, int by_receiver, void **partitions, size_t npartitions,
                 const long *npoints, int nth) {
    if (e.by_receiver != by_receiver || e.counts.size() != npartitions) return false;
    size_t j = 0;
    for (size_t i = 0; i < npartitions; i++) {
        if (e.counts[i] != npoints[i]) return false;
        const PointsT<T> *p = reinterpret_cast<const PointsT<T> *>(partitions[i]);
        const PointsT<T> *q = e.raw.data() + j;
        const long n = npoints[i];
        int diff = 0;
#pragma omp parallel for num_threads(nth) if (n >= kParallelPoints) reduction(| : diff) schedule(static)
        for (long k = 0; k < n; k++)
            diff |= (p[k].iu != q[k].iu || p[k].ir != q[k].ir || memcmp(&p[k].c, &q[k].c, sizeof(T)) != 0) ? 1 : 0;
        if (diff) return false;
        j += (size_t)n;
    }
    return true;
}

template <class T>
void free_entry(CachedTable<T> *e, cudaStream_t s) {
    release(e->t, s);
    if (e->d_src) cudaFreeAsync(e->d_src, s);
    cudaStreamSynchronize(s);
    if (e->h_dst) cudaFreeHost(e->h_dst);
    if (e->h_src) cudaFreeHost(e->h_src);
    delete e;
}

template <class T>
struct TableCache {
    std::mutex mu;
    std::vector<CachedTable<T> *> entries;
    unsigned long long clock = 0;
};

template <class T>
TableCache<T> &table_cache() {
    static TableCache<T> *c = new TableCache<T>();  // never destroyed: no CUDA calls at process exit
    return *c;
}

// the entry for these partitions (built and uploaded on a miss), or nullptr on allocation failure
template <class T>
CachedTable<T> *lookup(TableCache<T> &cache, int by_receiver, void **partitions, size_t npartitions,
                       const long *npoints, cudaStream_t s, int nth) {
    for (CachedTable<T> *e : cache.entries)
        if (same_points(*e, by_receiver, partitions, npartitions, npoints, nth)) {
            e->last_use = ++cache.clock;
            return e;
        }
    CachedTable<T> *e = new CachedTable<T>();
    e->by_receiver = by_receiver;
    e->raw = flatten<T>(partitions, npartitions, npoints);
    e->counts.assign(npoints, npoints + npartitions);
    build(e->t, e->raw, by_receiver);
    for (long g = 0; g < e->t.ngroups; g++) e->longest = std::max(e->longest, e->t.start[g + 1] - e->t.start[g]);
    const size_t ng = (size_t)e->t.ngroups, np = (size_t)e->t.npoints;
    bool ok = upload(e->t, s);
    ok = ok && wfd::dMallocAsync(&e->d_src, sizeof(T) * (np + 1), s) == cudaSuccess;
    ok = ok && wfd::dMallocHost(&e->h_dst, sizeof(T) * (ng + 1)) == cudaSuccess;
    ok = ok && wfd::dMallocHost(&e->h_src, sizeof(T) * (np + 1)) == cudaSuccess;
    if (!ok) {
        free_entry(e, s);
        return nullptr;
    }
    if ((int)cache.entries.size() >= kCacheEntries) {
        auto lru = std::min_element(cache.entries.begin(), cache.entries.end(),
                                    [](const CachedTable<T> *a, const CachedTable<T> *b) {
                                        return a->last_use < b->last_use;
                                    });
        free_entry(*lru, s);
        cache.entries.erase(lru);
    }
    e->last_use = ++cache.clock;
    cache.entries.push_back(e);
    return e;
}

// Drop-in inject (by_receiver = 0) / extract (1). dst is written at key*dst_stride + dst_off,
// src is read at other*src_stride + src_off. Device (or managed) arrays are read and written in
// place by one kernel; host arrays go through the entry's pinned staging (the values the points
// read, and the current values of the locations they write, up; the new values back).
template <class T>
void dropin(int by_receiver, T *dst, long dst_stride, long dst_off, const T *src, long src_stride, long src_off,
            void **partitions, size_t npartitions, const long *npoints, size_t nthreads) {
    long total = 0;
    for (size_t i = 0; i < npartitions; i++) total += npoints[i];
    if (total <= 0) return;
    const int nth = nthreads > 1 ? (int)(nthreads < 256 ? nthreads : 256) : 1;
    cudaStream_t s = st_stream();
    TableCache<T> &cache = table_cache<T>();
    std::lock_guard<std::mutex> lk(cache.mu);
    CachedTable<T> *e = lookup(cache, by_receiver, partitions, npartitions, npoints, s, nth);
    if (!e) {
        set_global_error(WFD_ERR_ALLOC, "point table allocation failed");
        return;
    }
    const Table<T> &t = e->t;
    const bool dst_dev = device_accessible(dst);
    const bool src_dev = device_accessible(src);
    const long ng = t.ngroups, np = t.npoints;
    // The kernel reads and writes the pinned staging itself: each written location once and coalesced, and the
    // values read where they are few. More go through the device.
    const bool copy = np > kMappedPoints || e->longest > kMappedRun;
    if (!src_dev) {
#pragma omp parallel for num_threads(nth) if (np >= kParallelPoints) schedule(static)
        for (long j = 0; j < np; j++) e->h_src[j] = src[t.other[j] * src_stride + src_off];
        if (copy) cudaMemcpyAsync(e->d_src, e->h_src, sizeof(T) * (size_t)np, cudaMemcpyHostToDevice, s);
    }
    if (!dst_dev) {
#pragma omp parallel for num_threads(nth) if (ng >= kParallelPoints) schedule(static)
        for (long g = 0; g < ng; g++) e->h_dst[g] = dst[t.key[g] * dst_stride + dst_off];
    }
    k_scatter_groups<T><<<nb(ng), 256, 0, s>>>(ng, t.d_key, t.d_start, t.d_other, t.d_c,
                                               dst_dev ? dst : e->h_dst, dst_dev ? dst_stride : 0,
                                               dst_dev ? dst_off : 0, dst_dev ? 0 : 1,
                                               src_dev ? src : (copy ? e->d_src : e->h_src), src_dev ? src_stride : 0,
                                               src_dev ? src_off : 0, src_dev ? 0 : 1);
    cudaError_t err = cudaStreamSynchronize(s);
    if (err != cudaSuccess) {
        set_global_error(WFD_ERR_CUDA, cudaGetErrorString(err));
        return;
    }
    if (!dst_dev) {
#pragma omp parallel for num_threads(nth) if (ng >= kParallelPoints) schedule(static)
        for (long g = 0; g < ng; g++) dst[t.key[g] * dst_stride + dst_off] = e->h_dst[g];
    }
}

struct DeviceTable {
    Table<float> t;
};

}  // namespace
}  // namespace wfd

using wfd::DeviceTable;

// ---- drop-in libspacetime exports (spacetime.cc:144-204) ---------------------------------------------
extern "C" void injectdata_float(float *field, float *data, size_t it, size_t nt, SourcePoint32 **partitions,
                                 size_t npartitions, long *npoints_per_partition, size_t nthreads) {
    wfd::dropin<float>(0, field, 1, 0, data, (long)nt, (long)it - 1, (void **)partitions, npartitions,
                       npoints_per_partition, nthreads);
}

extern "C" void injectdata_double(double *field, double *data, size_t it, size_t nt, SourcePoint64 **partitions,
                                  size_t npartitions, long *npoints_per_partition, size_t nthreads) {
    wfd::dropin<double>(0, field, 1, 0, data, (long)nt, (long)it - 1, (void **)partitions, npartitions,
                        npoints_per_partition, nthreads);
}

extern "C" void extractdata_float(float *data, float *field, SourcePoint32 **partitions, size_t npartitions,
                                  long *npoints_per_partition, size_t it, size_t nt, size_t nthreads) {
    wfd::dropin<float>(1, data, (long)nt, (long)it - 1, field, 1, 0, (void **)partitions, npartitions,
                       npoints_per_partition, nthreads);
}

extern "C" void extractdata_double(double *data, double *field, SourcePoint64 **partitions, size_t npartitions,
                                   long *npoints_per_partition, size_t it, size_t nt, size_t nthreads) {
    wfd::dropin<double>(1, data, (long)nt, (long)it - 1, field, 1, 0, (void **)partitions, npartitions,
                        npoints_per_partition, nthreads);
}

// ---- add-on: device-resident point tables ------------------------------------------------------------
extern "C" void *WFD_Points_Create(const SourcePoint32 *points, long npoints, int by_receiver) {
    if (npoints < 0 || (npoints > 0 && !points)) {
        wfd::set_global_error(WFD_ERR_ARG, "WFD_Points_Create: bad point list");
        return nullptr;
    }
    std::vector<wfd::PointsT<float>> pts((size_t)npoints);
    for (long i = 0; i < npoints; i++) {
        if (points[i].iu < 1 || points[i].ir < 1) {  // 1-based indices (spacetime.jl:793-797)
            wfd::set_global_error(WFD_ERR_ARG, "WFD_Points_Create: indices are 1-based");
            return nullptr;
        }
        pts[i] = {points[i].iu, points[i].ir, points[i].c};
    }
    DeviceTable *d = new DeviceTable();
    wfd::build(d->t, pts, by_receiver);
    cudaStream_t s = wfd::st_stream();
    if (!wfd::upload(d->t, s) || cudaStreamSynchronize(s) != cudaSuccess) {
        wfd::release(d->t, s);
        delete d;
        wfd::set_global_error(WFD_ERR_ALLOC, "WFD_Points_Create: device allocation failed");
        return nullptr;
    }
    return d;
}

extern "C" void WFD_Points_Free(void *table) {
    DeviceTable *d = reinterpret_cast<DeviceTable *>(table);
    if (!d) return;
    cudaStream_t s = wfd::st_stream();
    wfd::release(d->t, s);
    cudaStreamSynchronize(s);
    delete d;
}

extern "C" long WFD_Points_Groups(void *table) {
    DeviceTable *d = reinterpret_cast<DeviceTable *>(table);
    return d ? d->t.ngroups : -1;
}

extern "C" int WFD_Inject(void *table, float *field, const float *data, long it, long nt, void *stream) {
    DeviceTable *d = reinterpret_cast<DeviceTable *>(table);
    if (!d || d->t.by_receiver || it < 1 || it > nt) return WFD_ERR_ARG;
    if (!d->t.ngroups) return WFD_OK;
    wfd::k_scatter_groups<float><<<wfd::nb(d->t.ngroups), 256, 0, (cudaStream_t)stream>>>(
        d->t.ngroups, d->t.d_key, d->t.d_start, d->t.d_other, d->t.d_c, field, 1, 0, 0, data, nt, it - 1, 0);
    return cudaGetLastError() == cudaSuccess ? WFD_OK : WFD_ERR_CUDA;
}

extern "C" int WFD_Extract(void *table, float *data, const float *field, long it, long nt, void *stream) {
    DeviceTable *d = reinterpret_cast<DeviceTable *>(table);
    if (!d || !d->t.by_receiver || it < 1 || it > nt) return WFD_ERR_ARG;
    if (!d->t.ngroups) return WFD_OK;
    wfd::k_scatter_groups<float><<<wfd::nb(d->t.ngroups), 256, 0, (cudaStream_t)stream>>>(
        d->t.ngroups, d->t.d_key, d->t.d_start, d->t.d_other, d->t.d_c, data, nt, it - 1, 0, field, 1, 0, 0);
    return cudaGetLastError() == cudaSuccess ? WFD_OK : WFD_ERR_CUDA;
}

extern "C" int WFD_ExtractInterp(void *table, float *coarse, const float *field, const float *h, long nh, long it,
                                 long nm, long nd, void *stream) {
    DeviceTable *d = reinterpret_cast<DeviceTable *>(table);
    if (!d || !d->t.by_receiver || !coarse || !field || !h || nh < 1 || nd < 7 || it < 1 || it > nm) return WFD_ERR_ARG;
    if (!d->t.ngroups) return WFD_OK;
    wfd::launch_extract_interp(d->t.ngroups, d->t.d_key, d->t.d_start, d->t.d_other, d->t.d_c, field, h, nh, it - 1,
                               nm, nd, coarse, (cudaStream_t)stream);
    return cudaGetLastError() == cudaSuccess ? WFD_OK : WFD_ERR_CUDA;
}

// ---- add-on: a whole time loop in a CUDA graph ---------------------------------------------------------
namespace {

using wfd::Prop;

int run_step(Prop *p, DeviceTable *src, const float *wav, DeviceTable *rec, float *trc, long nt, long *d_it) {
    if (int rc = wfd::prop_step(p, false, false)) return rc;
    float *pc = p->field[wfd::F_PCUR];
    cudaStream_t s = p->stream;
    const bool inject = src && src->t.ngroups && !p->inject_done;  // unless the step kernel did it
    p->step_kernels += (inject ? 1 : 0) + 1;  // launches per step of the loop
    if (inject)
        wfd::k_scatter_groups_devit<<<wfd::nb(src->t.ngroups), 256, 0, s>>>(
            src->t.ngroups, src->t.d_key, src->t.d_start, src->t.d_other, src->t.d_c, 0, pc, const_cast<float *>(wav),
            nt, d_it);
    // extraction and the advance of the time index in one launch (d_it[1] counts finished blocks)
    unsigned *done = reinterpret_cast<unsigned *>(d_it + 1);
    if (rec && rec->t.ngroups)
        wfd::k_extract_tick<<<wfd::nb(rec->t.ngroups), 256, 0, s>>>(rec->t.ngroups, rec->t.d_key, rec->t.d_start,
                                                                    rec->t.d_other, rec->t.d_c, pc, trc, nt, d_it,
                                                                    done);
    else
        wfd::k_extract_tick<<<1, 32, 0, s>>>(0, nullptr, nullptr, nullptr, nullptr, pc, trc, nt, d_it, done);
    return cudaGetLastError() == cudaSuccess ? WFD_OK : wfd::prop_fail(p, WFD_ERR_CUDA, "time loop launch");
}

}  // namespace

extern "C" int WFD_Prop_Run(void *prop, long nsteps, long it0, void *src_table, const float *wavelet, void *rec_table,
                            float *traces, long nt, int use_graph) {
    wfd::Prop *p = reinterpret_cast<wfd::Prop *>(prop);
    DeviceTable *src = reinterpret_cast<DeviceTable *>(src_table), *rec = reinterpret_cast<DeviceTable *>(rec_table);
    if (!p || nsteps < 0 || (src && (src->t.by_receiver || !wavelet)) || (rec && (!rec->t.by_receiver || !traces)))
        return WFD_ERR_ARG;
    if (p->status) return p->status;
    cudaStream_t s = p->stream;
    // scratch of the unfused passes must exist before a capture (no allocation inside a graph); the fused 3D Iso step
    // takes every grid
    if (!p->fused || p->ndim == 2 || (p->nz % 4 != 0 && p->phys != wfd::ISO))
        if (!wfd::ensure_scratch(p, p->phys == wfd::ISO ? 3 : 6)) return p->status;
    const bool run2d = p->ndim == 2 && p->fused && !p->illum && nsteps > 0 && (!src || src->t.ngroups <= 1024);
    long *d_it = nullptr;
    // d_it[0]: the time index; d_it[1]: the finished-block count of the extraction launch;
    // d_it[2..3]: the barrier words of the persistent 2D loop (count, generation, status)
    if (wfd::dMallocAsync(&d_it, 4 * sizeof(long), s) != cudaSuccess)
        return wfd::prop_fail(p, WFD_ERR_ALLOC, "time index allocation failed");
    const long init[4] = {it0, 0, 0, 0};
    cudaMemcpyAsync(d_it, init, sizeof init, cudaMemcpyHostToDevice, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return wfd::prop_fail(p, WFD_ERR_CUDA, "time index upload");
    // 2D: the whole loop in one cooperative launch (grid-wide barrier between steps)
    if (run2d) {
        wfd::Fields F = p->fields();
        F.inj = wfd::StepInject{};
        if (src && src->t.ngroups)
            F.inj = wfd::StepInject{src->t.ngroups, src->t.d_key, src->t.d_start, src->t.d_other, src->t.d_c,
                                    wavelet, nt, d_it};
        wfd::RunExtract ex{};
        if (rec && rec->t.ngroups)
            ex = wfd::RunExtract{rec->t.ngroups, rec->t.d_key, rec->t.d_start, rec->t.d_other, rec->t.d_c, traces, nt};
        unsigned *words = reinterpret_cast<unsigned *>(d_it + 2);
        const wfd::Grid g = p->grid();
        int r = -1;
        if (p->phys == wfd::ISO)
            r = p->strict ? wfd_strict::iso2d_run(g, F, nsteps, it0, ex, words, s)
                          : wfd_fast::iso2d_run(g, F, nsteps, it0, ex, words, s);  // tiles all resident, or -1
        else
            r = p->strict ? wfd_strict::aniso2d_run(g, p->phys, F, nsteps, it0, ex, words, s)
                          : wfd_fast::aniso2d_run(g, p->phys, F, nsteps, it0, ex, words, s);  // the same
        if (r < 0 && !p->strict)
            r = wfd_fast::loop2d_run(g, p->phys, F, p->scratch(), nsteps, it0, ex, words, s);
        if (r == 0) {
            unsigned status = 0;
            cudaMemcpyAsync(&status, words + 2, sizeof status, cudaMemcpyDeviceToHost, s);
            const cudaError_t e = cudaStreamSynchronize(s);
            cudaFreeAsync(d_it, s);
            if (e != cudaSuccess) return wfd::prop_fail(p, WFD_ERR_CUDA, std::string("time loop: ") + cudaGetErrorString(e));
            if (status) return wfd::prop_fail(p, WFD_ERR_TIMEOUT, "time loop: a grid-wide barrier timed out");
            if (nsteps & 1) {
                std::swap(p->field[wfd::F_PCUR], p->field[wfd::F_POLD]);
                if (p->phys != wfd::ISO) std::swap(p->field[wfd::F_MCUR], p->field[wfd::F_MOLD]);
            }
            p->steps += nsteps;
            p->step_kernels = 1;
            p->run_launches = 1;
            return WFD_OK;
        }
        if (r > 0) {
            cudaFreeAsync(d_it, s);
            return wfd::prop_fail(p, WFD_ERR_CUDA, "time loop: cooperative launch failed");
        }
    }
    // a step kernel that can apply the injection itself (the 2D Iso kernel) gets the source table;
    // the per-CTA scan of the groups stays cheap for tables of up to 1024 groups
    p->inj = wfd::StepInject{};
    if (src && src->t.ngroups && src->t.ngroups <= 1024)
        p->inj = wfd::StepInject{src->t.ngroups, src->t.d_key, src->t.d_start, src->t.d_other, src->t.d_c,
                                 wavelet, nt, d_it};
    long done = 0;
    int rc = WFD_OK;
    if (use_graph && nsteps >= 2) {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            rc = wfd::prop_fail(p, WFD_ERR_CUDA, "begin capture");
        } else {
            // two steps: the pointer swap of each is done on the host during the capture, so the
            // graph replays the pair with the pointers back where they started
            rc = run_step(p, src, wavelet, rec, traces, nt, d_it);
            if (!rc) rc = run_step(p, src, wavelet, rec, traces, nt, d_it);
            const cudaError_t e = cudaStreamEndCapture(s, &graph);
            if (!rc && e != cudaSuccess) rc = wfd::prop_fail(p, WFD_ERR_CUDA, "end capture");
            if (!rc && cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess)
                rc = wfd::prop_fail(p, WFD_ERR_CUDA, "graph instantiation");
            if (graph) cudaGraphDestroy(graph);
            p->steps -= 2;  // counted again per replay
            for (; !rc && done + 2 <= nsteps; done += 2) {
                if (cudaGraphLaunch(exec, s) != cudaSuccess) rc = wfd::prop_fail(p, WFD_ERR_CUDA, "graph launch");
                p->steps += 2;
            }
            if (exec) {
                cudaStreamSynchronize(s);
                cudaGraphExecDestroy(exec);
            }
        }
    }
    for (; !rc && done < nsteps; done++) rc = run_step(p, src, wavelet, rec, traces, nt, d_it);
    p->run_launches = nsteps * (long)p->step_kernels;
    p->inj = wfd::StepInject{};
    cudaFreeAsync(d_it, s);
    return rc;
}
