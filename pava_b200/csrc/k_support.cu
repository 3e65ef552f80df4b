// Support kernels: CSR validation, the augmented row pointer and the deterministic carry fixup
// shared by the CVR and CSR5 forms.

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

#include "pava_internal.h"

namespace pava {

// ---- device memory ----------------------------------------------------------------------------
// cudaMalloc and cudaFree cost 0.1-1 ms each for buffers of this size (mapping, and a device-wide
// wait), more than the conversion kernels: a 23.9 M nonzero CSR5 conversion took 4.6-11 ms of
// which the kernels are 0.46 ms, COO -> CSR of 13.5 M entries 7.7-9.6 ms against 1.5 ms.  Out of a
// pool that keeps up to POOL_KEEP bytes they take 0.55 and 1.7 ms.

namespace {

constexpr int POOL_DEVICES = 64;
struct DevicePool {
    cudaMemPool_t pool = nullptr;
    void *anchor = nullptr;       // keeps the driver's block of small allocations mapped
    std::vector<void *> waiting;  // freed while the device could not be waited for
    size_t large = 0;             // bytes of the large blocks that are in use out of the pool
};
std::mutex g_pool_mutex;
// The blocks of at least LARGE_MIN bytes that pool_malloc gave and that are in use.
struct LargeBlock {
    DevicePool *from;
    size_t bytes;
    bool plain;  // by cudaMalloc
};
std::unordered_map<void *, LargeBlock> &g_large = *new std::unordered_map<void *, LargeBlock>();
// Takes p off the list; whether cudaMalloc gave it.  g_pool_mutex held.
bool forget_large(void *p) {
    const auto it = g_large.find(p);
    if (it == g_large.end()) return false;
    const bool plain = it->second.plain;
    if (!plain) it->second.from->large -= it->second.bytes;
    g_large.erase(it);
    return plain;
}
// One per device and context: a program may alternate contexts on a device, and a context keeps its
// pool.  A device reset ends a context and what its pool held; contexts are never numbered alike, so
// the entry it leaves is not met again.  Never destroyed: handles may be freed at process exit.
std::map<std::pair<int, unsigned long long>, DevicePool> &g_pools =
    *new std::map<std::pair<int, unsigned long long>, DevicePool>();

// Identity of the current context; 0 when the driver cannot tell.
unsigned long long context_id() {
    typedef int (*get_t)(void **);
    typedef int (*id_t)(void *, unsigned long long *);
    static void *get = nullptr, *id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &get, 12000, cudaEnableDefault, &q) !=
                cudaSuccess || q != cudaDriverEntryPointSuccess)
            get = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &id, 12000, cudaEnableDefault, &q) !=
                cudaSuccess || q != cudaDriverEntryPointSuccess)
            id = nullptr;
    });
    void *ctx = nullptr;
    unsigned long long v = 0;
    if (!get || !id || ((get_t)get)(&ctx) != 0 || !ctx || ((id_t)id)(ctx, &v) != 0) return 0;
    return v;
}

// The current device's and context's entry; g_pool_mutex held.
cudaError_t device_entry(DevicePool **out, int *dev) {
    cudaError_t e = cudaGetDevice(dev);
    if (e != cudaSuccess) return e;
    if (*dev < 0 || *dev >= POOL_DEVICES) return cudaErrorInvalidDevice;
    unsigned long long ctx = context_id();
    if (ctx == 0) {  // a thread's first call: let the runtime make its context current
        e = cudaFree(nullptr);
        if (e != cudaSuccess) return e;
        ctx = context_id();
    }
    *out = &g_pools[{*dev, ctx}];
    return cudaSuccess;
}

// The same with its pool, made on first use.
cudaError_t device_pool(DevicePool **out) {
    int dev = 0;
    cudaError_t e = device_entry(out, &dev);
    if (e != cudaSuccess || (*out)->pool) return e;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    e = cudaMemPoolCreate(&(*out)->pool, &props);
    if (e != cudaSuccess) {
        (*out)->pool = nullptr;
        return e;
    }
    if (!(*out)->anchor && cudaMalloc(&(*out)->anchor, 1) != cudaSuccess) {
        (*out)->anchor = nullptr;  // device_wait tries again
        cudaGetLastError();
    }
    uint64_t keep = POOL_KEEP;
    return cudaMemPoolSetAttribute((*out)->pool, cudaMemPoolAttrReleaseThreshold, &keep);
}

// Waits for all work of the device, as cudaFree always does, by an allocation that is freed at once.
// cudaDeviceSynchronize would end a stream capture that another thread, or this one in relaxed mode, is
// making; cudaMalloc and cudaFree are allowed beside one.  5 us with the anchor (640 without, as
// the driver then maps and unmaps a block each time), 3 us for cudaDeviceSynchronize.
cudaError_t device_wait() {
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool *d = nullptr;
        int dev = 0;
        cudaError_t e = device_entry(&d, &dev);
        if (e == cudaSuccess && !d->anchor) {
            e = cudaMalloc(&d->anchor, 1);
            if (e != cudaSuccess) d->anchor = nullptr;
        }
        if (e != cudaSuccess) {
            cudaGetLastError();  // not the next launch's error
            return e;
        }
    }
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, 1);
    if (e == cudaSuccess) e = cudaFree(p);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

cudaError_t current_pool(cudaMemPool_t *pool) {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    DevicePool *d = nullptr;
    const cudaError_t e = device_pool(&d);
    if (e == cudaSuccess) *pool = d->pool;
    return e;
}

// Large blocks that the pool would not keep once they are freed come from cudaMalloc.  What a pool
// holds above its threshold is mapped and unmapped for each use, at several times cudaMalloc's price:
// blocks of 1.28, 0.64 and 0.32 GB taken and given back in turn take 14.0 ms from the pool, 3.6 from
// cudaMalloc; one of 5 GB 50 and 4.8.  Conversion of 200 M nonzeros to CSR5 22.2 -> 4.2 ms,
// to plain CSR 21.5 -> 2.7; COO -> CSR of 80 M entries 20 -> 7.1; CSR5 of 20 M beside a live matrix of
// 1.4 GB 2.9 -> 0.22.  The sizes in use are counted here: the pool's own count still holds, for a
// while, what has been freed.  One block, cudaMalloc / the pool's mapping: 4 and 32 MB 0.64 / 0.42 ms, 64 MB
// 0.65 / 0.80, 256 MB 0.79 / 3.3, 1 GB 1.7 / 12.6.
constexpr size_t LARGE_MIN = (size_t)64 << 20;

// cudaMalloc and cudaFree beside a capture on another stream, in whichever mode.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace

cudaError_t pool_malloc(void **p, size_t bytes, cudaStream_t s) {
    *p = nullptr;
    cudaMemPool_t pool = nullptr;
    DevicePool *d = nullptr;
    bool plain = false;
    if (bytes == 0) bytes = 1;
    cudaError_t e = cudaSuccess;
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        e = device_pool(&d);
        if (e != cudaSuccess) return e;
        pool = d->pool;
        plain = bytes >= LARGE_MIN && d->large + bytes > POOL_KEEP;
    }
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (plain && cudaStreamIsCapturing(s, &capturing) == cudaSuccess &&
        capturing == cudaStreamCaptureStatusNone) {
        RelaxedCapture relaxed;
        if (cudaMalloc(p, bytes) == cudaSuccess) {
            std::lock_guard<std::mutex> lock(g_pool_mutex);
            g_large[*p] = {d, bytes, true};
            return cudaSuccess;
        }
        cudaGetLastError();  // the pool may hold it
        *p = nullptr;
    }
    e = cudaMallocFromPoolAsync(p, bytes, pool, s);
    if (e == cudaErrorMemoryAllocation) {  // memory freed on other streams may still be on its way
        cudaGetLastError();
        if (device_wait() == cudaSuccess || cudaDeviceSynchronize() == cudaSuccess) {
            pool_trim(0);
            e = cudaMallocFromPoolAsync(p, bytes, pool, s);
        }
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        return e;
    }
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    forget_large(*p);  // an address of a context that a reset ended
    if (bytes >= LARGE_MIN) {
        d->large += bytes;
        g_large[*p] = {d, bytes, false};
    }
    return cudaSuccess;
}

cudaError_t plain_malloc(void **p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {  // the pool may hold it
        cudaGetLastError();
        if (device_wait() == cudaSuccess || cudaDeviceSynchronize() == cudaSuccess) {
            pool_trim(0);
            e = cudaMalloc(p, bytes);
        }
    }
    if (e != cudaSuccess) *p = nullptr;
    return e;
}

void pool_free(void *p, cudaStream_t s) {
    if (!p) return;
    bool plain;
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        plain = forget_large(p);
    }
    if (plain) {
        RelaxedCapture relaxed;
        cudaFree(p);  // waits for the device
    } else {
        cudaFreeAsync(p, s);
    }
}

void pool_free_synced(void *const *ps, int count) {
    int i0 = 0;
    while (i0 < count && !ps[i0]) ++i0;
    if (i0 == count) return;
    // the memory's own device, whichever is current
    int cur = 0;
    cudaPointerAttributes at = {};
    if (cudaGetDevice(&cur) != cudaSuccess || cudaPointerGetAttributes(&at, ps[i0]) != cudaSuccess ||
        at.device < 0 || at.device >= POOL_DEVICES)
        return;
    if (at.device != cur) cudaSetDevice(at.device);
    const bool waited = device_wait() == cudaSuccess;
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool *d = nullptr;
        int dev = 0;
        if (device_entry(&d, &dev) == cudaSuccess) {
            d->waiting.insert(d->waiting.end(), ps + i0, ps + count);
            for (int i = i0; i < count; ++i) forget_large(ps[i]);
            if (waited) {
                for (void *p : d->waiting) cudaFree(p);
                d->waiting.clear();
            }
        }
    }
    if (at.device != cur) cudaSetDevice(cur);
}

size_t pool_reserved() {
    cudaMemPool_t pool = nullptr;
    uint64_t held = 0;
    if (current_pool(&pool) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess)
        return 0;
    return (size_t)held;
}

void pool_trim(size_t keep) {
    cudaMemPool_t pool = nullptr;
    if (current_pool(&pool) == cudaSuccess) cudaMemPoolTrimTo(pool, keep);
}

cudaError_t pool_release(size_t keep) {
    cudaError_t e = device_wait();
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        DevicePool *d = nullptr;
        int dev = 0;
        e = device_entry(&d, &dev);
        if (e != cudaSuccess) return e;
        for (void *p : d->waiting) cudaFree(p);
        d->waiting.clear();
        pool = d->pool;
    }
    return pool ? cudaMemPoolTrimTo(pool, keep) : cudaSuccess;
}

namespace {

// Counts violations: row_ptr[0] != 0, row_ptr decreasing, row_ptr[m] != nnz, column outside
// [0, n); *longest (optional, zeroed by the caller) becomes the length of the longest row.  The reference performs no such check (its loader trusts the file).
// One pass at the copy bandwidth: columns as 16-byte vectors (from the first aligned one), four
// in flight per thread; the one-int-per-thread form read 96 MB in 82 us, this one in 21.
__global__ void __launch_bounds__(256)
validate_kernel(const int *__restrict__ rp, const int *__restrict__ ci, int m, int n, int nnz,
                int *__restrict__ err, int *__restrict__ longest) {
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    int bad = 0, most = 0;
    for (long long r = tid; r < m; r += stride) {
        const int a = rp[r], b = rp[r + 1];
        if (b < a) ++bad;
        else most = max(most, (int)((unsigned)b - (unsigned)a));
    }
    if (longest) {
        // one atomic per block, all to the same address; per warp they took 18 us for 3.8 M rows
        __shared__ int s_most;
        if (threadIdx.x == 0) s_most = 0;
        __syncthreads();
        most = __reduce_max_sync(FULL, most);
        if ((threadIdx.x & 31) == 0) atomicMax(&s_most, most);
        __syncthreads();
        if (threadIdx.x == 0 && s_most) atomicMax(longest, s_most);
    }
    if (tid == 0 && (rp[0] != 0 || rp[m] != nnz)) ++bad;
    if (bad == 0) {  // only scan columns against a sane row pointer
        const unsigned un = (unsigned)n;
        auto out = [&](int c) { return (unsigned)c >= un ? 1 : 0; };
        long long lead = (long long)((16 - (reinterpret_cast<uintptr_t>(ci) & 15)) & 15) / 4;
        if (lead > nnz) lead = nnz;
        const long long nv = (nnz - lead) / 4;
        const int4 *v = reinterpret_cast<const int4 *>(ci + lead);
        constexpr int U = 4;
        for (long long j = tid; j < nv; j += U * stride) {
            int4 a[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                a[u] = j + u * stride < nv ? __ldg(v + j + u * stride) : make_int4(0, 0, 0, 0);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u * stride < nv) bad += out(a[u].x) + out(a[u].y) + out(a[u].z) + out(a[u].w);
        }
        if (tid < lead) bad += out(ci[tid]);
        for (long long j = lead + 4 * nv + tid; j < nnz; j += stride) bad += out(ci[j]);
    }
    if (bad) atomicAdd(err, bad);
}

struct EmptyRow {
    const int *rp;
    __host__ __device__ int operator()(int r) const { return rp[r + 1] == rp[r] ? 1 : 0; }
};

// arp[r] = rp[r] + (empty rows before r), r in [0, m]; arp[m+1] is set by the caller.
__global__ void arp_kernel(const int *__restrict__ rp, const int *__restrict__ empties, int m,
                           int *__restrict__ arp) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r <= m) arp[r] = rp[r] + empties[r];
}

__global__ void set_int_kernel(int *p, int v) { *p = v; }

// One thread per chunk c1.  A row R that spans chunks c0 < c1 (it starts in c0 and ends in c1)
// gets y[R] = carry_tail[c0] + sum(carry_head[c0+1 .. c1]); chunks in between lie entirely
// inside R and hold their whole contribution in carry_head.  Nearly always c0 = c1 - 1, which the
// header of c1 - 1 tells, so one round of independent reads is enough.  Rows over up to nine
// chunks are summed by their thread, longer ones by the warp, one after the other, both in the same
// fixed order (lane-strided partial sums, then a fixed butterfly), so y is the same on every call.
// Bound by latency: a warp per chunk with the dependent reads header -> arp -> carries took 11.5 us
// for 32,245 chunks and 4.7 us for 640 after the SpMV kernel, this form 6.2 and 3.5 us.  Power-law
// matrices have many rows over three to nine chunks: summed by the warp too, they cost a product
// of 100,000 to 700,000 rows about 1 us.
// FRESH: the kernel before wrote the headers too (the allocation-free product), so they are read
// after the wait, and without __restrict__: as the carries they are written while this kernel
// waits, which rules out the read-only load path.
template <bool FRESH>
__global__ void __launch_bounds__(128)
carry_fixup_kernel(const char *meta, size_t stride, const int *arp, long long L,
                   const double *carry_head, const double *carry_tail, double *y,
                   long long nchunks, int m, unsigned long long *err) {
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const long long c1 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (FRESH) pdl_wait();
    // otherwise the headers belong to the matrix: read before the wait
    int R = -1;
    bool two = false;  // R starts in c1 - 1 and ends in c1
    long long c0 = c1;
    if (c1 > 0 && c1 < nchunks) {
        const ChunkHdr *H = reinterpret_cast<const ChunkHdr *>(meta + c1 * stride);
        const ChunkHdr *P = reinterpret_cast<const ChunkHdr *>(meta + (c1 - 1) * stride);
        const unsigned sh = H->shared, psh = P->shared;
        // R ends in c1, unless it runs through c1 and beyond
        if ((sh & 1u) && !((sh & 2u) && H->nrows == 1)) R = H->r_first;
        two = P->nrows > 1 || !(psh & 1u);
        if (R >= m || !guard(err, R >= -1, G_Y, R)) R = -1;
        if (R >= 0) c0 = two ? c1 - 1 : (long long)arp[R] / L;
        if (!guard(err, c0 >= 0 && c0 <= c1, G_CARRY, c0)) R = -1;
    }
    pdl_wait();  // the SpMV kernel's carries
    if (R >= 0 && two) y[R] = carry_tail[c1 - 1] + carry_head[c1];
    const bool few = c1 - c0 <= 8;
    if (R >= 0 && !two && few) {
        double h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = c0 + 1 + j <= c1 ? carry_head[c0 + 1 + j] : 0.0;
        // the order of warp_sum, so a row's sum does not depend on the branch
        y[R] = carry_tail[c0] + (((h[0] + h[4]) + (h[2] + h[6])) + ((h[1] + h[5]) + (h[3] + h[7])));
    }
    unsigned todo = __ballot_sync(FULL, R >= 0 && !few);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const int row = __shfl_sync(FULL, R, src);
        const long long c = __shfl_sync(FULL, c1, src), b = __shfl_sync(FULL, c0, src);
        double p = 0.0;
        for (long long j = b + 1 + lane; j <= c; j += 32) p += carry_head[j];
        p = warp_sum(p);
        if (lane == 0) y[row] = carry_tail[b] + p;
    }
}

// rows[t] = the row of augmented element t*T, for count runs of T elements.  A warp takes 32 rows
// at a time; each lane writes the runs that start in its row, and rows with many (a long row) are
// written by the whole warp.
__global__ void chunk_rows_kernel(const int *__restrict__ arp, int m, long long T, long long count,
                                  int *__restrict__ rows) {
    const int lane = threadIdx.x & 31;
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // rows 0 .. m
    long long t = 0, e = 0;
    if (r <= m) {
        t = ((long long)arp[r] + T - 1) / T;
        e = ((long long)arp[r + 1] + T - 1) / T;  // runs [t, e) start in the row
        if (e > count) e = count;
    }
    const bool many = e - t > 4;
    if (!many)
        for (; t < e; ++t) rows[t] = (int)r;
    unsigned todo = __ballot_sync(FULL, many);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const long long t0 = __shfl_sync(FULL, t, src), t1 = __shfl_sync(FULL, e, src);
        const int row = (int)__shfl_sync(FULL, r, src);
        for (long long q = t0 + lane; q < t1; q += 32) rows[q] = row;
    }
}

// Warp per chunk.  Chunk c holds the augmented elements [c*L, (c+1)*L); augmentation only
// inserts zero elements, so its nonzeros are the CSR's positions [p0, p1).  base = midpoint of
// their smallest and largest column: 16-bit offsets then reach any chunk whose columns span
// at most 65,534 (a chunk without nonzeros gets 0); *ovf is set where they do not.  first[c *
// stride] is the row of the chunk's first element.
__global__ void chunk_colbase_kernel(const int *__restrict__ rp, const int *__restrict__ ci,
                                     const int *__restrict__ arp, const int *__restrict__ first,
                                     int stride, int m, int nnz, long long nchunks, long long L,
                                     int *__restrict__ colbase, int *__restrict__ ovf) {
    const int lane = threadIdx.x & 31;
    const long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= nchunks) return;  // warp-uniform
    // CSR position of the augmented element that chunk q starts with
    auto pos = [&](long long q) -> int {
        if (q >= nchunks) return nnz;
        const int r = first[q * stride];
        if (r >= m) return nnz;
        const int len = rp[r + 1] - rp[r];
        const long long off = q * L - arp[r];
        return rp[r] + (int)(off > len ? len : off);
    };
    const int p0 = pos(c), p1 = pos(c + 1);
    int mn = 0x7fffffff, mx = -1;
#pragma unroll 8
    for (int p = p0 + lane; p < p1; p += 32) {
        const int col = ci[p];
        mn = col < mn ? col : mn;
        mx = col > mx ? col : mx;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int a = __shfl_xor_sync(FULL, mn, o), b = __shfl_xor_sync(FULL, mx, o);
        mn = a < mn ? a : mn;
        mx = b > mx ? b : mx;
    }
    if (lane == 0) {
        colbase[c] = mx >= 0 ? (int)(((long long)mn + mx) / 2) : 0;
        if (mx >= 0 && (long long)mx - mn > 65534) atomicOr(ovf, 1);
    }
}

// Block b: the distinct lines (16 columns) of LINE_WINDOW consecutive nonzeros from its part of the
// matrix, counted in a bitmap of hashed line numbers.
__global__ void __launch_bounds__(256)
sample_lines_kernel(const int *__restrict__ ci, int nnz, int *__restrict__ lines) {
    constexpr int WORDS = 1024;  // 32 K bits for at most 1,024 lines
    __shared__ unsigned bits[WORDS];
    for (int i = threadIdx.x; i < WORDS; i += 256) bits[i] = 0;
    __syncthreads();
    const long long p0 = (long long)(nnz - LINE_WINDOW) * blockIdx.x / LINE_WINDOWS;
    for (int i = threadIdx.x; i < LINE_WINDOW; i += 256) {
        const unsigned h = ((unsigned)ci[p0 + i] >> 4) * 2654435761u >> 17;
        atomicOr(&bits[h >> 5], 1u << (h & 31));
    }
    __syncthreads();
    int n = 0;
    for (int i = threadIdx.x; i < WORDS; i += 256) n += __popc(bits[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(FULL, n, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(lines, n);
}

}  // namespace

cudaError_t sample_lines(const int *ci, int nnz, int *lines, cudaStream_t s) {
    const cudaError_t e = cudaMemsetAsync(lines, 0, sizeof(int), s);
    if (e != cudaSuccess || nnz < LINE_WINDOW) return e;  // too small to matter: not scattered
    sample_lines_kernel<<<LINE_WINDOWS, 256, 0, s>>>(ci, nnz, lines);
    return cudaGetLastError();
}

cudaError_t launch_validate(const int *rp, const int *ci, int m, int n, int nnz, int *d_err,
                            bool want_longest, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(d_err, 0, sizeof(int) * (want_longest ? 2 : 1), s);
    if (e != cudaSuccess) return e;
    long long work = (long long)(m > nnz / 4 ? m : nnz / 4);
    long long blocks = (work + 255) / 256;
    if (blocks < 1) blocks = 1;
    if (blocks > 148 * 16) blocks = 148 * 16;
    validate_kernel<<<(unsigned)blocks, 256, 0, s>>>(rp, ci, m, n, nnz, d_err,
                                                     want_longest ? d_err + 1 : nullptr);
    return cudaGetLastError();
}

cudaError_t chunk_rows(const int *arp, int m, long long T, long long count, int *rows,
                       cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    chunk_rows_kernel<<<(unsigned)(((long long)m + 1 + 255) / 256), 256, 0, s>>>(arp, m, T, count,
                                                                                 rows);
    return cudaGetLastError();
}

cudaError_t chunk_colbase(const Handle &h, const int *rp, const int *ci, const int *first,
                          int stride, int *ovf, cudaStream_t s) {
    if (h.nchunks <= 0) return cudaSuccess;
    chunk_colbase_kernel<<<(unsigned)((h.nchunks * 32 + 255) / 256), 256, 0, s>>>(
        rp, ci, h.arp, first, stride, h.m, h.nnz, h.nchunks, h.L, h.colbase, ovf);
    return cudaGetLastError();
}

cudaError_t build_augmented_rowptr(const int *rp, int m, int *arp, int *d_nempty,
                                   cudaStream_t s) {
    // empties[r] = number of empty rows before r (exclusive scan of the empty-row flags)
    int *empties = nullptr;
    cudaError_t e = pool_malloc(&empties, (size_t)m + 1, s);
    if (e != cudaSuccess) return e;
    auto flags = thrust::make_transform_iterator(thrust::make_counting_iterator(0), EmptyRow{rp});
    // empties[0] = 0, empties[1..m] = inclusive scan of flag(0..m-1)
    size_t tmp_bytes = 0;
    cub::DeviceScan::InclusiveSum(nullptr, tmp_bytes, flags, empties + 1, m, s);
    void *tmp = nullptr;
    e = pool_malloc(&tmp, tmp_bytes, s);
    if (e != cudaSuccess) { pool_free(empties, s); return e; }
    cudaMemsetAsync(empties, 0, sizeof(int), s);
    if (m > 0) cub::DeviceScan::InclusiveSum(tmp, tmp_bytes, flags, empties + 1, m, s);
    arp_kernel<<<(unsigned)(((long long)m + 1 + 255) / 256), 256, 0, s>>>(rp, empties, m, arp);
    cudaMemcpyAsync(d_nempty, empties + m, sizeof(int), cudaMemcpyDeviceToDevice, s);
    pool_free(tmp, s);
    pool_free(empties, s);
    return cudaGetLastError();
}

cudaError_t set_int(int *p, int v, cudaStream_t s) {
    set_int_kernel<<<1, 1, 0, s>>>(p, v);
    return cudaGetLastError();
}

cudaError_t carry_fixup(const Handle &h, void *y, cudaStream_t s, bool fresh) {
    if (h.nchunks <= 0) return cudaSuccess;
    const long long blocks = (h.nchunks + 127) / 128;
    return launch_product(fresh ? carry_fixup_kernel<true> : carry_fixup_kernel<false>, (unsigned)blocks, 128, 0, s, (const char *)h.meta,
                          h.meta_stride, h.arp, h.L, h.carry_head, h.carry_tail, (double *)y,
                          h.nchunks, h.m, guard_word());
}

}  // namespace pava
