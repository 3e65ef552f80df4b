// COO -> sorted CSR on the device: the GPU form of the loader's conversion (readCOOMatrix's
// symmetric expansion and 1-based shift, utils/basicMatrix.cpp:63-253, and convertCOO2CSR,
// :350-415, which calls MKL's mkl_dcsrcoo there).
//
// Rows and the columns inside a row come out ascending and duplicates stay as separate entries in
// input order -- the same result as the host conversion, pava_coo_to_csr.  With `symmetric`,
// every off-diagonal entry (r, c) also yields (c, r), as a symmetric Matrix Market file stores
// one triangle; among equal (row, column) the entries come before the mirrored ones.
//
// The entries are bucketed by row (count, scan, scatter) and each row is sorted by (column,
// mirrored, input position), which are all different, so the result does not depend on the order
// in which the scatter's atomics ran.  Against one stable radix sort of (row << 32 | column) with
// its values -- 7 passes of 32 bytes per entry -- an entry is written and read once as a 16-byte
// record: 80^3 stencil from its triangle (6.9 M entries, 13.6 M nonzeros) 1.50 -> 0.30 ms of
// kernels.

#include <string.h>

#include <cub/cub.cuh>

#include "pava_internal.h"

namespace pava {

namespace {

unsigned grid_of(long long work, long long cap) {
    long long b = (work + 255) / 256;
    if (b < 1) b = 1;
    if (b > cap) b = cap;
    return (unsigned)b;
}

struct CooStat {
    unsigned long long mirrored;  // entries the symmetric expansion adds
    unsigned long long longs;     // rows longer than RANK_MAX << 32 | their nonzeros
    int bad, longest;             // entries outside the matrix, nonzeros of the longest long row
};

// A record of the scatter: key = column << 32 | mirrored << 31 | input position, and the value.
struct CooRec {
    unsigned long long key;
    double val;
};

// Adds `on` lanes' counts to their rows' counters and returns the lane's slot: one atomic per run of
// equal rows in neighbouring lanes (sorted inputs have long ones).  Where a lane's row is also that
// of the lane half a warp away and there are MATCH_MIN runs, one per different row: the atomics of a
// hot row in shuffled order go to one address, 0.3 ns each.  Whole conversion of 20 M entries, half
// of them in one row, shuffled: 8.05 -> 2.34 ms; in two rows that alternate 15.4 -> 3.4; random
// rows, which pay for the test, 1.19 -> 1.22, with every warp matched 1.23 (row order 0.77 -> 0.89
// then, 0.75 with the test).  All 32 lanes.
constexpr int MATCH_MIN = 8;
__device__ __forceinline__ int run_add(int *cnt, int row, bool on, int lane) {
    const int left = __shfl_up_sync(FULL, row, 1);
    const unsigned act = __ballot_sync(FULL, on);
    const bool lead = on && (lane == 0 || !((act >> (lane - 1)) & 1u) || left != row);
    const unsigned leads = __ballot_sync(FULL, lead);
    const int across = __shfl_xor_sync(FULL, row, 16);
    const bool far = on && ((act >> (lane ^ 16)) & 1u) && across == row;
    if (__popc(leads) >= MATCH_MIN && __any_sync(FULL, far)) {
        const unsigned same = __match_any_sync(FULL, on ? row : -1);
        const int first = __ffs(same) - 1;
        int base = 0;
        if (on && lane == first) base = atomicAdd(&cnt[row], __popc(same));
        base = __shfl_sync(FULL, base, first);
        return base + __popc(same & ((1u << lane) - 1u));
    }
    // a run ends before the next leader or the next inactive lane
    int base = 0, src = lane;
    if (on) src = 31 - __clz(leads & (0xffffffffu >> (31 - lane)));
    if (lead) {
        const unsigned stop = (leads | ~act) & ~(0xffffffffu >> (31 - lane));
        const int end = stop ? __ffs(stop) - 1 : 32;
        base = atomicAdd(&cnt[row], end - lane);
    }
    base = __shfl_sync(FULL, base, src);
    return base + (lane - src);
}

// Entries per row (mirrored ones included); counts indices out of range.
__global__ void __launch_bounds__(256)
coo_count_kernel(const int *__restrict__ rows, const int *__restrict__ cols, long long nnz,
                 int base, int m, int n, int symmetric, int *__restrict__ cnt,
                 CooStat *__restrict__ st) {
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    int nb = 0, nm = 0;
    for (long long k0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); k0 < nnz;
         k0 += stride) {
        const long long k = k0 + lane;
        const bool in = k < nnz;
        const long long r = in ? (long long)rows[k] - base : -1, c = in ? (long long)cols[k] - base : -1;
        const bool ok = r >= 0 && r < m && c >= 0 && c < n && (!symmetric || (c < m && r < n));
        nb += in && !ok;
        run_add(cnt, (int)r, ok, lane);
        if (symmetric) {
            const bool mir = ok && r != c;
            nm += mir;
            run_add(cnt, (int)c, mir, lane);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nb += __shfl_xor_sync(FULL, nb, o);
        nm += __shfl_xor_sync(FULL, nm, o);
    }
    // one atomic per block: all of them go to the same address
    __shared__ int s_bad, s_mir;
    if (threadIdx.x == 0) s_bad = s_mir = 0;
    __syncthreads();
    if (lane == 0 && nb) atomicAdd(&s_bad, nb);
    if (lane == 0 && nm) atomicAdd(&s_mir, nm);
    __syncthreads();
    if (threadIdx.x == 0 && s_bad) atomicAdd(&st->bad, s_bad);
    if (threadIdx.x == 0 && s_mir) atomicAdd(&st->mirrored, (unsigned long long)s_mir);
}

// Rows are sorted by counting, for each entry, the smaller keys of its row: up to RANK_MAX
// entries.  Longer rows are listed here, with ascending places in the packed array (one atomic
// hands out both: rows and nonzeros are below 2^31), and sorted by cub.
constexpr int RANK_MAX = 256;
__global__ void coo_long_kernel(const int *__restrict__ cnt, int m, CooStat *__restrict__ st,
                                const int *__restrict__ rp, int *__restrict__ row,
                                int *__restrict__ begin, int *__restrict__ end) {
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m) return;
    const int len = cnt ? cnt[r] : rp[r + 1] - rp[r];
    if (len <= RANK_MAX) return;
    const unsigned long long at = atomicAdd(&st->longs, (1ull << 32) | (unsigned)len);
    const unsigned q = (unsigned)(at >> 32), off = (unsigned)at;
    if (!row) {
        atomicMax(&st->longest, len);
    } else {
        row[q] = (int)r;
        begin[q] = (int)off;
        end[q] = (int)off + len;
    }
}

// Entry k into the next free slot of its row (cur: the rows' cursors, starting at rp).
__global__ void __launch_bounds__(256)
coo_scatter_kernel(const int *__restrict__ rows, const int *__restrict__ cols,
                   const double *__restrict__ vals, long long nnz, int base, int symmetric,
                   int *__restrict__ cur, CooRec *__restrict__ rec) {
    const int lane = threadIdx.x & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); k0 < nnz;
         k0 += stride) {
        const long long k = k0 + lane;
        const bool in = k < nnz;
        const int r = in ? rows[k] - base : -1, c = in ? cols[k] - base : -1;
        const double v = in ? vals[k] : 0.0;
        auto put = [&](int at, int col, unsigned tie) {
            const unsigned long long key = ((unsigned long long)(unsigned)col << 32) | tie;
            *reinterpret_cast<ulonglong2 *>(rec + at) =
                make_ulonglong2(key, (unsigned long long)__double_as_longlong(v));
        };
        const int at = run_add(cur, r, in, lane);
        if (in) put(at, c, (unsigned)k);
        if (symmetric) {
            const bool mir = in && r != c;
            const int at2 = run_add(cur, c, mir, lane);
            if (mir) put(at2, r, (unsigned)k | 0x80000000u);
        }
    }
}

// A warp per 32 rows, in batches of whole rows of at most CAP entries: keys in shared memory, an
// entry's place in its row is the number of smaller keys there.  Bound by the shared-memory reads
// (row length per entry) and the bytes (16 read, 12 written).
constexpr int SORT_WARPS = 4, CAP = 512;
static_assert(RANK_MAX <= CAP, "a row fits a batch");
__global__ void __launch_bounds__(SORT_WARPS * 32)
coo_sort_kernel(const int *__restrict__ rp, int m, const CooRec *__restrict__ rec,
                int *__restrict__ ci, double *__restrict__ v) {
    __shared__ unsigned long long s_key[SORT_WARPS][CAP];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long r = ((long long)blockIdx.x * SORT_WARPS + w) * 32 + lane;
    if (r - lane >= m) return;  // warp-uniform: no block-wide barrier below
    const int s = rp[r < m ? r : m], e = rp[r < m ? r + 1 : m];
    const bool is_long = e - s > RANK_MAX;
    unsigned long long *key = s_key[w];
    int i = 0;
    while (i < 32) {  // rows [i, j) of the 32
        const int base = __shfl_sync(FULL, s, i);
        const unsigned stop = __ballot_sync(FULL, lane >= i && (is_long || e - base > CAP));
        const int j = stop ? __ffs(stop) - 1 : 32;
        if (j == i) {  // a long row
            ++i;
            continue;
        }
        const int n = __shfl_sync(FULL, e, j - 1) - base;
        for (int q = lane; q < n; q += 32) key[q] = rec[base + q].key;
        __syncwarp();
        for (int q0 = 0; q0 < n; q0 += 32) {
            const int q = q0 + lane < n ? q0 + lane : n - 1;
            int row = i;  // the last row of the batch that starts at or before q
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                const int t = row + d;
                const int st = __shfl_sync(FULL, s, t & 31) - base;
                if (t < j && st <= q) row = t;
            }
            const int a = __shfl_sync(FULL, s, row) - base, b = __shfl_sync(FULL, e, row) - base;
            const unsigned long long mine = key[q];
            int rank = 0;
#pragma unroll 4
            for (int t = a; t < b; ++t) rank += key[t] < mine;
            if (q0 + lane < n) {
                ci[base + a + rank] = (int)(mine >> 32);
                v[base + a + rank] = rec[base + q].val;
            }
        }
        __syncwarp();  // the next batch overwrites the keys
        i = j;
    }
}

// Long rows: keys out to a packed array, and the sorted keys back as columns and values.
__global__ void coo_long_pack_kernel(const int *__restrict__ rp, const int *__restrict__ row,
                                     const int *__restrict__ begin, const CooRec *__restrict__ rec,
                                     unsigned long long *__restrict__ keys) {
    const int r = row[blockIdx.x], a = rp[r], len = rp[r + 1] - a, o = begin[blockIdx.x];
    for (int t = threadIdx.x; t < len; t += blockDim.x) keys[o + t] = rec[a + t].key;
}
__global__ void coo_long_unpack_kernel(const int *__restrict__ rp, const int *__restrict__ row,
                                       const int *__restrict__ begin,
                                       const unsigned long long *__restrict__ keys,
                                       const double *__restrict__ vals, int *__restrict__ ci,
                                       double *__restrict__ v) {
    const int r = row[blockIdx.x], a = rp[r], len = rp[r + 1] - a, o = begin[blockIdx.x];
    for (int t = threadIdx.x; t < len; t += blockDim.x) {
        const unsigned long long key = keys[o + t];
        ci[a + t] = (int)(key >> 32);
        v[a + t] = vals[key & 0x7fffffffull];
    }
}

// cub's segmented sort and the two kernels above give a row to one block, about 13 ns per entry: a
// row of 20 M entries took 390 ms.  Where the longest row has WIDE_MIN entries and there is less to
// sort than WIDE_ROWS such rows, all long rows are sorted by the whole device instead: a radix sort
// of the keys, then, where there are several rows, a stable one of the rows' numbers in the list.
// Whole conversion, segmented / wide: one row of 8000 225 / 201 us, of 32000 515 / 201, of 3 M
// 40.6 / 0.59 ms, of 20 M 390 / 2.9 ms; 100 rows of 8000 265 / 318 us, of 16000 411 / 440, of
// 32000 742 / 663; 300 rows of 16000 780 / 934 us, of 32000 1.52 / 1.61 ms.
constexpr int WIDE_MIN = 16384, WIDE_ROWS = 148;

// Packed place t -> the listed row that holds it: the last one that begins at or before t.
__device__ __forceinline__ int listed_row(const int *__restrict__ begin, int nl, int t) {
    int lo = 0, hi = nl;
    while (hi - lo > 1) {
        const int mid = lo + (hi - lo) / 2;
        if (begin[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}
__global__ void __launch_bounds__(256)
coo_wide_pack_kernel(const int *__restrict__ rp, const int *__restrict__ row,
                     const int *__restrict__ begin, int nl, int total,
                     const CooRec *__restrict__ rec, unsigned long long *__restrict__ keys,
                     int *__restrict__ which) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int q = listed_row(begin, nl, (int)t);
    keys[t] = rec[rp[row[q]] + ((int)t - begin[q])].key;
    if (which) which[t] = q;
}
__global__ void __launch_bounds__(256)
coo_wide_unpack_kernel(const int *__restrict__ rp, const int *__restrict__ row,
                       const int *__restrict__ begin, int total,
                       const unsigned long long *__restrict__ keys, const int *__restrict__ which,
                       const double *__restrict__ vals, int *__restrict__ ci,
                       double *__restrict__ v) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int q = which ? which[t] : 0;
    const int at = rp[row[q]] + ((int)t - begin[q]);
    const unsigned long long key = keys[t];
    ci[at] = (int)(key >> 32);
    v[at] = vals[key & 0x7fffffffull];
}

int bits_of(unsigned x) {  // of the values below x
    int b = 1;
    while (b < 32 && (x - 1) >> b) ++b;
    return b;
}

// The long rows' entries from rec, sorted, into ci and v.  `held` takes what is still to be freed.
// Once packed, rec is where the sorts put their other copy: it is read last by the pack kernels.
cudaError_t sort_long_rows(int m, int n, const CooStat &h, CooStat *d_st, const int *rp,
                           CooRec *rec, const double *vals, int *ci, double *v, void **held,
                           cudaStream_t s) {
    const int nl = (int)(h.longs >> 32), lt = (int)(unsigned)h.longs;
    const bool wide = h.longest >= WIDE_MIN && lt / h.longest < WIDE_ROWS;
    const bool several = wide && nl > 1;
    const size_t n_l = (size_t)nl, n_t = (size_t)lt;
    int *seg = nullptr, *which = nullptr;
    unsigned long long *keys = nullptr;
    cudaError_t e = pool_malloc(&seg, 3 * n_l, s);
    held[0] = seg;
    if (e == cudaSuccess) e = pool_malloc(&keys, n_t, s);
    held[1] = keys;
    if (e == cudaSuccess && several) e = pool_malloc(&which, n_t, s);
    held[2] = which;
    if (e == cudaSuccess) e = cudaMemsetAsync(d_st, 0, sizeof(CooStat), s);
    if (e != cudaSuccess) return e;
    const int *row = seg, *begin = seg + n_l, *end = seg + 2 * n_l;
    coo_long_kernel<<<(unsigned)(((long long)m + 255) / 256), 256, 0, s>>>(
        nullptr, m, d_st, rp, seg, seg + n_l, seg + 2 * n_l);
    const unsigned blocks = (unsigned)((n_t + 255) / 256);
    if (wide)
        coo_wide_pack_kernel<<<blocks, 256, 0, s>>>(rp, row, begin, nl, lt, rec, keys, which);
    else
        coo_long_pack_kernel<<<(unsigned)nl, 256, 0, s>>>(rp, row, begin, rec, keys);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // Two buffers each: a sort leaves its result in either
    cub::DoubleBuffer<unsigned long long> kb(keys, reinterpret_cast<unsigned long long *>(rec));
    cub::DoubleBuffer<int> wb(which, which ? reinterpret_cast<int *>(rec) + 2 * n_t : nullptr);
    const int key_bits = 32 + bits_of((unsigned)n), row_bits = bits_of((unsigned)nl);
    auto sort = [&](int step, void *tmp, size_t &tb) {
        if (!wide) return cub::DeviceSegmentedSort::SortKeys(tmp, tb, kb, lt, nl, begin, end, s);
        if (!several) return cub::DeviceRadixSort::SortKeys(tmp, tb, kb, lt, 0, key_bits, s);
        if (step == 0) return cub::DeviceRadixSort::SortPairs(tmp, tb, kb, wb, lt, 0, key_bits, s);
        return cub::DeviceRadixSort::SortPairs(tmp, tb, wb, kb, lt, 0, row_bits, s);
    };
    size_t tb = 0, tb2 = 0;
    e = sort(0, nullptr, tb);
    if (e == cudaSuccess && several) e = sort(1, nullptr, tb2);
    if (tb < tb2) tb = tb2;
    char *tmp = nullptr;
    if (e == cudaSuccess) e = pool_malloc(&tmp, tb, s);
    held[3] = tmp;
    if (e == cudaSuccess) e = sort(0, tmp, tb);
    if (e == cudaSuccess && several) e = sort(1, tmp, tb);
    if (e != cudaSuccess) return e;
    if (wide)
        coo_wide_unpack_kernel<<<blocks, 256, 0, s>>>(rp, row, begin, lt, kb.Current(),
                                                      wb.Current(), vals, ci, v);
    else
        coo_long_unpack_kernel<<<(unsigned)nl, 256, 0, s>>>(rp, row, begin, kb.Current(), vals, ci,
                                                           v);
    return cudaGetLastError();
}

}  // namespace

}  // namespace pava

namespace {

// pooled: the result's arrays come from the library's memory pool, else from cudaMalloc, which CUDA
// IPC and peer access need.
pava_status coo_to_csr(int m, int n, long long nnz, const int *rows, const int *cols,
                       const double *vals, int index_base, int symmetric, void *stream,
                       pava_csr *out, bool pooled) {
    using namespace pava;
    if (!out) { set_last_error("out is NULL"); return PAVA_E_INVALID_ARG; }
    memset(out, 0, sizeof(*out));
    if (m < 0 || n < 0 || nnz < 0 || (nnz > 0 && (!rows || !cols || !vals)) ||
        (index_base != 0 && index_base != 1)) {
        set_last_error("bad sizes, NULL arrays or index base other than 0 / 1");
        return PAVA_E_INVALID_ARG;
    }
    if (nnz > 2147483000LL) { set_last_error("more than 2^31 entries"); return PAVA_E_TOO_LARGE; }
    cudaStream_t s = (cudaStream_t)stream;
    int *cnt = nullptr, *cur = nullptr, *rp = nullptr, *ci = nullptr;
    CooStat *d_st = nullptr;
    CooRec *rec = nullptr;
    double *v = nullptr;
    void *tmp = nullptr, *held_long[4] = {};
    // it allocates and waits: not on a stream that is being captured.  Nothing is held yet, and a
    // wait or a trim here would end the caller's capture.
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s, &capturing);
    if (e == cudaSuccess && capturing != cudaStreamCaptureStatusNone)
        e = cudaErrorStreamCaptureUnsupported;
    if (e != cudaSuccess) {
        set_last_error(std::string("COO -> CSR: ") + cudaGetErrorString(e));
        return PAVA_E_CUDA;
    }
    const size_t held = pool_reserved();
    auto cleanup = [&]() {
        pool_free(cnt, s); pool_free(cur, s); pool_free(d_st, s); pool_free(rec, s);
        pool_free(tmp, s);
        for (void *p : held_long) pool_free(p, s);
    };
    auto give_back = [&]() {
        cleanup();
        if (pooled) { pool_free(rp, s); pool_free(ci, s); pool_free(v, s); }
        cudaStreamSynchronize(s);
        if (!pooled) { cudaFree(rp); cudaFree(ci); cudaFree(v); }
        pool_trim(held);
    };
    auto result_malloc = [&](auto **p, size_t count) {
        return pooled ? pool_malloc(p, count, s) : plain_malloc((void **)p, sizeof(**p) * (count ? count : 1));
    };
    auto fail_e = [&](cudaError_t err) {
        give_back();
        set_last_error(std::string("COO -> CSR: ") + cudaGetErrorString(err));
        return err == cudaErrorMemoryAllocation ? PAVA_E_NOMEM : PAVA_E_CUDA;
    };
    // entries per row -> row pointer
    e = pool_malloc(&cnt, (size_t)m + 1, s);
    if (e == cudaSuccess) e = result_malloc(&rp, (size_t)m + 1);
    if (e == cudaSuccess) e = pool_malloc(&d_st, 1, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, sizeof(int) * ((size_t)m + 1), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_st, 0, sizeof(CooStat), s);
    if (e == cudaSuccess && nnz > 0) {
        coo_count_kernel<<<grid_of(nnz, 148 * 16), 256, 0, s>>>(rows, cols, nnz, index_base, m, n, symmetric,
                                                      cnt, d_st);
        e = cudaGetLastError();
    }
    const unsigned row_blocks = (unsigned)(((long long)m + 255) / 256);
    if (e == cudaSuccess && m > 0) {
        coo_long_kernel<<<row_blocks, 256, 0, s>>>(cnt, m, d_st, nullptr, nullptr, nullptr, nullptr);
        e = cudaGetLastError();
    }
    size_t tb = 0;
    if (e == cudaSuccess)
        e = cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, rp, (long long)m + 1, s);
    if (e == cudaSuccess) e = pool_malloc(&tmp, tb, s);
    if (e == cudaSuccess)
        e = cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, rp, (long long)m + 1, s);
    CooStat h = {};
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d_st, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail_e(e);
    if (h.bad) {
        give_back();
        set_last_error("COO -> CSR: " + std::to_string(h.bad) + " entries outside the matrix");
        return PAVA_E_INVALID_CSR;
    }
    const long long total = nnz + (long long)h.mirrored;
    if (total > 2147483000LL) {
        give_back();
        set_last_error("more than 2^31 entries after the symmetric expansion");
        return PAVA_E_TOO_LARGE;
    }
    const size_t tz = (size_t)(total ? total : 1);
    if (e == cudaSuccess) e = result_malloc(&ci, tz);
    if (e == cudaSuccess) e = result_malloc(&v, tz);
    if (total > 0) {
        if (e == cudaSuccess) e = pool_malloc(&rec, tz, s);
        cur = cnt;  // the counts are in rp: their array becomes the rows' cursors
        cnt = nullptr;
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(cur, rp, sizeof(int) * (size_t)m, cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) {
            coo_scatter_kernel<<<grid_of(nnz, 16384), 256, 0, s>>>(rows, cols, vals, nnz, index_base,
                                                            symmetric, cur, rec);
            const long long warps = ((long long)m + 31) / 32;
            coo_sort_kernel<<<(unsigned)((warps + SORT_WARPS - 1) / SORT_WARPS), SORT_WARPS * 32, 0,
                              s>>>(rp, m, rec, ci, v);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess && h.longs)
        e = sort_long_rows(m, n, h, d_st, rp, rec, vals, ci, v, held_long, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail_e(e);
    cleanup();
    out->m = m;
    out->n = n;
    out->nnz = (int)total;
    out->row_ptr = rp;
    out->col_idx = ci;
    out->vals = v;
    out->on_device = 1;
    return PAVA_SUCCESS;
}

}  // namespace

extern "C" {

pava_status pava_coo_to_csr_device(int m, int n, long long nnz, const int *rows, const int *cols,
                                   const double *vals, int index_base, int symmetric, void *stream,
                                   pava_csr *out) {
    return coo_to_csr(m, n, nnz, rows, cols, vals, index_base, symmetric, stream, out, false);
}

pava_status pava_coo_to_csr_device_pooled(int m, int n, long long nnz, const int *rows,
                                          const int *cols, const double *vals, int index_base,
                                          int symmetric, void *stream, pava_csr *out) {
    return coo_to_csr(m, n, nnz, rows, cols, vals, index_base, symmetric, stream, out, true);
}

pava_status pava_free_device_csr_async(pava_csr *A, void *stream) {
    if (!A) return PAVA_SUCCESS;
    if (A->on_device) {
        pava::pool_free((void *)A->row_ptr, (cudaStream_t)stream);
        pava::pool_free((void *)A->col_idx, (cudaStream_t)stream);
        pava::pool_free((void *)A->vals, (cudaStream_t)stream);
    }
    memset(A, 0, sizeof(*A));
    return PAVA_SUCCESS;
}

}  // extern "C"
