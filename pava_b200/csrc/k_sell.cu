// Sliced ELLPACK (SELL): conversion and SpMV for sm_100a.
//
// A slice is 32 consecutive rows, one per lane of a warp.  Each slice stores its rows padded to
// the length of its longest row (rounded up to 4), in the 4-step block layout of k_stream.cuh:
// element i of the slice's lane k (row 32 s + k) sits at off_s + vals_offset(i, k), so at step
// i the 32 lanes read one 16-byte vector each per stream and gather x for the i-th nonzero of
// 32 consecutive rows.  On matrices whose neighbouring rows have the same pattern (stencils,
// banded and block structures) those 32 gathers land on one or two 128-byte lines, where the
// CVR and CSR5 walks (a lane runs through consecutive nonzeros of a few rows) spread them over
// many lines.  Every row is summed by one lane from its first to its last nonzero, so there
// are no row-start flags, no cross-lane combine and no carries: one pass, one coalesced y
// store per slice, no fixup launch.  Padding elements (value 0, no column) read no x.
//
// The SpMV stages the value and column streams through shared memory with bulk asynchronous
// copies (cp.async.bulk, completion counted on an mbarrier): a warp keeps two pieces of its
// slices in flight in its own shared-memory stages while it sums a third from shared memory,
// so the bytes in flight per SM are set by shared memory (~200 KB), not by registers.
//
// The price is the padding, so the form is for matrices whose rows in a slice have similar
// lengths; pava_create refuses it (PAVA_E_UNSUPPORTED_PARAMS) when padding would more than
// double the stored elements.  No counterpart in the reference (pava's engines are CVR and
// CSR5); it is a third engine form beside them, offered by the autotuner and the selector.

#include <atomic>
#include <climits>

#include <cub/cub.cuh>

#include "k_bulk.cuh"
#include "k_stream.cuh"
#include "pava_internal.h"

namespace pava {

namespace {

constexpr int SELL_WARPS = 8;

// Warp per slice: the slice's blocks of 4 steps (its longest row, rounded up), whether any lane
// pads, and (for 16-bit offsets) the base column, the middle of the slice's column range; *ovf is
// set where that range is too wide for them.  A slice's columns are contiguous in the CSR and
// read in order (row by row per lane they took 38 us for 25 M nonzeros).
__global__ void sell_plan_kernel(const int *__restrict__ rp, const int *__restrict__ ci, int m,
                                 long long nslices, int want_base, SellSlice *__restrict__ meta,
                                 int *__restrict__ nblk_out, int *__restrict__ ovf) {
    const int lane = threadIdx.x & 31;
    const long long s = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (s >= nslices) return;  // warp-uniform
    const long long r = s * 32 + lane;
    const int a = r < m ? rp[r] : 0, len = r < m ? rp[r + 1] - a : 0;
    int mx = len;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int t = __shfl_xor_sync(FULL, mx, o);
        mx = t > mx ? t : mx;
    }
    const int nblk = (mx + 3) / 4;
    const bool pads = __any_sync(FULL, len < 4 * nblk);
    int mn = len;  // the shortest row: blocks before mn / 4 hold no padding
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int t = __shfl_xor_sync(FULL, mn, o);
        mn = t < mn ? t : mn;
    }
    int cmin = 0x7fffffff, cmax = -1;
    if (want_base) {
        const int last = (int)(m - s * 32 < 32 ? m - s * 32 : 32) - 1;
        const int p0 = __shfl_sync(FULL, a, 0), p1 = __shfl_sync(FULL, a + len, last);
#pragma unroll 8
        for (int p = p0 + lane; p < p1; p += 32) {
            const int c = ci[p];
            cmin = c < cmin ? c : cmin;
            cmax = c > cmax ? c : cmax;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int u = __shfl_xor_sync(FULL, cmin, o), w = __shfl_xor_sync(FULL, cmax, o);
            cmin = u < cmin ? u : cmin;
            cmax = w > cmax ? w : cmax;
        }
    }
    if (lane == 0) {
        meta[s].off = 0;
        meta[s].nblk = nblk;
        meta[s].colbase = cmax >= 0 ? (int)(((long long)cmin + cmax) / 2) : 0;
        meta[s].flags = pads ? 1u | ((unsigned)(mn / 4) << 1) : 0u;
        nblk_out[s] = nblk;
        if (cmax >= 0 && (long long)cmax - cmin > 65534) atomicOr(ovf, 1);
    }
}

// Warp per slice: the slice's rows go into the block layout, padded with (0, no column), PS steps
// at a time through shared memory: each half-warp reads PS consecutive elements of a row (128
// bytes of values), and each lane then writes its own row's elements as whole vectors.  Bound by
// the bytes; with each lane reading its own row (32 L1 wavefronts per load) and writing 8-byte
// pieces it took 558 us for the 128^3 stencil in FP32, 259 us for 25 M banded nonzeros in FP64
// with 16-bit offsets; now 186 and 114 us.  blk_off[s] = the slice's first block.
constexpr int FILL_WARPS = 4, PS = 16;
template <typename VT, typename IT>
__global__ void __launch_bounds__(FILL_WARPS * 32)
sell_fill_kernel(const int *__restrict__ rp, const int *__restrict__ ci,
                 const double *__restrict__ v, int m, long long nslices,
                 const int *__restrict__ blk_off, SellSlice *__restrict__ meta,
                 VT *__restrict__ vals, IT *__restrict__ cols) {
    __shared__ VT s_val[FILL_WARPS][32 * (PS + 1)];
    __shared__ IT s_col[FILL_WARPS][32 * (PS + 1)];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long s = (long long)blockIdx.x * FILL_WARPS + w;
    if (s >= nslices) return;  // warp-uniform: no block-wide barrier below
    const long long off = (long long)blk_off[s] * 128;
    const int nblk = meta[s].nblk, base = meta[s].colbase;
    const long long r = s * 32 + lane;
    const int a = r < m ? rp[r] : 0, len = r < m ? rp[r + 1] - a : 0;
    VT *vo = vals + off;
    IT *co = cols + off;
    const int hi = lane >> 4, li = lane & (PS - 1);
    for (int b0 = 0; b0 < nblk; b0 += PS / 4) {
        const int i = 4 * b0 + li;
        constexpr int U = 8;  // pairs of rows in flight
#pragma unroll
        for (int k0 = 0; k0 < 32; k0 += 2 * U) {
            double val[U];
            int col[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = k0 + 2 * u + hi;
                const int ak = __shfl_sync(FULL, a, k), lk = __shfl_sync(FULL, len, k);
                val[u] = 0.0;
                col[u] = -1;
                if (i < lk) {
                    val[u] = v[ak + i];
                    col[u] = ci[ak + i];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int slot = (k0 + 2 * u + hi) * (PS + 1) + li;
                s_val[w][slot] = (VT)val[u];
                s_col[w][slot] = sizeof(IT) == 2 ? (IT)(col[u] < 0 ? DELTA_NONE : col[u] - base)
                                                 : (IT)col[u];
            }
        }
        __syncwarp();
        const VT *sv = &s_val[w][lane * (PS + 1)];
        const IT *sc = &s_col[w][lane * (PS + 1)];
#pragma unroll
        for (int q = 0; q < PS / 4; ++q) {
            const int b = b0 + q;
            if (b >= nblk) break;
            if constexpr (sizeof(VT) == 8) {
                double2 *o = reinterpret_cast<double2 *>(vo);
                o[(2 * b) * 32 + lane] = make_double2(sv[4 * q], sv[4 * q + 1]);
                o[(2 * b + 1) * 32 + lane] = make_double2(sv[4 * q + 2], sv[4 * q + 3]);
            } else {
                reinterpret_cast<float4 *>(vo)[b * 32 + lane] =
                    make_float4(sv[4 * q], sv[4 * q + 1], sv[4 * q + 2], sv[4 * q + 3]);
            }
            if constexpr (sizeof(IT) == 4)
                reinterpret_cast<int4 *>(co)[b * 32 + lane] =
                    make_int4(sc[4 * q], sc[4 * q + 1], sc[4 * q + 2], sc[4 * q + 3]);
            else
                reinterpret_cast<short4 *>(co)[b * 32 + lane] =
                    make_short4(sc[4 * q], sc[4 * q + 1], sc[4 * q + 2], sc[4 * q + 3]);
        }
        __syncwarp();  // the next steps overwrite the staged ones
    }
    if (lane == 0) meta[s].off = (int)off;
}

// Row sums.  FP64: FMA.  FP32 values and x: a product of two FP32 numbers is exact in FP64
// (24 + 24 significant bits < 53), so the FP32 form widens both factors and sums the exact
// products with FP64 FMAs -- an FP64 sum of exact terms, one rounding per nonzero.
template <typename VT> struct RowAcc;
template <> struct RowAcc<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double v, double x) { s = fma(v, x, s); }
    __device__ __forceinline__ double value() const { return s; }
    __device__ __forceinline__ void reset() { s = 0.0; }
};
template <> struct RowAcc<float> {
    double s = 0.0;
    __device__ __forceinline__ void add(float v, float x) { s = fma((double)v, (double)x, s); }
    __device__ __forceinline__ double value() const { return s; }
    __device__ __forceinline__ void reset() { s = 0.0; }
};

// Bulk-copy staging.  A stage holds one piece: up to KB consecutive blocks of one slice
// (KB = the blocks of about 3 KB of value and column stream); each warp owns STAGES stages and
// an mbarrier per stage; CTAS_PER_SM CTAs of SELL_WARPS warps share an SM.
constexpr int STAGE_BYTES = 3072, STAGES = 2, CTAS_PER_SM = 4;
template <typename VT, typename IT> struct Stage {
    static constexpr int BPB = 128 * (int)(sizeof(VT) + sizeof(IT));  // bytes per block
    static constexpr int KB = STAGE_BYTES / BPB > 0 ? STAGE_BYTES / BPB : 1;
    static constexpr int VBYTES = KB * 128 * (int)sizeof(VT), CBYTES = KB * 128 * (int)sizeof(IT);
    static constexpr int WARP_BYTES = STAGES * (VBYTES + CBYTES) + 128;  // + barriers
    static constexpr int CTA_BYTES = SELL_WARPS * WARP_BYTES;
    static_assert(STAGES * 8 <= 128 && WARP_BYTES % 128 == 0, "stage layout");
};

// SpMV.  Warps take slices in turn (grid-stride: the warps of the grid work on neighbouring
// slices at any time, so the streams are read close to in order).  Each warp walks its slices
// as a sequence of pieces (<= KB blocks of one slice) with two cursors: the producer (lane 0
// issues the bulk copies of a piece into the next free stage) runs STAGES pieces ahead of the
// consumer, which waits for its stage's copies, sums the piece's blocks from shared memory
// -- gathering the x of block i + 1 while block i is summed -- and hands the stage back.  A
// slice's last piece stores its 32 rows; empty slices (no blocks) store zero rows.  A wait
// that gives up counts itself in wait_err[0] (the first slice in wait_err[1]); the warp then
// waits, again bounded, for the copies it still has in flight and stops.
template <typename VT, typename IT>
__global__ void __launch_bounds__(SELL_WARPS * 32, CTAS_PER_SM)
sell_spmv_kernel(const SellSlice *__restrict__ meta, const VT *__restrict__ vals,
                 const IT *__restrict__ cols, const VT *x,
                 double *__restrict__ y, ChunkWalk<SELL_WARPS> walk, int m, int n,
                 unsigned long long *err, unsigned long long *wait_err) {
    using ST = Stage<VT, IT>;
    constexpr int KB = ST::KB;
    extern __shared__ __align__(128) unsigned char smem[];
    pdl_trigger();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned char *wbase = smem + w * ST::WARP_BYTES;  // [barriers | value stages | column stages]
    const unsigned bar0 = (unsigned)__cvta_generic_to_shared(wbase);
    const VT *sv = reinterpret_cast<const VT *>(wbase + 128);
    const IT *sc = reinterpret_cast<const IT *>(wbase + 128 + STAGES * ST::VBYTES);
    const unsigned sv0 = bar0 + 128, sc0 = bar0 + 128 + STAGES * ST::VBYTES;
    if (lane == 0) {
        for (int k = 0; k < STAGES; ++k) mbar_init(bar0 + 8 * k);
        mbar_init_fence();
    }
    __syncwarp();
    const uint64_t pl = policy_evict_last();
    const unsigned first = walk.first();

    // producer cursor: slice ps (with blocks), next block pb
    unsigned ps = first;
    int pb = 0;
    SellSlice pm{0, 0, 0, 0u};
    if (walk.ok(ps)) pm = meta[ps];
    while (walk.ok(ps) && pm.nblk == 0) {
        ps = walk.next(ps);
        if (walk.ok(ps)) pm = meta[ps];
    }
    auto issue = [&](int k) {
        const int len = min(KB, pm.nblk - pb);
        const long long e0 = (long long)pm.off + (long long)pb * 128;
        if (lane == 0) {
            const unsigned vb = (unsigned)(len * 128 * (int)sizeof(VT));
            const unsigned cb = (unsigned)(len * 128 * (int)sizeof(IT));
            proxy_fence();  // the stage's last reads come before the copy's writes
            mbar_expect_tx(bar0 + 8 * k, vb + cb);
            bulk_g2s(sv0 + k * ST::VBYTES, vals + e0, vb, bar0 + 8 * k);
            bulk_g2s(sc0 + k * ST::CBYTES, cols + e0, cb, bar0 + 8 * k);
        }
        pb += KB;
        if (pb >= pm.nblk) {
            pb = 0;
            do {
                ps = walk.next(ps);
                if (walk.ok(ps)) pm = meta[ps];
            } while (walk.ok(ps) && pm.nblk == 0);
        }
    };
    int pending = 0;
#pragma unroll
    for (int k = 0; k < STAGES; ++k)
        if (walk.ok(ps)) { issue(k); ++pending; }

    pdl_wait();  // x, and y, which the product before may still use: only copies of the format above

    // consumer cursor: slice cs, next block cb; it writes the rows of empty slices
    unsigned cs = first;
    int cb = 0;
    SellSlice cm{0, 0, 0, 0u};
    auto skip_empty = [&]() {
        while (walk.ok(cs)) {
            cm = meta[cs];
            if (cm.nblk > 0) break;
            const long long r = cs * 32ll + lane;
            if (r < m) y[r] = 0.0;
            cs = walk.next(cs);
        }
    };
    skip_empty();
    unsigned phases = 0;  // bit k: parity the consumer waits for on stage k
    int k = 0;
    RowAcc<VT> acc;
    while (walk.ok(cs)) {
        if (!mbar_wait(bar0 + 8 * k, (phases >> k) & 1u)) {
            if (lane == 0) {
                atomicAdd(&wait_err[0], 1ull);
                atomicCAS(&wait_err[1], 0ull, (unsigned long long)cs + 1);
            }
            break;
        }
        phases ^= 1u << k;
        --pending;
        const int len = min(KB, cm.nblk - cb);
        const VT *pv = sv + k * (ST::VBYTES / (int)sizeof(VT));
        const IT *pc = sc + k * (ST::CBYTES / (int)sizeof(IT));
        const int xbase = sizeof(IT) == 2 ? cm.colbase : 0;  // base of the 16-bit offsets
        const VT *xb = x + xbase;
        const int xlo = -xbase, xhi = n - xbase;
        // blocks from pad_from on hold padding: their gathers test each column
        const int pad_from = (cm.flags & 1u) ? (int)(cm.flags >> 1) - cb : INT_MAX;
        auto gather4 = [&](const CBlk<IT> &cbk, VT (&xs)[4], int i) {
            if (i >= pad_from) {
#pragma unroll
                for (int q = 0; q < 4; ++q) xs[q] = cbk.gather(q, xb, pl, xlo, xhi, err);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) xs[q] = cbk.gather_all(q, xb, pl, xlo, xhi, err);
            }
        };
        VT xs[2][4];
        gather4(CBlk<IT>::load_smem(pc, 0, lane), xs[0], 0);
#pragma unroll
        for (int i = 0; i < KB; ++i) {
            if (i < len) {
                if (i + 1 < len)
                    gather4(CBlk<IT>::load_smem(pc, i + 1, lane), xs[(i + 1) & 1], i + 1);
                const VBlk<VT> vv = VBlk<VT>::load_smem(pv, i, lane);
#pragma unroll
                for (int q = 0; q < 4; ++q) acc.add(vv.get(q), xs[i & 1][q]);
            }
        }
        cb += KB;
        if (cb >= cm.nblk) {  // the slice's last piece
            const long long r = cs * 32ll + lane;
            if (r < m) y[r] = acc.value();
            acc.reset();
            cb = 0;
            cs = walk.next(cs);
            skip_empty();
        }
        __syncwarp();  // every lane is done with stage k
        if (walk.ok(ps)) { issue(k); ++pending; }
        k = k + 1 == STAGES ? 0 : k + 1;
    }
    // only after a wait gave up: let the copies still in flight land before the CTA exits
    for (; pending > 0; --pending) {
        mbar_wait(bar0 + 8 * k, (phases >> k) & 1u);
        phases ^= 1u << k;
        k = k + 1 == STAGES ? 0 : k + 1;
    }
}

template <typename VT, typename IT>
cudaError_t fill_t(Handle &h, const int *rp, const int *ci, const double *v, const int *blk_off,
                   cudaStream_t s) {
    const long long ctas = (h.nchunks + FILL_WARPS - 1) / FILL_WARPS;
    sell_fill_kernel<VT, IT><<<(unsigned)ctas, FILL_WARPS * 32, 0, s>>>(
        rp, ci, v, h.m, h.nchunks, blk_off, (SellSlice *)h.meta, (VT *)h.vals, (IT *)h.cols);
    return cudaGetLastError();
}

template <typename VT, typename IT>
cudaError_t spmv_t(const Handle &h, const void *x, void *y, cudaStream_t s) {
    using ST = Stage<VT, IT>;
    // more than the default 48 KB of dynamic shared memory: opted into once per device
    static std::atomic<unsigned long long> opted{0};
    if (h.device < 0 || h.device >= 64) return cudaErrorInvalidDevice;
    const unsigned long long bit = 1ull << h.device;
    if (!(opted.load() & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(
            sell_spmv_kernel<VT, IT>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST::CTA_BYTES);
        if (e != cudaSuccess) return e;
        opted.fetch_or(bit);
    }
    const long long cap = (long long)h.sm_count * CTAS_PER_SM;
    const unsigned grid = (unsigned)(h.nchunks < cap ? h.nchunks : cap);
    return launch_product(sell_spmv_kernel<VT, IT>, grid, SELL_WARPS * 32, ST::CTA_BYTES, s,
                          (const SellSlice *)h.meta, (const VT *)h.vals, (const IT *)h.cols,
                          (const VT *)x, (double *)y, ChunkWalk<SELL_WARPS>::over(h.nchunks, grid),
                          h.m, h.n, guard_word(), wait_word());
}

}  // namespace

cudaError_t sell_plan(Handle &h, const int *rp, const int *ci, bool want_base, int *d_blk_off,
                      int *d_res, cudaStream_t s) {
    const long long ns = h.nchunks;
    const long long threads = ns * 32;
    int *nblk = nullptr;
    cudaError_t e = pool_malloc(&nblk, (size_t)(ns + 1), s);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(d_res + 1, 0, sizeof(int), s);
    if (e == cudaSuccess) {
        sell_plan_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(
            rp, ci, h.m, ns, want_base ? 1 : 0, (SellSlice *)h.meta, nblk, d_res + 1);
        e = cudaGetLastError();
    }
    // blk_off[0..ns] = exclusive scan of nblk (blk_off[ns] = total blocks)
    if (e == cudaSuccess) e = cudaMemsetAsync(nblk + ns, 0, sizeof(int), s);
    size_t tmp_bytes = 0;
    if (e == cudaSuccess)
        e = cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, nblk, d_blk_off, (int)(ns + 1), s);
    void *tmp = nullptr;
    if (e == cudaSuccess) e = pool_malloc(&tmp, tmp_bytes, s);
    if (e == cudaSuccess)
        e = cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, nblk, d_blk_off, (int)(ns + 1), s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_res, d_blk_off + ns, sizeof(int), cudaMemcpyDeviceToDevice, s);
    pool_free(tmp, s);
    pool_free(nblk, s);
    return e;
}

cudaError_t sell_fill(Handle &h, const int *rp, const int *ci, const double *v,
                      const int *d_blk_off, cudaStream_t s) {
    if (h.nchunks <= 0) return cudaSuccess;
    const bool f32 = h.precision == PAVA_PREC_FP32C, d16 = h.index_mode == PAVA_INDEX_DELTA16;
    if (!f32 && !d16) return fill_t<double, int>(h, rp, ci, v, d_blk_off, s);
    if (!f32 && d16) return fill_t<double, short>(h, rp, ci, v, d_blk_off, s);
    if (f32 && !d16) return fill_t<float, int>(h, rp, ci, v, d_blk_off, s);
    return fill_t<float, short>(h, rp, ci, v, d_blk_off, s);
}

cudaError_t sell_spmv(const Handle &h, const void *x, void *y, cudaStream_t s) {
    if (h.nchunks <= 0) return cudaSuccess;
    const bool f32 = h.precision == PAVA_PREC_FP32C, d16 = h.index_mode == PAVA_INDEX_DELTA16;
    if (!f32 && !d16) return spmv_t<double, int>(h, x, y, s);
    if (!f32 && d16) return spmv_t<double, short>(h, x, y, s);
    if (f32 && !d16) return spmv_t<float, int>(h, x, y, s);
    return spmv_t<float, short>(h, x, y, s);
}

}  // namespace pava
