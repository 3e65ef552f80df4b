// SELL SpMM: Y = A X for k right-hand sides (X row-major n x k, Y row-major m x k) on a SELL
// handle.
//
// A CTA of 32 G threads takes one 32-row slice at a time: G lanes per row (4, 8 or 16), 32 / G rows
// per warp.  Thread t owns row t / G of the slice and, of that row's k outputs, the KPL columns of
// slot g = t % G (VW = 2: the pairs g, g + G, ... of adjacent columns, each read as one vector)
// -- so the G lanes of a row read a whole row of X per nonzero, and each thread keeps its KPL sums
// in registers for the whole slice.  CTAs take runs of one or two neighbouring slices in
// turn.
//
// The slice's value and column streams come into shared memory by bulk asynchronous copies
// (k_bulk.cuh), KB blocks per piece, two pieces in flight per CTA: thread 0 issues the copies of
// the piece after next while the CTA sums the current one.  A row's four elements of a block are
// one 16-byte shared-memory read per stream (the G lanes of the row read the same address: a
// broadcast), where the row-group kernel (k_group.cu) passes every element to the lanes of its
// row by shuffles.  Padding (value 0, no column) reads a row of zeros instead of X; the blocks before
// the slice's shortest row ends carry no test for it.  The CTA meets once per piece: each thread
// waits for the copies on the mbarrier, and the barrier that hands the piece back also carries
// whether a wait gave up.
//
// What bounds it: the X reads, 8 k bytes per nonzero into registers (128 bytes per SM and clock:
// 179 us for 25 M banded nonzeros at k = 32) and their latency, so the reads of all four elements
// of a block are in flight before the first is used, without predicates, and the cursor of the
// copies lives in shared memory to leave the registers to them.  FP64, 32-bit / 16-bit columns,
// L2 flushed, against reads used one by one, a select per column for padding and two barriers per
// piece: banded (1,048,576 rows, 24 each) k = 8 195 / 202 -> 115 / 107 us, k = 32 336 / 357 -> 328 /
// 320; stencil 100^3 k = 8 181 / 189 -> 119 / 109, k = 32 335 / 390 -> 330 / 324; dense blocks
// (400,000 rows) k = 8 181 / 186 -> 82 / 78, k = 32 274 / 297 -> 261 / 258.  One 1,024-thread CTA per
// SM whose groups share runs of 8-32 slices raised the L1 hit rate from 75 to 90 % on the
// banded matrix and ran it like this form (k = 32: 317 us), but the blocks in 290.
//
// No counterpart in the reference (its SpMV takes one vector; main.cpp:554-587 runs one matrix
// and one vector at a time).

#include <atomic>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "k_bulk.cuh"
#include "k_stream.cuh"
#include "pava_internal.h"

namespace pava {

namespace {

// The shape of G lanes per row: 32 G threads per CTA (32 rows), 32 / G CTAs per SM (32 warps), pieces
// of KB blocks (100 KB of stages per SM for FP64 values and 32-bit columns with 8 or 16 lanes, which
// leaves L1 room for the X rows neighbouring slices share).  Four lanes take pieces of 8 blocks, but of 4
// for FP64 with five columns per lane or more, where 200 KB of stages left X no L1: stencil 90^3, k = 29,
// 770 -> 430 us.  Eight columns per lane spill 50 to 120 bytes at 64 registers: FP64 pairs read the X of
// one element at a time for 32-bit columns (k = 64, stencil 60^3 160 -> 150 us) and run 24 warps with 80
// registers for 16-bit ones (Laplacian 900^2 231 -> 214); so do single FP32 columns beside 32-bit ones
// (k = 63, Laplacian 900^2 267 -> 240), which beside 16-bit ones is slower (1.3 times).
constexpr int SPMM_UNROLL = 2;  // blocks of a piece unrolled together
// Neighbouring slices a CTA takes in a row: they share X rows, but long runs keep distant regions
// of X alive at once (stencil, k = 16: 249, 251, 254 and 304 us at 1, 2, 4 and 16; FP32C 214, 202,
// 200, 208).  One at a time where the matrix has few runs per resident CTA: fewer than 4 for FP32
// (stencil 80^3, k = 32: 202 us one at a time, 196 in runs), 16 for FP64 (169 and 175).
constexpr int RUN = 2;  // a power of two
template <typename VT, typename IT, int G, int KPL, int VW> struct SpmmShape {
    static_assert(G == 4 || G == 8 || G == 16, "lanes per row");
    static constexpr bool F64 = sizeof(VT) == 8, I32 = sizeof(IT) == 4, WIDE = KPL >= 7;
    static constexpr bool FEWER = WIDE && G <= 8 && (F64 ? VW == 2 && !I32 : VW == 1 && I32);
    static constexpr int THREADS = 32 * G, CTAS_PER_SM = (FEWER ? 24 : 32) / G;
    static constexpr int KB = G == 4 ? (F64 && KPL >= 5 ? 4 : 8) : G;
    // elements of a block whose X reads are in flight together, four where registers allow (pads: in
    // blocks with padding)
    static constexpr int together(bool pads) {
        return VW == 1 && KPL >= 3 ? 1 : F64 && I32 && WIDE ? 1 : KPL > 4 || pads ? 2 : 4;
    }
};
template <typename VT, typename IT, int G, int KPL, int VW> struct SpmmStage {
    static constexpr int VBYTES = SpmmShape<VT, IT, G, KPL, VW>::KB * 128 * (int)sizeof(VT);
    static constexpr int CBYTES = SpmmShape<VT, IT, G, KPL, VW>::KB * 128 * (int)sizeof(IT);
    static constexpr int BYTES = 2 * (VBYTES + CBYTES) + 128;  // two pieces + barriers
};

// What padding reads in place of a row of X: it adds 0 * 0, whatever X holds.  Aligned for the pair
// reads (ld_x2).
__device__ __align__(16) double g_zero_row[SELL_SPMM_MAX_K];

// Column of sum p of a lane whose column slot is lg (0 .. G-1).
template <int G, int VW>
__device__ __forceinline__ int spmm_col(int lg, int p) {
    return VW == 1 ? lg + G * p : 2 * (lg + G * (p >> 1)) + (p & 1);
}

// The four elements of row r in block i of a shared-memory piece: columns (I32) or 16-bit
// offsets widened to int (DELTA_NONE stays -32768), and values.
__device__ __forceinline__ void row_cols(const int *pc, int i, int r, int (&c)[4]) {
    const int4 a = reinterpret_cast<const int4 *>(pc)[i * 32 + r];
    c[0] = a.x; c[1] = a.y; c[2] = a.z; c[3] = a.w;
}
__device__ __forceinline__ void row_cols(const short *pc, int i, int r, int (&c)[4]) {
    const uint2 a = reinterpret_cast<const uint2 *>(pc)[i * 32 + r];
    c[0] = (int)(a.x << 16) >> 16; c[1] = (int)a.x >> 16;
    c[2] = (int)(a.y << 16) >> 16; c[3] = (int)a.y >> 16;
}

// LD: the type of X's leading dimension; int makes a row address one multiply-add.
template <typename VT, typename IT, int G, int KPL, int VW, typename LD>
__global__ void __launch_bounds__(SpmmShape<VT, IT, G, KPL, VW>::THREADS, SpmmShape<VT, IT, G, KPL, VW>::CTAS_PER_SM)
sell_spmm_kernel(const SellSlice *__restrict__ meta, const VT *__restrict__ vals,
                 const IT *__restrict__ cols, const VT *X, LD ldx,
                 double *__restrict__ Y, long long ldy, int ns, int run, int m, int n, int k,
                  unsigned long long *err, unsigned long long *wait_err) {
    using ST = SpmmStage<VT, IT, G, KPL, VW>;
    constexpr int KB = SpmmShape<VT, IT, G, KPL, VW>::KB;
    extern __shared__ __align__(128) unsigned char smem[];
    pdl_trigger();
    const int tid = threadIdx.x;
    const int r = tid / G;   // the thread's row within the slice
    const int lg = tid % G;  // its column slot
    const unsigned bar0 = (unsigned)__cvta_generic_to_shared(smem);  // two barriers
    const VT *sv = reinterpret_cast<const VT *>(smem + 128);
    const IT *sc = reinterpret_cast<const IT *>(smem + 128 + 2 * ST::VBYTES);
    const unsigned sv0 = bar0 + 128, sc0 = bar0 + 128 + 2 * ST::VBYTES;
    if (tid == 0) {
        mbar_init(bar0);
        mbar_init(bar0 + 8);
        mbar_init_fence();
    }
    __syncthreads();
    const uint64_t pl = policy_evict_last();

    // the CTA's slices: runs of `run` (a power of two), in turn over the grid
    const int first = (int)blockIdx.x * run, hop = ((int)gridDim.x - 1) * run + 1;
    auto next = [&](int s) { return s + (((s + 1) & (run - 1)) ? 1 : hop); };

    // Producer: thread 0 issues the copies of the slices' pieces.  Its cursor lives in shared memory,
    // so that it costs no registers: slice, next block, the slice's offset and blocks, and the
    // copies issued that the consumer has not waited for.
    int *cur = reinterpret_cast<int *>(smem + 16);
    auto p_find = [&](int ps) {
        SellSlice pm{0, 0, 0, 0u};
        for (; ps < ns; ps = next(ps)) {
            pm = meta[ps];
            if (pm.nblk > 0) break;
        }
        cur[0] = ps;
        cur[1] = 0;
        cur[2] = pm.off;
        cur[3] = pm.nblk;
    };
    auto issue = [&](int kk) {  // thread 0 alone
        const int ps = cur[0], pb = cur[1], off = cur[2], nblk = cur[3];
        if (ps >= ns) return;
        const int len = min(KB, nblk - pb);
        const long long e0 = (long long)off + (long long)pb * 128;
        const unsigned vb = (unsigned)(len * 128 * (int)sizeof(VT));
        const unsigned cb = (unsigned)(len * 128 * (int)sizeof(IT));
        proxy_fence();  // the stage's last reads come before the copy's writes
        mbar_expect_tx(bar0 + 8 * kk, vb + cb);
        bulk_g2s(sv0 + kk * ST::VBYTES, vals + e0, vb, bar0 + 8 * kk);
        bulk_g2s(sc0 + kk * ST::CBYTES, cols + e0, cb, bar0 + 8 * kk);
        cur[4] += 1;
        if (pb + KB < nblk) cur[1] = pb + KB;
        else p_find(next(ps));
    };
    if (tid == 0) {
        cur[4] = 0;
        p_find(first);
        issue(0);
        issue(1);
    }
    pdl_wait();  // X, and Y, which the product before may still use: only copies of the format above

    // consumer cursor; the rows of empty slices are written as zeros
    int cs = first, cb = 0;
    int nblk = 0, base = 0, pads = 0;  // of slice cs: blocks, base column, first block with padding
    auto store_row = [&](int slice, const double (&acc)[KPL]) {
        const long long row = (long long)slice * 32 + r;
        if (row >= m) return;
        double *yr = Y + row * ldy;
#pragma unroll
        for (int p = 0; p < KPL; p += VW) {
            const int c = spmm_col<G, VW>(lg, p);
            if (c >= k) continue;
            if constexpr (VW == 2)
                *reinterpret_cast<double2 *>(yr + c) = make_double2(acc[p], acc[p + 1]);
            else
                yr[c] = acc[p];
        }
    };
    auto c_find = [&]() {
        double zero[KPL];
#pragma unroll
        for (int p = 0; p < KPL; ++p) zero[p] = 0.0;
        for (; cs < ns; cs = next(cs)) {
            const SellSlice cm = meta[cs];
            nblk = cm.nblk;
            base = sizeof(IT) == 2 ? cm.colbase : 0;
            pads = (cm.flags & 1u) ? (int)(cm.flags >> 1) : nblk;
            if (nblk > 0) break;
            store_row(cs, zero);
        }
    };
    c_find();
    unsigned phases = 0;  // bit kk: the parity awaited on stage kk
    int kk = 0;
    double acc[KPL];
#pragma unroll
    for (int p = 0; p < KPL; ++p) acc[p] = 0.0;
    // Column offsets of the lane's reads.  Only the last slot can lie past k: a pair of it reads the
    // last columns, whose line other lanes read anyway; a single column of it is not read.
    int xoff[KPL / VW];
#pragma unroll
    for (int p = 0; p < KPL; p += VW) {
        const int c = spmm_col<G, VW>(lg, p);
        xoff[p / VW] = c < k ? c : k - VW;
    }
    const bool last = VW == 2 || spmm_col<G, VW>(lg, KPL - VW) < k;
    auto sum_block = [&](const VT *pv, const IT *pc, int i, auto pads_tag) {
        constexpr bool PADS = decltype(pads_tag)::value;
        constexpr int QB = SpmmShape<VT, IT, G, KPL, VW>::together(PADS);
        int c[4];
        row_cols(pc, i, r, c);
        const VBlk<VT> vv = VBlk<VT>::load_smem(pv, i, r);
#pragma unroll
        for (int q0 = 0; q0 < 4; q0 += QB) {
            VT xv[QB][KPL];
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                const int cq = c[q0 + q];
                const bool real = !PADS || (sizeof(IT) == 2 ? cq != DELTA_NONE : cq >= 0);
                const bool use = real && guard(err, cq + base >= 0 && cq + base < n, G_X, cq + base);
                const VT *xr = use ? X + (long long)(cq + base) * ldx
                                   : reinterpret_cast<const VT *>(g_zero_row);
#pragma unroll
                for (int p = 0; p < KPL; p += VW) {
                    if constexpr (VW == 2) {
                        const auto x2 = ld_x2(xr + xoff[p / 2], pl);
                        xv[q][p] = x2.x;
                        xv[q][p + 1] = x2.y;
                    } else {
                        xv[q][p] = p < KPL - 1 || last ? ld_x(xr + xoff[p], pl) : VT(0);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                const double v = (double)vv.get(q0 + q);
#pragma unroll
                for (int p = 0; p < KPL; ++p) acc[p] = fma(v, (double)xv[q][p], acc[p]);
            }
        }
    };
    while (cs < ns) {
        const bool ok = mbar_wait(bar0 + 8 * kk, (phases >> kk) & 1u);
        phases ^= 1u << kk;
        const int len = ok ? min(KB, nblk - cb) : 0;
        const VT *pv = sv + kk * (ST::VBYTES / (int)sizeof(VT));
        const IT *pc = sc + kk * (ST::CBYTES / (int)sizeof(IT));
        const int clean = max(0, min(len, pads - cb));  // blocks before the padding
#pragma unroll SPMM_UNROLL
        for (int i = 0; i < clean; ++i) sum_block(pv, pc, i, std::false_type());
#pragma unroll SPMM_UNROLL
        for (int i = clean; i < len; ++i) sum_block(pv, pc, i, std::true_type());
        const int done = cs;
        cb += KB;
        if (cb >= nblk) {  // the slice's last piece
            if (ok) store_row(cs, acc);  // after a wait that gave up the sums are partial
#pragma unroll
            for (int p = 0; p < KPL; ++p) acc[p] = 0.0;
            cb = 0;
            cs = next(cs);
            c_find();
        }
        // every thread is done with stage kk; the CTA gives up together if any wait did
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicAdd(&wait_err[0], 1ull);
                atomicCAS(&wait_err[1], 0ull, (unsigned long long)done + 1);
                // the copies still in flight land before the CTA exits: this piece's, the next's
                mbar_wait(bar0 + 8 * kk, ((phases >> kk) & 1u) ^ 1u);
                if (cur[4] > 1) mbar_wait(bar0 + 8 * (kk ^ 1), (phases >> (kk ^ 1)) & 1u);
            }
            break;
        }
        if (tid == 0) {
            cur[4] -= 1;
            issue(kk);
        }
        kk ^= 1;
    }
}

template <typename VT, typename IT, int G, int KPL, int VW, typename LD = int>
cudaError_t spmm_launch(const Handle &h, const VT *X, long long ldx, double *Y, long long ldy,
                        int k, cudaStream_t s) {
    using ST = SpmmStage<VT, IT, G, KPL, VW>;
    constexpr auto kernel = sell_spmm_kernel<VT, IT, G, KPL, VW, LD>;
    // more than the default 48 KB of dynamic shared memory: opted into once per device
    static std::atomic<unsigned long long> opted{0};
    if (h.device < 0 || h.device >= 64) return cudaErrorInvalidDevice;
    const unsigned long long bit = 1ull << h.device;
    if (!(opted.load() & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(
            kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ST::BYTES);
        if (e != cudaSuccess) return e;
        opted.fetch_or(bit);
    }
    const long long cap = (long long)h.sm_count * SpmmShape<VT, IT, G, KPL, VW>::CTAS_PER_SM;
    const int run = h.nchunks >= (sizeof(VT) == 8 ? 16 : 4) * RUN * cap ? RUN : 1;
    const long long runs = (h.nchunks + run - 1) / run;
    const unsigned grid = (unsigned)(runs < cap ? runs : cap);
    return launch_product(kernel, grid, SpmmShape<VT, IT, G, KPL, VW>::THREADS, ST::BYTES, s,
                          (const SellSlice *)h.meta, (const VT *)h.vals, (const IT *)h.cols, X,
                          (LD)ldx, Y, ldy, (int)h.nchunks, run, h.m, h.n, k, guard_word(), wait_word());
}

// KPL = ceil(k / G), so that a lane reads no slot that no lane needs (k = 21 on eight lanes: three,
// not four); pairs per read where they can be, with KPL rounded up to even.  Single columns are read
// element by element (QB = 1): two or four elements at once spill.  In a loop, us, KPL a power of two
// with four elements in flight / this: k = 21, stencil 60^3 107 / 81 (FP32 91 / 71), dense blocks
// 200,000 rows 185 / 126 (176 / 123); k = 13 dense blocks 106 / 83.
template <typename VT, typename IT, int G, int KPL>
cudaError_t spmm_vw(const Handle &h, const VT *X, long long ldx, double *Y, long long ldy,
                    int k, cudaStream_t s) {
    if (ldx > INT_MAX)  // 64-bit row offsets: one kernel for every k
        return spmm_launch<VT, IT, 8, 8, 1, long long>(h, X, ldx, Y, ldy, k, s);
    const bool vec2 = KPL >= 2 && k % 2 == 0 && ldx % 2 == 0 && ldy % 2 == 0 &&
                      reinterpret_cast<uintptr_t>(X) % (2 * sizeof(VT)) == 0 &&
                      reinterpret_cast<uintptr_t>(Y) % 16 == 0;
    if constexpr (KPL >= 2)
        if (vec2) return spmm_launch<VT, IT, G, KPL + KPL % 2, 2>(h, X, ldx, Y, ldy, k, s);
    return spmm_launch<VT, IT, G, KPL, 1>(h, X, ldx, Y, ldy, k, s);
}

template <typename VT, typename IT, int G>
cudaError_t spmm_g(const Handle &h, const VT *X, long long ldx, double *Y, long long ldy, int k,
                   cudaStream_t s) {
    switch ((k + G - 1) / G) {
        case 1: return spmm_vw<VT, IT, G, 1>(h, X, ldx, Y, ldy, k, s);
        case 2: return spmm_vw<VT, IT, G, 2>(h, X, ldx, Y, ldy, k, s);
        case 3: return spmm_vw<VT, IT, G, 3>(h, X, ldx, Y, ldy, k, s);
        case 4: return spmm_vw<VT, IT, G, 4>(h, X, ldx, Y, ldy, k, s);
    }
    if constexpr (G <= 8) {
        switch ((k + G - 1) / G) {
            case 5: return spmm_vw<VT, IT, G, 5>(h, X, ldx, Y, ldy, k, s);
            case 6: return spmm_vw<VT, IT, G, 6>(h, X, ldx, Y, ldy, k, s);
            case 7: return spmm_vw<VT, IT, G, 7>(h, X, ldx, Y, ldy, k, s);
            case 8: return spmm_vw<VT, IT, G, 8>(h, X, ldx, Y, ldy, k, s);
        }
    }
    return cudaErrorInvalidValue;
}

template <typename VT, typename IT>
cudaError_t spmm_k(const Handle &h, const VT *X, long long ldx, double *Y, long long ldy, int k,
                   cudaStream_t s) {
    // 16 elements per row and more; very long rows are "short" again for even k
    const bool long_rows = (long long)h.nnz >= 16LL * h.m && (k % 2 || (long long)h.nnz <= 32LL * h.m);
    switch (sell_spmm_lanes(h.lanes_per_row, k, sizeof(VT) == 4, long_rows)) {
        case 4: return spmm_g<VT, IT, 4>(h, X, ldx, Y, ldy, k, s);
        case 8: return spmm_g<VT, IT, 8>(h, X, ldx, Y, ldy, k, s);
        case 16: return spmm_g<VT, IT, 16>(h, X, ldx, Y, ldy, k, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t sell_spmm(const Handle &h, const void *X, long long ldx, void *Y, long long ldy,
                      int k, cudaStream_t s) {
    if (h.nchunks <= 0 || k <= 0) return cudaSuccess;
    if (k > SELL_SPMM_MAX_K) return cudaErrorInvalidValue;
    const bool f32 = h.precision == PAVA_PREC_FP32C, d16 = h.index_mode == PAVA_INDEX_DELTA16;
    double *y = (double *)Y;
    if (!f32 && !d16) return spmm_k<double, int>(h, (const double *)X, ldx, y, ldy, k, s);
    if (!f32 && d16) return spmm_k<double, short>(h, (const double *)X, ldx, y, ldy, k, s);
    if (f32 && !d16) return spmm_k<float, int>(h, (const float *)X, ldx, y, ldy, k, s);
    return spmm_k<float, short>(h, (const float *)X, ldx, y, ldy, k, s);
}

}  // namespace pava
