// SpMM on plain CSR for k right-hand sides (Y = A X, X row-major n x k): the kernel of handles whose
// shape is left to the engine (but for small matrices and very uneven rows, pava_spmm), and of the row-group shapes that give each of a row's lanes its own
// columns (csr_staged_shape); k_group.cu runs the other shapes that options name.
//
// A warp takes 32 / G rows at a time, G lanes per row; lane g of a row's G owns the KPL columns of
// slot g (VW = 2: the pairs g, g + G, ... of adjacent columns, each read as one vector), so the G
// lanes of a row read a whole row of X per nonzero and keep its sums in registers.  The rows'
// elements pass through a small stage of the warp's own in shared memory, PS per row at a time:
// half-warps read PS consecutive elements of a row (whole lines), and the G lanes of a row read
// its elements back four at a time, one broadcast 16-byte read per four columns and two values.
// The next PS elements are loaded while these are summed.  No barrier beyond the warp's.
//
// What bounds it: the X reads through L1.  The row groups (k_group.cu) pass each element to the
// lanes of its row by three shuffles and read the rows' elements GL at a time, one line per row and
// load: together about as many L1 cycles as the X reads of k = 8.  FP64 / FP32 storage, L2 flushed, us,
// the shape the engine chose before / the best row-group shape / this kernel: banded (1,048,576
// rows, 24 each) k = 8 254 / 188 / 154 and 340 / 217 / 140, k = 16 621 / 295 / 267 and 693 / 383 /
// 211, k = 32 1,234 / 506 / 366 and 1,420 / 734 / 365; stencil 100^3 k = 8 312 / 209 / 168, k = 32
// 1,237 / 582 / 410; dense blocks (400,000 rows) k = 8 189 / 148 / 117, k = 32 814 / 371 / 251.  In a
// loop, FP64 / FP32, the shape before / this kernel: banded 300,007 rows k = 33 499 / 248 and 680 / 241,
// k = 64 396 / 242 and 490 / 193, k = 127 953 / 549 and 1,638 / 463, k = 128 591 / 435 and 993 / 328 (the
// 8-column forms for odd k spill 150 to 200 bytes; they are still the faster ones).
// Without the next round's elements in flight k = 8 took 161, 174 and 118 us; with three CTAs per
// SM 164, 182 and 117.
//
// The persistent grid and the tiles of 4 (32 / G) rows per warp are those of k_group.cu.  The
// reference multiplies one vector at a time (main.cpp:554-587).

#include <climits>
#include <cstdint>
#include <type_traits>

#include "k_stream.cuh"
#include "pava_internal.h"

namespace pava {

namespace {

constexpr int WARPS = 8, PS = 16, MAX_K = 128;
constexpr int LDC = PS + 4;                                            // ints per row of the stage
template <typename VT> constexpr int LDV = sizeof(VT) == 8 ? PS + 2 : PS + 4;  // values per row

// What elements past a row's end read in place of a row of X: they add 0 * 0.  Aligned for the pair
// reads (ld_x2), which fault on an address that is no multiple of 16.
__device__ __align__(16) double g_zeros[MAX_K];

template <int G, int VW>
__device__ __forceinline__ int slot_col(int lg, int p) {
    return VW == 1 ? lg + G * p : 2 * (lg + G * (p >> 1)) + (p & 1);
}

template <typename VT> __device__ __forceinline__ void row_vals(const VT *p, VT (&v)[4]);
template <> __device__ __forceinline__ void row_vals(const double *p, double (&v)[4]) {
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <> __device__ __forceinline__ void row_vals(const float *p, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4 *>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}

// LD: the type of X's leading dimension; int (VW = 2) makes a row address one multiply-add.
template <typename VT, int G, int KPL, int VW, typename LD>
__global__ void __launch_bounds__(WARPS * 32, 4)
csr_spmm_kernel(const int *__restrict__ rp, const int *__restrict__ ci, const VT *__restrict__ v,
                const VT *X, LD ldx, double *__restrict__ Y, long long ldy, int m,
                int n, int k, unsigned long long *err) {
    constexpr int R = 32 / G;               // rows at a time
    constexpr int NU = R * PS / 32;         // elements a lane stages per piece
    __shared__ __align__(16) VT s_val[WARPS][R * LDV<VT>];
    __shared__ __align__(16) int s_col[WARPS][R * LDC];
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int row = lane / G, lg = lane % G;    // this lane's row of the R and its column slot
    const int half = lane >> 4, li = lane & 15; // staging: row 2 u + half, element li of the piece
    const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
    int xoff[KPL / VW];  // column offsets of the lane's reads; a slot past k reads column 0
#pragma unroll
    for (int p = 0; p < KPL; p += VW) {
        const int c = slot_col<G, VW>(lg, p);
        xoff[p / VW] = c < k ? c : 0;
    }
    const VT *pv = &s_val[w][row * LDV<VT>];
    const int *pc = &s_col[w][row * LDC];

    double acc[KPL];
    auto sum4 = [&](int i, auto pads_tag) {  // elements i .. i + 3 of the stage
        constexpr bool PADS = decltype(pads_tag)::value;
        // elements whose X reads are in flight together
        constexpr int QB = KPL >= 8 ? 2 : 4;
        const int4 c4 = *reinterpret_cast<const int4 *>(pc + i);
        const int c[4] = {c4.x, c4.y, c4.z, c4.w};
        VT val[4];
        row_vals(pv + i, val);
#pragma unroll
        for (int q0 = 0; q0 < 4; q0 += QB) {
            VT xv[QB][KPL];
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                const int col = c[q0 + q];
                const bool use = (!PADS || col >= 0) && guard(err, col >= 0 && col < n, G_X, col);
                const VT *xr = use ? X + (long long)col * ldx : reinterpret_cast<const VT *>(g_zeros);
#pragma unroll
                for (int p = 0; p < KPL; p += VW) {
                    if constexpr (VW == 2) {
                        const auto x2 = ld_x2(xr + xoff[p / 2], pl);
                        xv[q][p] = x2.x;
                        xv[q][p + 1] = x2.y;
                    } else {
                        xv[q][p] = ld_x(xr + xoff[p], pl);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < QB; ++q)
#pragma unroll
                for (int p = 0; p < KPL; ++p)  // FP32 products are exact in FP64
                    acc[p] = fma((double)val[q0 + q], (double)xv[q][p], acc[p]);
        }
    };

    // Rounds of R rows, four to a tile; while one is summed, the row pointers of the next and then
    // its first elements are loaded.
    const unsigned um = (unsigned)m, ntiles = (um + 4 * R - 1) / (4 * R);
    const unsigned hop = (gridDim.x * WARPS - 1) * (4 * R);  // from a tile's end to the warp's next
    unsigned r = (blockIdx.x * WARPS + w) * (4 * R) + row, i4 = 0;
    auto bounds = [&](unsigned rr, int &a, int &len) {
        a = len = 0;
        if (rr < um) {
            a = rp[rr];
            len = rp[rr + 1] - a;
        }
    };
    VT val[NU];
    int col[NU];
    auto load = [&](int a, int len, int i0) {  // elements i0 .. i0 + PS - 1 of the R rows
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            const int src = (2 * u + half) * G;
            const int ru = __shfl_sync(FULL, a, src), lu = __shfl_sync(FULL, len, src);
            const bool in = lu - i0 > li;
            val[u] = in ? ld_val(v + ru + (i0 + li), pf) : VT(0);
            col[u] = in ? ld_col(ci + ru + (i0 + li), pf) : -1;
        }
    };
    if (blockIdx.x * WARPS + w >= ntiles) return;  // warp-uniform
    int a, len;
    bounds(r, a, len);
    load(a, len, 0);
    for (;;) {
        // the next round: in this tile, or the first of the warp's next tile
        const bool tile_end = i4 == 3;
        const unsigned rn = r + R + (tile_end ? hop : 0u);
        const bool more = rn - row < um && rn >= r;  // a round with rows; no wrap past 2^32
        int an = 0, ln = 0;
        if (more) bounds(rn, an, ln);
        int longest = len, shortest = len;
#pragma unroll
        for (int o = 16; o >= G; o >>= 1) {
            longest = max(longest, __shfl_xor_sync(FULL, longest, o));
            shortest = min(shortest, __shfl_xor_sync(FULL, shortest, o));
        }
#pragma unroll
        for (int p = 0; p < KPL; ++p) acc[p] = 0.0;
        for (int i0 = 0;;) {
            const int left = longest - i0;
            __syncwarp();  // the last piece's reads are done
#pragma unroll
            for (int u = 0; u < NU; ++u) {
                s_val[w][(2 * u + half) * LDV<VT> + li] = val[u];
                s_col[w][(2 * u + half) * LDC + li] = col[u];
            }
            __syncwarp();
            if (left > PS) load(a, len, i0 + PS);
            else load(an, ln, 0);
            if (shortest - i0 >= PS) {
#pragma unroll
                for (int i = 0; i < PS; i += 4) sum4(i, std::false_type());
            } else {
                const int e = left < PS ? left : PS, clean = shortest - i0;
                int i = 0;
#pragma unroll 1
                for (; i + 4 <= clean; i += 4) sum4(i, std::false_type());
#pragma unroll 1
                for (; i < e; i += 4) sum4(i, std::true_type());
            }
            if (left <= PS) break;  // no i0 past the longest row: it cannot overflow
            i0 += PS;
        }
        if (r < um) {
            double *yr = Y + (long long)r * ldy;
#pragma unroll
            for (int p = 0; p < KPL; p += VW) {
                const int c = slot_col<G, VW>(lg, p);
                if (c >= k) continue;
                if constexpr (VW == 2)
                    *reinterpret_cast<double2 *>(yr + c) = make_double2(acc[p], acc[p + 1]);
                else
                    yr[c] = acc[p];
            }
        }
        if (!more) break;
        r = rn;
        a = an;
        len = ln;
        i4 = tile_end ? 0 : i4 + 1;
    }
}

template <typename VT, int G, int KPL>
cudaError_t launch(const Handle &h, const VT *X, long long ldx, double *Y, long long ldy, int k,
                   cudaStream_t s) {
    constexpr int R = 32 / G;
    const long long ntiles = ((long long)h.m + 4 * R - 1) / (4 * R);
    const long long want = (ntiles + WARPS - 1) / WARPS, cap = (long long)h.sm_count * 4;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    // pairs per read and store where every pair is whole and aligned
    const bool vec2 = KPL >= 2 && k % 2 == 0 && ldx % 2 == 0 && ldy % 2 == 0 && ldx <= INT_MAX &&
                      reinterpret_cast<uintptr_t>(X) % (2 * sizeof(VT)) == 0 &&
                      reinterpret_cast<uintptr_t>(Y) % 16 == 0;
    if constexpr (KPL >= 2)
        if (vec2)
            return launch_product(csr_spmm_kernel<VT, G, KPL, 2, int>, grid, WARPS * 32, 0, s, h.rp,
                                  h.ci, (const VT *)h.v, X, (int)ldx, Y, ldy, h.m, h.n, k,
                                  guard_word());
    return launch_product(csr_spmm_kernel<VT, G, KPL, 1, long long>, grid, WARPS * 32, 0, s, h.rp,
                          h.ci, (const VT *)h.v, X, ldx, Y, ldy, h.m, h.n, k, guard_word());
}

// Lanes per row and columns per lane for k: four lanes up to 16 columns, so that eight rows' X reads
// are in flight per warp, eight up to 64, sixteen above.
template <typename VT>
cudaError_t launch_k(const Handle &h, const VT *X, long long ldx, double *Y, long long ldy, int k,
                     cudaStream_t s) {
    if (k <= 4) return launch<VT, 4, 1>(h, X, ldx, Y, ldy, k, s);
    if (k <= 8) return launch<VT, 4, 2>(h, X, ldx, Y, ldy, k, s);
    if (k <= 16) return launch<VT, 4, 4>(h, X, ldx, Y, ldy, k, s);
    if (k <= 32) return launch<VT, 8, 4>(h, X, ldx, Y, ldy, k, s);
    if (k <= 64) return launch<VT, 8, 8>(h, X, ldx, Y, ldy, k, s);
    if (k <= MAX_K) return launch<VT, 16, 8>(h, X, ldx, Y, ldy, k, s);
    return cudaErrorInvalidValue;
}

}  // namespace

// Row-group shapes this kernel serves, with the same sums in the same order: as many lanes across k
// as per row (4 or 8), a tile of four rounds.
bool csr_staged_shape(const Handle &g, int k) {
    const bool shape = g.lanes_per_row == 4 || (g.lanes_per_row == 8 && g.cols_per_lane == 4);
    return k > 1 && shape && !g.x_window && g.col_lanes == g.lanes_per_row &&
           g.rows_per_tile == 4 * (32 / g.lanes_per_row);
}

cudaError_t csr_spmm_staged(const Handle &h, const void *X, long long ldx, void *Y, long long ldy,
                            int k, int lanes, int cols, cudaStream_t s) {
    if (h.m <= 0 || k <= 0) return cudaSuccess;
    auto go = [&](auto tag) {
        using VT = decltype(tag);
        const VT *x = (const VT *)X;
        double *y = (double *)Y;
        if (lanes == 0) return launch_k<VT>(h, x, ldx, y, ldy, k, s);
        if (lanes == 4 && cols == 1) return launch<VT, 4, 1>(h, x, ldx, y, ldy, k, s);
        if (lanes == 4 && cols == 2) return launch<VT, 4, 2>(h, x, ldx, y, ldy, k, s);
        if (lanes == 4 && cols == 4) return launch<VT, 4, 4>(h, x, ldx, y, ldy, k, s);
        if (lanes == 8 && cols == 4) return launch<VT, 8, 4>(h, x, ldx, y, ldy, k, s);
        return cudaErrorInvalidValue;
    };
    return h.precision == PAVA_PREC_FP32C ? go(float()) : go(double());
}

}  // namespace pava
