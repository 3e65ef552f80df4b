// CSR row-group kernel: SpMV and multi-RHS SpMM (Y = A X, X row-major n x k) on plain CSR,
// FP64 or FP32 storage (one right-hand side: compensated FP32 sums), for short-row and batched
// matrices.  SpMM without a shape of its own runs k_csr_spmm.cu instead.
//
// A group of GL lanes (a power of two <= 32) owns one row at a time.  Inside the group, KC
// lanes span the k right-hand sides (lane c holds columns c, c + KC, ..., KPL of them) and
// ES = GL / KC element slices split the row's nonzeros (slice e takes elements e, e + ES, ...).
// For k = 32, GL = KC = 32 it is one warp per row reading 256-byte rows of X.  One right-hand
// side has a kernel of its own (csr_spmv_kernel).  A slice's partial sums are combined over the
// ES slices with a fixed xor butterfly, so every call gives the same bits.
//
// The launch is persistent: the grid is sized to the resident capacity of the GPU and warps
// take tiles of TR consecutive rows in grid-stride order (tile t to warp t mod warps), which
// keeps one launch per SpMV/SpMM whatever the number of rows -- the batched path (a
// block-diagonal union of many small matrices) relies on this.

#include <climits>
#include <cstdint>
#include <type_traits>

#include "k_stream.cuh"
#include "pava_internal.h"

namespace pava {

namespace {

// A row's sum for one right-hand side.  FP32 values and x: a product of two FP32 numbers is exact in
// FP64, so the exact products are summed there -- one conversion and one FMA per right-hand side,
// where a compensated FP32 sum takes ten operations, and more accurate.
struct ColAcc {
    double s = 0.0;
    __device__ __forceinline__ void add(double v, double x) { s = fma(v, x, s); }
    __device__ __forceinline__ double value() const { return s; }
};

// Rows shared by several column lanes (KCT = KC > 1, a compile-time count so that the KC
// elements of a round unroll): the group loads its row's nonzeros
// cooperatively, GL at a time (lane gi loads element base + gi, one coalesced load per lane and
// stream), with the next round's loads in flight while the current round is consumed; each
// element reaches the lanes that need it by shuffle.  Slice e takes elements e, e + ES, ... in
// ascending order, as the per-lane loop does, so the sums have the same bits.  The round count
// is the maximum over the warp's groups so that every shuffle has all 32 lanes.  With eight steps or more
// a round takes as many as the longest row still needs, rounded up to a half, a quarter or an eighth:
// rows of five in groups of 32 spent nearly all of it on nothing (Laplacian 700^2, k = 33, 32 lanes of
// which 16 across k: 816 us with all steps for every row, now 324).  With fewer steps the choice
// cost more than it saved (power law 200,003 rows, k = 2, two lanes: 555 -> 930 us), as did an end
// test between the steps, which kept the X reads of the next ones back (banded 300,007 rows, k = 8 on
// groups of four: 67 -> 96).  The X reads of UB elements are in flight together: an element past the
// row's end has column -1, for which xload gives zeros.
template <int KPL, int KCT, typename VT, typename XLOAD>
__device__ __forceinline__ void coop_row(int a, int b, int gi, int gl, int es, int e, int lane,
                                         const int *__restrict__ ci, const VT *__restrict__ v,
                                         XLOAD xload, ColAcc (&acc)[KPL], uint64_t pf) {
    constexpr int UB = KPL >= 4 ? 1 : (KCT < 4 / KPL ? KCT : 4 / KPL);
    const int most = __reduce_max_sync(FULL, b - a);  // elements of the warp's longest row
    const int rounds = (int)(((unsigned)most + gl - 1) / gl);
    const int gbase = lane & ~(gl - 1);
    VT pv = VT(0);
    int pc = -1;
    if (a + gi < b) {
        pv = ld_val(v + a + gi, pf);
        pc = ld_col(ci + a + gi, pf);
    }
    for (int rd = 0; rd < rounds; ++rd) {
        const VT cv = pv;
        const int cc = pc;
        const int base = a + rd * gl;
        pv = VT(0);
        pc = -1;
        if (base + gl + gi < b) {  // next round in flight
            pv = ld_val(v + base + gl + gi, pf);
            pc = ld_col(ci + base + gl + gi, pf);
        }
        auto steps = [&](auto count) {
            constexpr int N = decltype(count)::value, B = UB < N ? UB : N;
#pragma unroll
            for (int u0 = 0; u0 < N; u0 += B) {
                VT val[B], xv[B][KPL];
#pragma unroll
                for (int u = 0; u < B; ++u) {
                    const int o = gbase + e + (u0 + u) * es;
                    val[u] = __shfl_sync(FULL, cv, o);
                    xload(__shfl_sync(FULL, cc, o), xv[u]);
                }
#pragma unroll
                for (int u = 0; u < B; ++u)
#pragma unroll
                    for (int p = 0; p < KPL; ++p) acc[p].add((double)val[u], (double)xv[u][p]);
            }
        };
        if constexpr (KCT >= 8) {
            const int left = most - rd * gl;
            if (left > es * (KCT / 2)) steps(std::integral_constant<int, KCT>());
            else if (left > es * (KCT / 4)) steps(std::integral_constant<int, KCT / 2>());
            else if (left > es * (KCT / 8)) steps(std::integral_constant<int, KCT / 4>());
            else steps(std::integral_constant<int, KCT / 8>());
        } else {
            steps(std::integral_constant<int, KCT>());
        }
    }
}

// Column of accumulator p of a lane whose first column slot is cl: VW = 1 interleaves single
// columns across the KC lanes (cl + p KC); VW = 2 interleaves pairs (2 (cl + (p/2) KC) + p%2),
// so that a lane reads its two columns with one vector load and a group's KC lanes read
// 16 KC contiguous bytes.
template <int VW>
__device__ __forceinline__ int col_of(int cl, int p, int kc) {
    return VW == 1 ? cl + p * kc : 2 * (cl + (p >> 1) * kc) + (p & 1);
}

constexpr int GROUP_THREADS = 256;
// resident blocks per SM: more warps in flight for the narrow shapes
template <int KPL> constexpr int group_minb() { return KPL == 1 ? 6 : (KPL == 2 ? 5 : 4); }
// resident blocks per SM of the cooperative (k > 1) shapes
constexpr int COOP_MINB = 4;
// elements in flight per lane
template <int KPL> constexpr int group_unroll() { return KPL == 1 ? 4 : (KPL == 2 ? 2 : 1); }

template <int KPL, typename VT, int KCT, int VW>
__global__ void __launch_bounds__(GROUP_THREADS, KCT ? COOP_MINB : group_minb<KPL>())
csr_group_kernel(const int *__restrict__ rp, const int *__restrict__ ci,
                 const VT *__restrict__ v, const VT *X, long long ldx,
                 double *__restrict__ Y, long long ldy, int m, int k, int gl_shift,
                 int kc_shift, int tile_rows, unsigned by_cta, unsigned by_warp, int n,
                 unsigned long long *err) {
    constexpr int U = group_unroll<KPL>();
    pdl_wait();
    pdl_trigger();  // after the wait: one product ahead at most, see deal_tiles
    const int lane = threadIdx.x & 31;
    const int gl = 1 << gl_shift, kc = 1 << kc_shift;
    const int grp = lane >> gl_shift;          // group within the warp
    const int gpw = 32 >> gl_shift;            // groups (rows in flight) per warp
    const int gi = lane & (gl - 1);
    const int e = gi >> kc_shift;              // element slice
    const int es = gl >> kc_shift;             // slices per row
    const int cl = gi & (kc - 1);              // first column of this lane
    const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
    const long long ntiles = ((long long)m + tile_rows - 1) / tile_rows;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const int rounds = tile_rows / gpw;        // rows per group per tile

    // column offsets of the lane's reads; a slot past k reads nothing
    int xoff[KPL];
#pragma unroll
    for (int p = 0; p < KPL; ++p) {
        const int c = col_of<VW>(cl, p, kc);
        xoff[p] = c < k ? c : -1;
    }
    // the lane's KPL columns of X row `col` (zeros for column -1)
    auto xload = [&](int col, VT(&xv)[KPL]) {
        const bool in = col >= 0 && guard(err, col < n, G_X, col);
        const VT *xr = X + (long long)col * ldx;
#pragma unroll
        for (int p = 0; p < KPL; p += VW) {
            xv[p] = VT(0);
            if constexpr (VW == 2) xv[p + 1] = VT(0);
            if (!in || xoff[p] < 0) continue;
            if constexpr (VW == 2) {
                const auto x2 = ld_x2(xr + xoff[p], pl);
                xv[p] = x2.x;
                xv[p + 1] = x2.y;
            } else {
                xv[p] = ld_x(xr + xoff[p], pl);
            }
        }
    };

    for (long long t = (long long)blockIdx.x * by_cta + (threadIdx.x >> 5) * by_warp; t < ntiles;
         t += nwarps) {
        for (int i = 0; i < rounds; ++i) {
            const long long r = t * tile_rows + (long long)i * gpw + grp;
            const bool valid = r < m;
            int a = 0, b = 0;
            if (valid) {
                a = rp[r];
                b = rp[r + 1];
            }
            ColAcc acc[KPL];
            if constexpr (KCT != 0) {
                coop_row<KPL, KCT>(a, b, gi, gl, es, e, lane, ci, v, xload, acc, pf);
            } else {
                // U elements at a time: all value and column loads first, then all gathers, so up to U
                // memory round trips overlap even on short rows
                const unsigned len = (unsigned)(b - a);
                for (unsigned j = e; j < len; j += U * es) {
                    VT val[U], xv[U][KPL];
                    int col[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const bool in = j + u * es < len;
                        val[u] = in ? ld_val(v + a + (j + u * es), pf) : VT(0);
                        col[u] = in ? ld_col(ci + a + (j + u * es), pf) : -1;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) xload(col[u], xv[u]);
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int p = 0; p < KPL; ++p) acc[p].add((double)val[u], (double)xv[u][p]);
                }
            }
#pragma unroll
            for (int p = 0; p < KPL; ++p) {
                double s = acc[p].value();
                for (int o = kc; o < gl; o <<= 1) s += __shfl_xor_sync(FULL, s, o);
                if (valid && e == 0 && col_of<VW>(cl, p, kc) < k)
                    Y[r * ldy + col_of<VW>(cl, p, kc)] = s;
            }
        }
    }
}

// Windowed variant for k > 1 on matrices whose rows reach a narrow column range (banded,
// stencil-like): a CTA owns a tile of TR consecutive rows, finds the tile's column window
// [cmin, cmax], copies X[cmin .. cmax][0 .. k) into shared memory once, and its row groups
// read X from there.  Each X row is then fetched from L2 once per tile instead of once per
// nonzero that references it.  Tiles whose window does not fit take the global gathers.
constexpr int WINDOW_MINB = 2;
constexpr int WINDOW_SMEM = 100 * 1024;  // bytes of X per CTA (two CTAs per SM)

template <int KPL, typename VT, int KCT>
__global__ void __launch_bounds__(GROUP_THREADS, WINDOW_MINB)
csr_window_kernel(const int *__restrict__ rp, const int *__restrict__ ci,
                  const VT *__restrict__ v, const VT *X, long long ldx,
                  double *__restrict__ Y, long long ldy, int m, int k, int gl_shift,
                  int kc_shift, int tile_rows, int max_w, int n, unsigned long long *err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    VT *xs = reinterpret_cast<VT *>(smem_raw);
    constexpr int WARPS = GROUP_THREADS / 32;
    __shared__ int s_min[WARPS], s_max[WARPS];
    pdl_wait();
    pdl_trigger();  // after the wait: one product ahead at most, see deal_tiles
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int gl = 1 << gl_shift, kc = 1 << kc_shift;
    const int grp = lane >> gl_shift;
    const int gpw = 32 >> gl_shift;
    const int gi = lane & (gl - 1);
    const int e = gi >> kc_shift;
    const int es = gl >> kc_shift;
    const int cl = gi & (kc - 1);
    const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
    const long long ntiles = ((long long)m + tile_rows - 1) / tile_rows;
    const int rows_per_pass = WARPS * gpw;

    bool colok[KPL];
#pragma unroll
    for (int p = 0; p < KPL; ++p) colok[p] = cl + p * kc < k;

    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const long long r0 = t * tile_rows;
        const long long r1 = r0 + tile_rows < m ? r0 + tile_rows : m;
        // the tile's column window
        const int j0 = rp[r0], j1 = rp[r1];
        int cmin = INT_MAX, cmax = -1;
        for (int j = j0 + tid; j < j1; j += GROUP_THREADS) {
            const int c = ci[j];
            cmin = c < cmin ? c : cmin;
            cmax = c > cmax ? c : cmax;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int a = __shfl_xor_sync(FULL, cmin, o), b = __shfl_xor_sync(FULL, cmax, o);
            cmin = a < cmin ? a : cmin;
            cmax = b > cmax ? b : cmax;
        }
        if (lane == 0) {
            s_min[w] = cmin;
            s_max[w] = cmax;
        }
        __syncthreads();
        cmin = s_min[0];
        cmax = s_max[0];
#pragma unroll
        for (int q = 1; q < WARPS; ++q) {
            cmin = s_min[q] < cmin ? s_min[q] : cmin;
            cmax = s_max[q] > cmax ? s_max[q] : cmax;
        }
        const int W = cmax >= cmin ? cmax - cmin + 1 : 0;
        const bool staged = W > 0 && W <= max_w &&
                            guard(err, cmin >= 0 && cmax < n, G_X, cmin < 0 ? cmin : cmax);
        if (staged) {  // X[cmin .. cmax][0 .. k) -> xs, row stride k; SU loads in flight
            constexpr int SU = 8;
            const int total = W * k;  // <= WINDOW_SMEM / sizeof(VT)
            const VT *src = X + (long long)cmin * ldx;
            for (int q0 = tid; q0 < total; q0 += SU * GROUP_THREADS) {
                VT t[SU];
#pragma unroll
                for (int u = 0; u < SU; ++u) {
                    const int q = q0 + u * GROUP_THREADS;
                    if (q < total) {
                        if (ldx == k) {
                            t[u] = ld_x(src + q, pl);
                        } else {
                            const int wr = q / k;
                            t[u] = ld_x(src + (long long)wr * ldx + (q - wr * k), pl);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < SU; ++u) {
                    const int q = q0 + u * GROUP_THREADS;
                    if (q < total) xs[q] = t[u];
                }
            }
        }
        __syncthreads();
        for (long long rb = r0; rb < r1; rb += rows_per_pass) {
            const long long r = rb + (long long)w * gpw + grp;
            const bool valid = r < r1;
            int a = 0, b = 0;
            if (valid) {
                a = rp[r];
                b = rp[r + 1];
            }
            ColAcc acc[KPL];
            int j = a + e;
            if constexpr (KCT != 0) {
                if (staged)
                    coop_row<KPL, KCT>(
                        a, b, gi, gl, es, e, lane, ci, v,
                        [&](int col, VT(&xv)[KPL]) {
#pragma unroll
                            for (int p = 0; p < KPL; ++p)
                                xv[p] = col >= 0 && colok[p] ? xs[(col - cmin) * k + cl + p * kc]
                                                             : VT(0);
                        },
                        acc, pf);
                else
                    coop_row<KPL, KCT>(
                        a, b, gi, gl, es, e, lane, ci, v,
                        [&](int col, VT(&xv)[KPL]) {
                            const bool in = col >= 0 && guard(err, col < n, G_X, col);
#pragma unroll
                            for (int p = 0; p < KPL; ++p)
                                xv[p] = in && colok[p]
                                            ? ld_x(X + (long long)col * ldx + cl + p * kc, pl)
                                            : VT(0);
                        },
                        acc, pf);
                j = b;
            } else if (staged) {  // WU elements' values and columns in flight, then the shared reads
                constexpr int WU = 4;
                for (; j + (WU - 1) * es < b; j += WU * es) {
                    VT val[WU];
                    int col[WU];
#pragma unroll
                    for (int u = 0; u < WU; ++u) {
                        val[u] = ld_val(v + j + u * es, pf);
                        col[u] = ld_col(ci + j + u * es, pf);
                    }
#pragma unroll
                    for (int u = 0; u < WU; ++u) {
                        const VT *xr = xs + (col[u] - cmin) * k + cl;
#pragma unroll
                        for (int p = 0; p < KPL; ++p)
                            if (colok[p]) acc[p].add(val[u], xr[p * kc]);
                    }
                }
            }
            for (; j < b; j += es) {
                const VT val = ld_val(v + j, pf);
                const int col = ld_col(ci + j, pf);
                if (staged) {
                    const VT *xr = xs + (col - cmin) * k + cl;
#pragma unroll
                    for (int p = 0; p < KPL; ++p)
                        if (colok[p]) acc[p].add(val, xr[p * kc]);
                } else if (guard(err, col >= 0 && col < n, G_X, col)) {
                    const VT *xr = X + (long long)col * ldx + cl;
#pragma unroll
                    for (int p = 0; p < KPL; ++p)
                        if (colok[p]) acc[p].add(val, ld_x(xr + p * kc, pl));
                }
            }
#pragma unroll
            for (int p = 0; p < KPL; ++p) {
                double s = acc[p].value();
                for (int o = kc; o < gl; o <<= 1) s += __shfl_xor_sync(FULL, s, o);
                if (valid && e == 0 && colok[p]) Y[r * ldy + cl + p * kc] = s;
            }
        }
        __syncthreads();  // xs is restaged by the next tile
    }
}

// SpMV on plain CSR (one right-hand side): groups of GL lanes own a row at a time, lane gi taking
// elements gi, gi + GL, ...; a fixed butterfly adds the lanes.  Rows of very uneven length are kept
// off the critical path:
//
//  * a row longer than LONG = 4 U GL is summed by the whole warp, WU elements per lane at a time:
//    in its group it would run len / (U GL) dependent rounds while the other groups wait.  Narrow
//    groups (GL <= 4) keep them where so many of a warp's rows are long that one after the other
//    they would take more rounds (one lane per row, us, each row by the warp / this: banded 500,000
//    rows of 24 140 / 117 with L2 flushed, in tiles of 512 rows 494 / 129; power law 40,000 rows 45 / 43,
//    and 73 where half as many rows were enough to stay in the groups).  They have a loop of their own:
//    choosing before the short rows' loop cost Laplacian 1960^2 15 % (77 -> 88 us; this 74).  FP64 rows
//    of one lane stay with the warp where there are more tiles than warps (by_cta > 1), since a lane per
//    row reads a line per element then: dense blocks 300,000 rows in tiles of 32 219 / 96 us, stencil
//    110^3 in tiles of 128 528 / 288 by the groups / the warp, L2 flushed;
//  * a row longer than HUGE_ROW waits until the CTA's tiles are done and is summed by all of its
//    warps.  Each warp keeps up to LIST such rows (and sums further ones alone), so which rows
//    take which way depends on the matrix and the launch shape only, and results repeat bit
//    for bit.  Nothing is kept in global memory: calls on one handle may overlap.
//
// What bounds it: on power-law rows the chain row pointer -> values and columns -> x of each round
// and the gathers (one L1 wavefront each on random columns); on regular rows instruction issue.
// Compile-time GL and 32-bit offsets keep a round short enough for six CTAs per SM.  FP64, L2
// flushed, against one group per row whatever its length: power-law rows (700,001, mean 16,
// longest about 7,000) 457 -> 96 us, 4,194,304 rows 806 -> 400 us; 27-point stencil 128^3 190 ->
// 158 us, dense blocks 158 -> 132 us (8 lanes each).  Reading the row pointers of 32 rows at once,
// and keeping the next round's loads in flight at four CTAs per SM, were slower (96-107 us and
// 125 us on the 700,001 rows; 172 and 221 us on the stencil), as were HUGE_ROW = 2,048 (39
// against 33 us on 100,003 power-law rows) and seven or eight CTAs (spills).
constexpr int HUGE_ROW = 1024, LIST = 8;
constexpr int SPMV_MINB = 6;

template <int GL, typename VT>
__global__ void __launch_bounds__(GROUP_THREADS, SPMV_MINB)
csr_spmv_kernel(const int *__restrict__ rp, const int *__restrict__ ci, const VT *__restrict__ v,
                const VT *x, long long ldx, double *__restrict__ y, long long ldy,
                int m, int tile_rows, unsigned by_cta, unsigned by_warp, int n,
                unsigned long long *err) {
    constexpr int U = 4, WU = 4, GPW = 32 / GL, WARPS = GROUP_THREADS / 32;
    constexpr int LONG = GL < 32 ? 4 * U * GL : HUGE_ROW;
    __shared__ int s_list[WARPS][LIST], s_cnt[WARPS];
    __shared__ double s_sum[WARPS];
    pdl_wait();
    pdl_trigger();  // after the wait: one product ahead at most, see deal_tiles
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int grp = lane / GL, gi = lane % GL;
    const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
    const long long ntiles = ((long long)m + tile_rows - 1) / tile_rows;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    const int rounds = tile_rows / GPW;

    auto gather = [&](int col) -> VT {
        if (!guard(err, col >= 0 && col < n, G_X, col)) return VT(0);
        return ld_x(x + (long long)col * ldx, pl);
    };
    // elements [j0, j1) of a row, this thread taking j0 + first, then every `step`-th
    auto strided = [&](int j0, int j1, unsigned first, unsigned step) -> double {
        Acc<VT> acc;
        const VT *vr = v + j0;
        const int *cr = ci + j0;
        const unsigned len = (unsigned)(j1 - j0);  // unsigned offsets: no overflow near 2^31
        for (unsigned j = first; j < len; j += WU * step) {
            VT val[WU], xv[WU];
            int col[WU];
#pragma unroll
            for (int u = 0; u < WU; ++u) {
                const bool in = j + u * step < len;
                val[u] = in ? ld_val(vr + j + u * step, pf) : VT(0);
                col[u] = in ? ld_col(cr + j + u * step, pf) : -1;
            }
#pragma unroll
            for (int u = 0; u < WU; ++u) xv[u] = col[u] >= 0 ? gather(col[u]) : VT(0);
#pragma unroll
            for (int u = 0; u < WU; ++u)
                if (col[u] >= 0) acc.add(val[u], xv[u]);
        }
        return acc.value();
    };

    int cnt = 0;
    for (unsigned t = blockIdx.x * by_cta + w * by_warp; t < (unsigned)ntiles;
         t += (unsigned)nwarps) {
        // row of the tile's first round (< m + tile_rows <= 2^31 + 2^20: unsigned)
        unsigned r = t * (unsigned)tile_rows + grp;
        for (int i = 0; i < rounds; ++i, r += GPW) {
            int a = 0, b = 0;
            if (r < (unsigned)m) {
                a = rp[r];
                b = rp[r + 1];
            }
            const int len = b - a;
            const bool is_long = len > LONG;
            const VT *vr = v + a;
            const int *cr = ci + a;
            auto by_group = [&](int count) -> double {  // the row's first `count` elements, by its group
                Acc<VT> acc;
                for (int j = gi; j < count; j += U * GL) {
                    VT val[U];
                    int col[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const bool in = j + u * GL < len;
                        val[u] = in ? ld_val(vr + (j + u * GL), pf) : VT(0);
                        col[u] = in ? ld_col(cr + (j + u * GL), pf) : -1;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (col[u] >= 0) acc.add(val[u], gather(col[u]));
                }
                double s = acc.value();
#pragma unroll
                for (int o = 1; o < GL; o <<= 1) s += __shfl_xor_sync(FULL, s, o);
                return s;
            };
            const double s = by_group(is_long ? 0 : len);
            if (r < (unsigned)m && gi == 0 && !is_long) y[r * ldy] = s;
            unsigned todo = __ballot_sync(FULL, is_long && gi == 0);
            // many of them: the groups are done sooner, all at once
            if (GL <= 4 && todo && !(GL == 1 && sizeof(VT) == 8 && by_cta != 1u)) {
                const bool mid = is_long && len <= HUGE_ROW;
                const int most = __reduce_max_sync(FULL, mid ? len : 0);
                const int count = __popc(__ballot_sync(FULL, mid && gi == 0));
                if (count * ((most + 32 * WU - 1) / (32 * WU)) >= (most + U * GL - 1) / (U * GL)) {
                    const double sm = by_group(mid ? len : 0);
                    if (mid && gi == 0) y[r * ldy] = sm;
                    todo = __ballot_sync(FULL, is_long && !mid && gi == 0);
                }
            }
            // long rows, one after the other, by the whole warp
            while (todo) {
                const int src = __ffs(todo) - 1;
                todo &= todo - 1;
                const int al = __shfl_sync(FULL, a, src), bl = __shfl_sync(FULL, b, src);
                const int rl = __shfl_sync(FULL, (int)r, src);
                if (bl - al > HUGE_ROW && cnt < LIST) {
                    if (lane == 0) s_list[w][cnt] = rl;
                    ++cnt;
                    continue;
                }
                const double sl = warp_sum(strided(al, bl, lane, 32));
                if (lane == 0) y[rl * ldy] = sl;
            }
        }
    }
    if (lane == 0) s_cnt[w] = cnt;
    if (!__syncthreads_or(cnt)) return;  // nearly always: no list to walk, which took 2.5 us
    for (int q = 0; q < WARPS * LIST; ++q) {
        if (q % LIST >= s_cnt[q / LIST]) {
            q |= LIST - 1;  // the warp's list is done; the same for every thread
            continue;
        }
        const int rl = s_list[q / LIST][q % LIST];
        const double t = warp_sum(strided(rp[rl], rp[rl + 1], threadIdx.x, GROUP_THREADS));
        if (lane == 0) s_sum[w] = t;
        __syncthreads();
        if (threadIdx.x == 0) {
            double sum = s_sum[0];
#pragma unroll
            for (int k = 1; k < WARPS; ++k) sum += s_sum[k];
            y[rl * ldy] = sum;
        }
        __syncthreads();  // s_sum is written again by the next row
    }
}

// The grid for ntiles tiles of a warp each with `resident` CTAs per SM, and the first tile of warp w of CTA
// b, b * by_cta + w * by_warp.  Up to a full GPU tile t goes to warp t / grid of CTA t % grid and every
// SM gets as many CTAs, so that every SM has an even share: FP32C SpMV in a loop, us, before / after:
// banded 30,000 rows 13.7 / 10.4, dense blocks 30,000 18.6 / 14.1, power law 40,000 21.6 / 17.7.
// A product's CTAs come in while those of the product before run (of that one only: the kernels let
// their dependents launch after their own wait).  Where both do not fit at once, the SMs whose CTAs end
// first would get more of the next, so more than half a GPU takes all of it, and every place is used
// once.  In a loop, us, before / after: SpMV of banded 500,000 rows, one lane each, 121 / 89, dense blocks
// 300,000 rows, two lanes, 93 / 67; k = 2 on banded 300,007 rows, one lane, 100 / 54.
struct TileDeal {
    unsigned grid, by_cta, by_warp;
};
TileDeal deal_tiles(long long ntiles, int sms, int resident) {
    constexpr int WARPS = GROUP_THREADS / 32;
    const long long want = (ntiles + WARPS - 1) / WARPS;
    long long per_sm = (want + sms - 1) / sms;
    if (per_sm < 1) per_sm = 1;
    if (2 * per_sm > resident) per_sm = resident;
    const unsigned grid = (unsigned)(per_sm * sms);
    const bool one_each = ntiles <= (long long)grid * WARPS;
    return {grid, one_each ? 1u : (unsigned)WARPS, one_each ? grid : 1u};
}

int ilog2(int v) {
    int s = 0;
    while ((1 << s) < v) ++s;
    return s;
}

// Calls f(std::integral_constant<int, KC>) for the column-lane count kc (1 = not cooperative).
template <typename F>
cudaError_t with_kc(int kc, F f) {
    switch (kc) {
        case 1: return f(std::integral_constant<int, 0>());
        case 2: return f(std::integral_constant<int, 2>());
        case 4: return f(std::integral_constant<int, 4>());
        case 8: return f(std::integral_constant<int, 8>());
        case 16: return f(std::integral_constant<int, 16>());
        case 32: return f(std::integral_constant<int, 32>());
        default: return cudaErrorInvalidValue;
    }
}

template <int KPL, typename VT>
cudaError_t launch_window(const Handle &h, const VT *x, long long ldx, double *y, long long ldy,
                          int k, cudaStream_t s) {
    const int tr = h.rows_per_tile;
    const long long ntiles = ((long long)h.m + tr - 1) / tr;
    const long long cap = (long long)h.sm_count * WINDOW_MINB;
    const unsigned grid = (unsigned)(ntiles < cap ? (ntiles > 0 ? ntiles : 1) : cap);
    const int max_w = (int)(WINDOW_SMEM / ((size_t)k * sizeof(VT)));
    const size_t smem = (size_t)max_w * k * sizeof(VT);
    return with_kc(h.col_lanes, [&](auto KCC) {
        constexpr int KCT = decltype(KCC)::value;
        // per launch: the attribute belongs to the current device
        const cudaError_t attr = cudaFuncSetAttribute(
            csr_window_kernel<KPL, VT, KCT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
            WINDOW_SMEM);
        if (attr != cudaSuccess) return attr;
        return launch_product(csr_window_kernel<KPL, VT, KCT>, grid, GROUP_THREADS, smem, s, h.rp,
                              h.ci, (const VT *)h.v, x, ldx, y, ldy, h.m, k,
                              ilog2(h.lanes_per_row), ilog2(h.col_lanes), tr, max_w, h.n,
                              guard_word());
    });
}

// One right-hand side, one column lane: the SpMV kernel for the group width.
template <typename VT>
cudaError_t launch_spmv(const Handle &h, const VT *x, long long ldx, double *y, long long ldy,
                        cudaStream_t s) {
    const int tr = h.rows_per_tile;
    const TileDeal d = deal_tiles(((long long)h.m + tr - 1) / tr, h.sm_count, SPMV_MINB);
    auto go = [&](auto GLC) {
        return launch_product(csr_spmv_kernel<decltype(GLC)::value, VT>, d.grid, GROUP_THREADS, 0, s,
                              h.rp, h.ci, (const VT *)h.v, x, ldx, y, ldy, h.m, tr, d.by_cta,
                              d.by_warp, h.n, guard_word());
    };
    switch (h.lanes_per_row) {
        case 1: return go(std::integral_constant<int, 1>());
        case 2: return go(std::integral_constant<int, 2>());
        case 4: return go(std::integral_constant<int, 4>());
        case 8: return go(std::integral_constant<int, 8>());
        case 16: return go(std::integral_constant<int, 16>());
        case 32: return go(std::integral_constant<int, 32>());
        default: return cudaErrorInvalidValue;
    }
}

template <int KPL, typename VT>
cudaError_t launch_rows(const Handle &h, const VT *x, long long ldx, double *y, long long ldy,
                        int k, cudaStream_t s) {
    const int kc = h.col_lanes;
    const int tr = h.rows_per_tile;
    const TileDeal d = deal_tiles(((long long)h.m + tr - 1) / tr, h.sm_count,
                                  kc > 1 ? COOP_MINB : group_minb<KPL>());
    const int gs = ilog2(h.lanes_per_row), ks = ilog2(kc);
    // pairs of columns per vector read when every pair is whole and 2-element aligned
    const bool vec2 = KPL >= 2 && k % 2 == 0 && ldx % 2 == 0 &&
                      reinterpret_cast<uintptr_t>(x) % (2 * sizeof(VT)) == 0;
    return with_kc(kc, [&](auto KCC) {
        constexpr int KCT = decltype(KCC)::value;
        constexpr int VW2 = KPL >= 2 ? 2 : 1;
        if constexpr (KPL == 1 && KCT == 0) {
            return cudaErrorInvalidValue;  // one column in one lane: launch_spmv
        } else {
            auto go = [&](auto kernel) {
                return launch_product(kernel, d.grid, GROUP_THREADS, 0, s, h.rp, h.ci,
                                      (const VT *)h.v, x, ldx, y, ldy, h.m, k, gs, ks, tr, d.by_cta,
                                      d.by_warp, h.n, guard_word());
            };
            return vec2 ? go(csr_group_kernel<KPL, VT, KCT, VW2>)
                        : go(csr_group_kernel<KPL, VT, KCT, 1>);
        }
    });
}

template <typename VT>
cudaError_t launch_group(const Handle &h, const void *X, long long ldx, void *Y, long long ldy,
                         int k, cudaStream_t s) {
    const VT *x = (const VT *)X;
    double *y = (double *)Y;
    if (h.x_window) {
        switch (h.cols_per_lane) {
            case 1: return launch_window<1, VT>(h, x, ldx, y, ldy, k, s);
            case 2: return launch_window<2, VT>(h, x, ldx, y, ldy, k, s);
            case 4: return launch_window<4, VT>(h, x, ldx, y, ldy, k, s);
            default: return cudaErrorInvalidValue;
        }
    }
    if (k == 1 && h.col_lanes == 1 && h.cols_per_lane == 1)
        return launch_spmv<VT>(h, x, ldx, y, ldy, s);
    switch (h.cols_per_lane) {
        case 1: return launch_rows<1, VT>(h, x, ldx, y, ldy, k, s);
        case 2: return launch_rows<2, VT>(h, x, ldx, y, ldy, k, s);
        case 4: return launch_rows<4, VT>(h, x, ldx, y, ldy, k, s);
        default: return cudaErrorInvalidValue;
    }
}

__global__ void narrow_kernel(const double *__restrict__ src, float *__restrict__ dst,
                              long long n) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        dst[i] = (float)src[i];
}

}  // namespace

cudaError_t csr_spmm(const Handle &h, const void *X, long long ldx, void *Y, long long ldy,
                     int k, cudaStream_t s) {
    if (h.m <= 0 || k <= 0) return cudaSuccess;
    if (csr_staged_shape(h, k))
        return csr_spmm_staged(h, X, ldx, Y, ldy, k, h.lanes_per_row, h.cols_per_lane, s);
    if (h.precision == PAVA_PREC_FP32C) return launch_group<float>(h, X, ldx, Y, ldy, k, s);
    return launch_group<double>(h, X, ldx, Y, ldy, k, s);
}

cudaError_t csr_spmv(const Handle &h, const void *x, void *y, cudaStream_t s) {
    return csr_spmm(h, x, 1, y, 1, 1, s);
}

cudaError_t narrow_to_float(const double *src, float *dst, long long n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    long long blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    narrow_kernel<<<(unsigned)blocks, 256, 0, s>>>(src, dst, n);
    return cudaGetLastError();
}

}  // namespace pava
