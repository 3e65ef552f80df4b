// GPU CSR5: CSR -> CSR5 conversion and CSR5 SpMV for sm_100a.
//
// The reference's CSR5 (csr5/, anonymouslib for AVX-512) cuts the nnz range into tiles of
// omega lanes x sigma elements (omega = 8 there), stores a tile pointer (the tile's first row,
// format_avx512.h:8-28), per-lane bit flags marking row starts (format_avx512.h:85-121) and
// transposes each tile so that step i of all lanes is contiguous (format_avx512.h:365-426).
// The SpMV does a per-lane segmented sum, a cross-lane scan (hscan_avx512) and adds the
// partial row that crosses thread boundaries through a calibrator (csr5_spmv_avx512.h:52-308).
//
// Here omega is the warp (32 lanes) and sigma is a multiple of 4 (default 16):
//  * a tile descriptor is one 32-bit row-start mask per lane.  The y_offset and
//    scansum_offset fields the reference packs beside the flags (format_avx512.h:123-233) are
//    recomputed per tile from the masks with a warp scan and ballot, which costs a few
//    instructions instead of descriptor bytes.
//  * empty rows are given one zero element in column -1 (see k_cvr.cu), so every row of a
//    tile is consecutive and no descriptor-offset table (format_avx512.h:271-363) is needed.
//  * a warp walks G consecutive tiles (a chunk) carrying the open row in registers; the
//    chunk's shared first/last rows go to the carry slots combined by k_support.cu, the
//    deterministic form of the calibrator (csr5_spmv_avx512.h:292-308).  The reference's
//    serial tail partition (:311-342) does not exist: the last tile is padded.
//
// Tile t (32*sigma elements; element (lane l, step i) = original position t*32*sigma +
// l*sigma + i) holds its values and columns in the 4-step block layout of k_stream.cuh, so a
// chunk of G tiles is one run of G*sigma/4 blocks;
//   desc[t*32 + l]  bit i: element (l, i) is the first element of a row
//   tile_ptr[t]     row of element (0, 0)

#include <type_traits>

#include "k_stream.cuh"
#include "pava_internal.h"

namespace pava {

namespace {

// 16-bit offset of a column from the chunk's base (a conversion whose columns are out of reach
// never gets here), or the column itself.
template <typename IT> __device__ __forceinline__ IT enc_col(int col, int base) {
    return sizeof(IT) == 2 ? (IT)(col < 0 ? DELTA_NONE : col - base) : (IT)col;
}

// CSR -> CSR5, a warp per tile.  The tile's values and columns are read from the CSR in order
// (coalesced) into shared memory, one slot of padding after each lane's SIGMA elements, and
// leave as whole 16-byte vectors per lane; row starts and the zero elements of empty rows are
// marked in bitmaps of the tile's SIGMA words.  What bounds it: the bytes (12 read and 10-12
// written per nonzero).  Reading the CSR lane by lane (32 runs of SIGMA elements at once) took
// 64 L1 wavefronts per 32 elements: 223 us for 23.9 M nonzeros (sigma 16, 16-bit offsets), and
// finding each lane's row by bisection; this one takes 99 us (the bytes: 81 us).
//
// The last tile of a chunk writes its header: r_first, nrows, shared.  aux bits 1..31 are the
// base column of the chunk's 16-bit offsets, bit 0 says that the chunk holds elements that read no
// x (the zero element of an empty row, or the padding of the last chunk); chunks without them
// skip that check.  aux starts at 0 and is or-ed by the chunk's tiles.
template <int SIGMA> constexpr int conv_warps() { return SIGMA > 16 ? 2 : 4; }

template <int SIGMA, typename VT, typename IT>
__global__ void __launch_bounds__(conv_warps<SIGMA>() * 32)
csr5_convert_kernel(const int *__restrict__ rp, const int *__restrict__ ci,
                    const double *__restrict__ v, const int *__restrict__ arp, int m,
                    long long ntiles, int G, VT *__restrict__ vals, IT *__restrict__ cols,
                    unsigned *__restrict__ desc, const int *__restrict__ tile_ptr,
                    ChunkHdr *__restrict__ hdr, const int *__restrict__ colbase,
                    const int *__restrict__ ovf) {
    constexpr int W = conv_warps<SIGMA>(), T = 32 * SIGMA, LD = SIGMA + 1;
    __shared__ VT s_val[W][32 * LD];
    __shared__ IT s_col[W][32 * LD];
    __shared__ unsigned s_start[W][SIGMA + 1], s_dummy[W][SIGMA];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long t = (long long)blockIdx.x * W + w;
    if (t >= ntiles) return;                     // warp-uniform: no block-wide barrier below
    if (sizeof(IT) == 2 && *ovf) return;
    const long long c = t / G;
    const int tbase = (int)(t * T);              // the padded element space is below 2^31
    const int base = sizeof(IT) == 2 ? colbase[c] : 0;
    const int r0 = tile_ptr[t];                  // row of the first element, <= m
    const int pad0 = arp[m] - tbase;             // offset of the padding
    if (lane < SIGMA) s_start[w][lane] = s_dummy[w][lane] = 0u;
    if (lane == 0) s_start[w][SIGMA] = 0u;
    __syncwarp();
    // starts of the tile's rows r0, r0 + 1, ... (every row has an element, so at most T of them)
    for (int r = r0 + lane;; r += 32) {
        int off = T;
        if (r <= m) {
            off = arp[r] - tbase;                // r0 may have started before the tile
            if (off >= 0 && off < T) {
                atomicOr(&s_start[w][off >> 5], 1u << (off & 31));
                if (r < m && rp[r + 1] == rp[r]) atomicOr(&s_dummy[w][off >> 5], 1u << (off & 31));
            }
        }
        if (__shfl_sync(FULL, off, 31) >= T) break;
    }
    __syncwarp();
    const unsigned lt = lanemask_lt();
    // CSR position of offset 0 (row m, all padding, reads nothing)
    int p = r0 < m ? rp[r0] + (tbase - arp[r0]) : 0;
    bool none = false;
    constexpr int U = SIGMA % 8 == 0 ? 8 : 4;  // rounds of 32 elements in flight
#pragma unroll 1
    for (int it = 0; it < SIGMA; it += U) {
        double val[U];
        int col[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned dm = s_dummy[w][it + u];
            const bool dummy = ((dm >> lane) & 1u) || (it + u) * 32 + lane >= pad0;
            const int q = p + lane - __popc(dm & lt);
            p += 32 - __popc(dm);
            none |= dummy;
            val[u] = 0.0;
            col[u] = -1;
            if (!dummy) {
                val[u] = v[q];
                col[u] = ci[q];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int off = (it + u) * 32 + lane, slot = off + off / SIGMA;
            s_val[w][slot] = (VT)val[u];
            s_col[w][slot] = enc_col<IT>(col[u], base);
        }
    }
    __syncwarp();
    // the lane's SIGMA start bits
    const int b0 = lane * SIGMA;
    unsigned F = s_start[w][b0 >> 5] >> (b0 & 31);
    if ((b0 & 31) + SIGMA > 32) F |= s_start[w][(b0 >> 5) + 1] << (32 - (b0 & 31));
    if (SIGMA < 32) F &= (1u << (SIGMA & 31)) - 1u;
    desc[t * 32 + lane] = F;
    VT *vt = vals + t * T;
    IT *ct = cols + t * T;
    const VT *sv = &s_val[w][lane * LD];
    const IT *sc = &s_col[w][lane * LD];
#pragma unroll
    for (int b = 0; b < SIGMA / 4; ++b) {
        if constexpr (sizeof(VT) == 8) {
            double2 *o = reinterpret_cast<double2 *>(vt);
            o[(2 * b) * 32 + lane] = make_double2(sv[4 * b], sv[4 * b + 1]);
            o[(2 * b + 1) * 32 + lane] = make_double2(sv[4 * b + 2], sv[4 * b + 3]);
        } else {
            reinterpret_cast<float4 *>(vt)[b * 32 + lane] =
                make_float4(sv[4 * b], sv[4 * b + 1], sv[4 * b + 2], sv[4 * b + 3]);
        }
        if constexpr (sizeof(IT) == 4)
            reinterpret_cast<int4 *>(ct)[b * 32 + lane] =
                make_int4(sc[4 * b], sc[4 * b + 1], sc[4 * b + 2], sc[4 * b + 3]);
        else
            reinterpret_cast<short4 *>(ct)[b * 32 + lane] =
                make_short4(sc[4 * b], sc[4 * b + 1], sc[4 * b + 2], sc[4 * b + 3]);
    }
    none = __any_sync(FULL, none);
    int nst = __popc(F);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nst += __shfl_xor_sync(FULL, nst, o);
    if (lane == 0) {
        const bool last = t % G == G - 1;
        const int or_aux = (last ? (int)((unsigned)base << 1) : 0) | (none ? 1 : 0);
        if (or_aux) atomicOr(&hdr[c].aux, or_aux);
        if (last) {
            const long long s = c * G * (long long)T, e = s + G * (long long)T;
            const int r_first = tile_ptr[c * G];
            const int r_last = r0 + nst - (int)(F & 1u);  // the row of the last element
            unsigned sh = 0;
            if ((long long)arp[r_first] < s) sh |= 1u;
            if ((long long)arp[r_last + 1] > e) sh |= 2u;
            hdr[c].r_first = r_first;
            hdr[c].nrows = r_last - r_first + 1;
            hdr[c].shared = sh;
        }
    }
}

// Tile end: the cross-lane combine of the lanes' open row pieces.  head is the piece a lane
// adds to the row open at its start (its whole sum when no row starts in the lane), tail the
// sum since the lane's last row start (seen: a row starts in the lane), rowcur the row of that
// tail, next_row the row open at the tile's end.  Rows that end in the tile go to y (or to
// the chunk's carry slots); the open row's sum stays in carry_row / carry_val.  The FP64
// kernel has the same steps inline: calling this helper there changed its register allocation
// and doubled its spills at 80 registers.
__device__ __forceinline__ void tile_combine(double head, double tail, bool seen, int rowcur,
                                             int next_row, int lane, int r_first, int r_last,
                                             unsigned shared, long long c, double *y,
                                             double *carry_head, double *carry_tail, int m,
                                             int &carry_row, double &carry_val,
                                             unsigned long long *err) {
    const unsigned sm = __ballot_sync(FULL, seen);
    const double Hs = seg_suffix(head, !seen, lane);
    double Hn = __shfl_down_sync(FULL, Hs, 1);
    if (lane == 31) Hn = 0.0;
    const double H0 = __shfl_sync(FULL, Hs, 0);
    if (sm == 0) {
        carry_val += H0;  // the whole tile continues the open row
    } else {
        const int lstar = 31 - __clz(sm);
        const double own_l = tail + Hn;
        if (seen && lane != lstar && rowcur < m && guard(err, rowcur >= 0, G_Y, rowcur))
            y[rowcur] = own_l;
        const double own = __shfl_sync(FULL, own_l, lstar);
        if (carry_row >= 0 && lane == 0)
            flush_row(carry_row, carry_val + H0, r_first, r_last, shared, c, y, carry_head,
                      carry_tail, m, err);
        carry_row = next_row;
        carry_val = own;
    }
}

// Warps per CTA and CTAs per SM: one CTA of 24 or 20 warps, or three of 8 (csr5_spmv chooses).
// FP64: 24 warps with 80 registers for 16-bit columns; 20 with 96 for 32-bit ones, which spill at 80 and
// keep more of a chunk in flight at 96.  A product in a loop, us, 24 / 20 warps: 32-bit columns, stencil
// 72^3 37.3 / 30.1, 128^3 158 / 150, dense blocks 17 M nonzeros 56 / 45, power law 66 M 338 / 294;
// 16-bit columns, stencil 100^3 66.6 / 70.4, 128^3 135 / 143, Laplacian 2000^2 62 / 67 (dense blocks
// 8.6 M 31.4 / 28.2).  16 warps with 128 registers: power law 302 where 20 took 300.
// One CTA puts that many neighbouring chunks on the SM, which share lines of x: 256 stacked small
// matrices FP32 67 -> 51 us, FP64 105 -> 85, stencil 128^3 FP64 138 -> 135, power law of 102,000 rows
// FP64 16.0 -> 12.0, against CTAs of 8 or 4 warps; CTAs of 12 or 10 lie between.
template <int W> struct Csr5Shape {
    static_assert(W == 24 || W == 20 || W == 8, "launch shape");
    static constexpr int WARPS = W, CTAS = W == 8 ? 3 : 1;
};

// CSR5 SpMV (FP64 values; the FP32 form is csr5_spmv_f32_kernel below): one warp per chunk of
// G tiles, walked as one pipelined run of 4-step blocks
// (values two blocks ahead, columns three, x one); tile descriptors one tile ahead.
//
// Row ends inside a tile: when no lane of the warp starts more than KSTK rows in the tile
// (the usual case), an element that starts a row parks the lane's finished piece in the
// lane's next shared-memory slot (a predicated store) and restarts the accumulator (a select),
// so the step has no branch; at the tile end piece 0 (the end of the row the lane started
// with) joins the cross-lane combine and pieces 1 .. k-1, rows that start and end in the
// lane, go to y.  Other tiles write each finished row as it ends.
template <int SIGMA, typename VT, typename IT, int W>
__global__ void __launch_bounds__(Csr5Shape<W>::WARPS * 32, Csr5Shape<W>::CTAS)
csr5_spmv_kernel(const ChunkHdr *__restrict__ hdr, const int *__restrict__ tile_ptr,
                 const unsigned *__restrict__ desc, const VT *__restrict__ vals,
                 const IT *__restrict__ cols, const VT *x,
                 double *__restrict__ y, double *__restrict__ carry_head,
                 double *__restrict__ carry_tail, ChunkWalk<Csr5Shape<W>::WARPS> walk,
                 int G, int m, int n,
                 unsigned long long *err) {
    constexpr int NBT = SIGMA / 4;  // blocks per tile
    constexpr int SPMV_WARPS = Csr5Shape<W>::WARPS;
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
    constexpr int KSTK = 4;
    constexpr unsigned SLOT = SPMV_WARPS * 32 * 8;  // bytes between a thread's slots
    __shared__ __align__(16) double s_piece[KSTK * SPMV_WARPS * 32];
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(&s_piece[threadIdx.x]);

    for (unsigned c = walk.first(); walk.ok(c); c = walk.next(c)) {
        const ChunkHdr H = hdr[c];
        const int r_first = H.r_first, r_last = H.r_first + H.nrows - 1;
        const unsigned shared = H.shared;
        int carry_row = (shared & 1u) ? r_first : -1;
        double carry_val = 0.0;
        const long long t0 = (long long)c * G;
        const VT *vb = vals + t0 * 32 * SIGMA;
        const IT *cb = cols + t0 * 32 * SIGMA;
        const int xbase = sizeof(IT) == 2 ? (int)((unsigned)H.aux >> 1) : 0;  // offsets' base
        const VT *xb = x + xbase;
        const int xlo = -xbase, xhi = n - xbase;  // the offsets that stay inside x
        const int NB = G * NBT;

        CBlk<IT> c1 = CBlk<IT>::load(cb, 1, lane, pf);
        CBlk<IT> c2 = CBlk<IT>::load(cb, NB > 2 ? 2 : 1, lane, pf);
        VBlk<VT> v0 = VBlk<VT>::load(vb, 0, lane, pf), v1 = VBlk<VT>::load(vb, 1, lane, pf);
        VT x0[4];
        {
            const CBlk<IT> c0 = CBlk<IT>::load(cb, 0, lane, pf);
            pdl_wait();  // x, and y and the carries, which the product before may still use
#pragma unroll
            for (int q = 0; q < 4; ++q) x0[q] = c0.gather(q, xb, pl, xlo, xhi, err);
        }
        unsigned Fn = ld_stream(desc + t0 * 32 + lane, pf);
        int rsn = tile_ptr[t0];

        unsigned F = 0;
        int rs = 0, b00 = 0, total = 0, rowcur = 0;
        Acc<VT> acc;
        double hpiece = 0.0;
        bool seen = false;
        int tt = 0;
        bool fast = false;
        int nst = 0, row0 = 0;
        unsigned sp = sbase;
#pragma unroll 1
        for (int blk = 0; blk < NB; ++blk) {
            CBlk<IT> cn = c2;
            VBlk<VT> vn = v1;
            if (blk + 3 < NB) cn = CBlk<IT>::load(cb, blk + 3, lane, pf);
            if (blk + 2 < NB) vn = VBlk<VT>::load(vb, blk + 2, lane, pf);
            VT x1[4];
            if (blk + 1 < NB) {
#pragma unroll
                for (int q = 0; q < 4; ++q) x1[q] = c1.gather(q, xb, pl, xlo, xhi, err);
            }
            const int qb = blk % NBT;
            if (qb == 0) {  // tile start
                F = Fn;
                rs = rsn;
                if (tt + 1 < G) {
                    Fn = ld_stream(desc + (t0 + tt + 1) * 32 + lane, pf);
                    rsn = tile_ptr[t0 + tt + 1];
                }
                b00 = (int)(__shfl_sync(FULL, F, 0) & 1u);
                nst = __popc(F);
                const int excl = warp_excl_scan(nst, lane);
                total = __shfl_sync(FULL, excl + nst, 31);
                rowcur = rs + excl - b00;  // row open when the lane starts
                row0 = rowcur;
                acc.reset();
                hpiece = 0.0;
                seen = false;
                fast = !__any_sync(FULL, nst > KSTK);
                sp = sbase;
            }
            const unsigned Fb = F >> (qb * 4);
            if (fast) {  // row ends park the piece in the lane's shared slots: no branch
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const bool st = (Fb >> q) & 1u;
                    acc.push(sp, st);
                    sp += st ? SLOT : 0u;
                    acc.add_restart(v0.get(q), x0[q], st);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if ((Fb >> q) & 1u) {
                        if (seen) {
                            if (rowcur < m && guard(err, rowcur >= 0, G_Y, rowcur)) y[rowcur] = acc.value();
                        } else {
                            hpiece = acc.value();
                            seen = true;
                        }
                        ++rowcur;
                        acc.reset();
                    }
                    acc.add(v0.get(q), x0[q]);
                }
            }
            if (qb == NBT - 1) {  // tile end: combine the lanes' open pieces
                if (fast) {
                    seen = nst > 0;
                    if (seen) hpiece = Acc<VT>::piece_at(sbase);
                    for (int k2 = 1; k2 < nst; ++k2)
                        if (row0 + k2 < m && guard(err, row0 + k2 >= 0 && k2 < KSTK, G_Y, row0 + k2))
                        y[row0 + k2] = Acc<VT>::piece_at(sbase + k2 * SLOT);
                    rowcur = row0 + nst;
                }
                if (!seen) hpiece = acc.value();
                const double tl = seen ? acc.value() : 0.0;
                const unsigned sm = __ballot_sync(FULL, seen);
                const double Hs = seg_suffix(hpiece, !seen, lane);
                double Hn = __shfl_down_sync(FULL, Hs, 1);
                if (lane == 31) Hn = 0.0;
                const double H0 = __shfl_sync(FULL, Hs, 0);
                if (sm == 0) {
                    carry_val += H0;  // the whole tile continues the open row
                } else {
                    const int lstar = 31 - __clz(sm);
                    const double own_l = tl + Hn;
                    if (seen && lane != lstar && rowcur < m && guard(err, rowcur >= 0, G_Y, rowcur))
            y[rowcur] = own_l;
                    const double own = __shfl_sync(FULL, own_l, lstar);
                    if (carry_row >= 0 && lane == 0)
                        flush_row(carry_row, carry_val + H0, r_first, r_last, shared, c, y,
                                  carry_head, carry_tail, m, err);
                    carry_row = rs + total - b00;
                    carry_val = own;
                }
                ++tt;
            }
            c1 = c2; c2 = cn;
            v0 = v1; v1 = vn;
#pragma unroll
            for (int q = 0; q < 4; ++q) x0[q] = x1[q];
        }
        if (carry_row >= 0 && lane == 0)
            flush_row(carry_row, carry_val, r_first, r_last, shared, c, y, carry_head,
                      carry_tail, m, err);
    }
}

template <bool B> struct Flag { static constexpr bool value = B; };

// CSR5 SpMV, FP32-compensated form: the same walk with a tile's sigma/4 blocks unrolled, so
// the block pipeline rotates by register renaming instead of moves, and the fast / slow
// choice and the tile-boundary checks are made once per tile instead of once per block.  The
// compensated add makes this form instruction-issue bound, where the saved instructions are
// time; the FP64 form is bandwidth bound, and unrolled it spills, so it keeps the block loop.
template <int SIGMA, typename IT, int W>
__global__ void __launch_bounds__(Csr5Shape<W>::WARPS * 32, Csr5Shape<W>::CTAS)
csr5_spmv_f32_kernel(const ChunkHdr *__restrict__ hdr, const int *__restrict__ tile_ptr,
                     const unsigned *__restrict__ desc, const float *__restrict__ vals,
                     const IT *__restrict__ cols, const float *x,
                     double *__restrict__ y, double *__restrict__ carry_head,
                     double *__restrict__ carry_tail,
                     ChunkWalk<Csr5Shape<W>::WARPS> walk, int G, int m, int n,
                     unsigned long long *err) {
    using VT = float;
    constexpr int NBT = SIGMA / 4;  // blocks per tile
    constexpr int SPMV_WARPS = Csr5Shape<W>::WARPS;
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
    constexpr int KSTK = 4;
    constexpr unsigned SLOT = SPMV_WARPS * 32 * 8;  // bytes between a thread's slots
    __shared__ __align__(16) double s_piece[KSTK * SPMV_WARPS * 32];
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(&s_piece[threadIdx.x]);

    for (unsigned c = walk.first(); walk.ok(c); c = walk.next(c)) {
        const ChunkHdr H = hdr[c];
        const int r_first = H.r_first, r_last = H.r_first + H.nrows - 1;
        const unsigned shared = H.shared;
        // chunks without elements that read no x skip the gather's test (16-bit offsets and
        // tiles of 24 or 32 steps; the other forms gained nothing from it or spilled)
        constexpr bool SKIP = sizeof(IT) == 2 && SIGMA >= 24;
        const bool chk = !SKIP || (H.aux & 1);
        int carry_row = (shared & 1u) ? r_first : -1;
        double carry_val = 0.0;
        const long long t0 = (long long)c * G;
        const VT *vb = vals + t0 * 32 * SIGMA;
        const IT *cb = cols + t0 * 32 * SIGMA;
        const int xbase = sizeof(IT) == 2 ? (int)((unsigned)H.aux >> 1) : 0;  // offsets' base
        const VT *xb = x + xbase;
        const int xlo = -xbase, xhi = n - xbase;  // the offsets that stay inside x
        const int NB = G * NBT;

        CBlk<IT> c1 = CBlk<IT>::load(cb, 1, lane, pf);
        CBlk<IT> c2 = CBlk<IT>::load(cb, NB > 2 ? 2 : 1, lane, pf);
        VBlk<VT> v0 = VBlk<VT>::load(vb, 0, lane, pf), v1 = VBlk<VT>::load(vb, 1, lane, pf);
        VT x0[4];
        {
            const CBlk<IT> c0 = CBlk<IT>::load(cb, 0, lane, pf);
            pdl_wait();  // x, and y and the carries, which the product before may still use
#pragma unroll
            for (int q = 0; q < 4; ++q) x0[q] = c0.gather(q, xb, pl, xlo, xhi, err);
        }
        unsigned Fn = ld_stream(desc + t0 * 32 + lane, pf);
        int rsn = tile_ptr[t0];

#pragma unroll 1
        for (int tt = 0; tt < G; ++tt) {
            // tile start: the lanes' row-start masks give each lane its first row
            const unsigned F = Fn;
            const int rs = rsn;
            if (tt + 1 < G) {
                Fn = ld_stream(desc + (t0 + tt + 1) * 32 + lane, pf);
                rsn = tile_ptr[t0 + tt + 1];
            }
            const int b00 = (int)(__shfl_sync(FULL, F, 0) & 1u);
            const int nst = __popc(F);
            const int excl = warp_excl_scan(nst, lane);
            const int total = __shfl_sync(FULL, excl + nst, 31);
            const int row0 = rs + excl - b00;  // row open when the lane starts
            const int rem = G - 1 - tt;        // tiles after this one
            int rowcur = row0;
            Acc<VT> acc;
            double hpiece = 0.0;
            bool seen = false;

            // The tile's blocks.  Block qb prefetches block qb + d of the chunk (columns d = 3,
            // values 2, x 1); that block lies (qb + d) / NBT tiles ahead, so only prefetches
            // past this tile compare against the tiles left.  CHK: the chunk has elements that
            // read no x, so each gather tests its column.
            auto walk = [&](auto fast_tag, auto chk_tag) {
                constexpr bool FAST = decltype(fast_tag)::value;
                constexpr bool CHK = decltype(chk_tag)::value;
                unsigned sp = sbase;
#pragma unroll
                for (int qb = 0; qb < NBT; ++qb) {
                    CBlk<IT> cn = c2;
                    VBlk<VT> vn = v1;
                    if ((qb + 3) / NBT == 0 || rem >= (qb + 3) / NBT)
                        cn = CBlk<IT>::load(cb, tt * NBT + qb + 3, lane, pf);
                    if ((qb + 2) / NBT == 0 || rem >= (qb + 2) / NBT)
                        vn = VBlk<VT>::load(vb, tt * NBT + qb + 2, lane, pf);
                    VT x1[4];
                    if ((qb + 1) / NBT == 0 || rem >= (qb + 1) / NBT) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            x1[q] = CHK ? c1.gather(q, xb, pl, xlo, xhi, err)
                                        : c1.gather_all(q, xb, pl, xlo, xhi, err);
                    }
                    if (FAST) {  // row ends park the piece in the lane's shared slots
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const bool st = (F >> (qb * 4 + q)) & 1u;
                            acc.push(sp, st);
                            sp += st ? SLOT : 0u;
                            acc.add_restart(v0.get(q), x0[q], st);
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            if ((F >> (qb * 4 + q)) & 1u) {
                                if (seen) {
                                    if (rowcur < m && guard(err, rowcur >= 0, G_Y, rowcur)) y[rowcur] = acc.value();
                                } else {
                                    hpiece = acc.value();
                                    seen = true;
                                }
                                ++rowcur;
                                acc.reset();
                            }
                            acc.add(v0.get(q), x0[q]);
                        }
                    }
                    c1 = c2; c2 = cn;
                    v0 = v1; v1 = vn;
#pragma unroll
                    for (int q = 0; q < 4; ++q) x0[q] = x1[q];
                }
            };
            if (!__any_sync(FULL, nst > KSTK)) {
                if (!SKIP || chk) walk(Flag<true>{}, Flag<true>{});
                else walk(Flag<true>{}, Flag<false>{});
                seen = nst > 0;
                if (seen) hpiece = Acc<VT>::piece_at(sbase);
                for (int k2 = 1; k2 < nst; ++k2)
                    if (row0 + k2 < m && guard(err, row0 + k2 >= 0 && k2 < KSTK, G_Y, row0 + k2))
                        y[row0 + k2] = Acc<VT>::piece_at(sbase + k2 * SLOT);
                rowcur = row0 + nst;
            } else {
                walk(Flag<false>{}, Flag<true>{});
            }
            const double a = acc.value();
            tile_combine(seen ? hpiece : a, seen ? a : 0.0, seen, rowcur, rs + total - b00,
                         lane, r_first, r_last, shared, c, y, carry_head, carry_tail, m,
                         carry_row, carry_val, err);
        }
        if (carry_row >= 0 && lane == 0)
            flush_row(carry_row, carry_val, r_first, r_last, shared, c, y, carry_head,
                      carry_tail, m, err);
    }
}

template <typename VT, typename IT>
cudaError_t convert_t(Handle &h, const int *rp, const int *ci, const double *v, const int *ovf,
                      cudaStream_t s) {
    // aux is or-ed together by the chunk's tiles
    cudaError_t err = cudaMemsetAsync(h.meta, 0, sizeof(ChunkHdr) * (size_t)h.nchunks, s);
    if (err != cudaSuccess) return err;
    auto go = [&](auto SG) {
        constexpr int SIGMA = decltype(SG)::value, W = conv_warps<SIGMA>();
        csr5_convert_kernel<SIGMA, VT, IT><<<(unsigned)((h.ntiles + W - 1) / W), W * 32, 0, s>>>(
            rp, ci, v, h.arp, h.m, h.ntiles, h.G, (VT *)h.vals, (IT *)h.cols, h.flags,
            h.tile_ptr, (ChunkHdr *)h.meta, h.colbase, ovf);
        return cudaGetLastError();
    };
    switch (h.sigma) {
        case 8: return go(std::integral_constant<int, 8>());
        case 12: return go(std::integral_constant<int, 12>());
        case 16: return go(std::integral_constant<int, 16>());
        case 24: return go(std::integral_constant<int, 24>());
        case 32: return go(std::integral_constant<int, 32>());
        default: return cudaErrorInvalidValue;
    }
}

template <int SG, typename VT, typename IT, int W>
cudaError_t launch_sg(const Handle &h, const void *x, void *y, cudaStream_t s) {
    using SH = Csr5Shape<W>;
    const long long cap = (long long)h.sm_count * SH::CTAS;
    const unsigned grid = (unsigned)(h.nchunks < cap ? h.nchunks : cap);
    auto go = [&](auto kernel) {
        return launch_product(kernel, grid, SH::WARPS * 32, 0, s, (const ChunkHdr *)h.meta,
                              h.tile_ptr, h.flags, (const VT *)h.vals, (const IT *)h.cols,
                              (const VT *)x, (double *)y, h.carry_head, h.carry_tail,
                              ChunkWalk<SH::WARPS>::over(h.nchunks, grid), h.G, h.m, h.n,
                              guard_word());
    };
    if constexpr (sizeof(VT) == 4) return go(csr5_spmv_f32_kernel<SG, IT, W>);
    else return go(csr5_spmv_kernel<SG, VT, IT, W>);
}

template <typename VT, typename IT, int W>
cudaError_t spmv_t(const Handle &h, const void *x, void *y, cudaStream_t s) {
    switch (h.sigma) {
        case 8: return launch_sg<8, VT, IT, W>(h, x, y, s);
        case 12: return launch_sg<12, VT, IT, W>(h, x, y, s);
        case 16: return launch_sg<16, VT, IT, W>(h, x, y, s);
        case 24: return launch_sg<24, VT, IT, W>(h, x, y, s);
        case 32: return launch_sg<32, VT, IT, W>(h, x, y, s);
        default: return cudaErrorInvalidValue;
    }
}

// Waves of chunks with `warps` resident warps per SM.
long long waves(const Handle &h, int warps) {
    const long long w = (long long)warps * h.sm_count;
    return (h.nchunks + w - 1) / w;
}

}  // namespace

cudaError_t csr5_convert(Handle &h, const int *rp, const int *ci, const double *v, const int *ovf,
                         cudaStream_t s) {
    if (h.ntiles <= 0) return cudaSuccess;
    const bool f32 = h.precision == PAVA_PREC_FP32C, d16 = h.index_mode == PAVA_INDEX_DELTA16;
    if (!f32 && !d16) return convert_t<double, int>(h, rp, ci, v, ovf, s);
    if (!f32 && d16) return convert_t<double, short>(h, rp, ci, v, ovf, s);
    if (f32 && !d16) return convert_t<float, int>(h, rp, ci, v, ovf, s);
    return convert_t<float, short>(h, rp, ci, v, ovf, s);
}

cudaError_t csr5_spmv(const Handle &h, const void *x, void *y, cudaStream_t s) {
    if (h.nchunks <= 0) return cudaSuccess;
    const bool f32 = h.precision == PAVA_PREC_FP32C, d16 = h.index_mode == PAVA_INDEX_DELTA16;
    if (d16 && !f32) return spmv_t<double, short, 24>(h, x, y, s);
    if (d16) {
        // One CTA of 24 warps, but three of 8 where neighbouring nonzeros share lines of x anyway and sigma
        // is 12, or 32 with more than one wave of chunks.  24 / three of 8, us: sigma 12 stencil 110^3
        // 88.0 / 77.1, banded 500,000 rows 35.8 / 30.8; sigma 32 stencil 110^3 58.3 / 53.6, banded
        // 1,048,576 rows 40.0 / 38.8, 60^3 in 1,377 chunks 16.2 / 19.6; sigma 8, 16 and 24 within 3 %,
        // mostly for 24; 256 stacked matrices (scattered) 48.8 / 67.3.
        const bool three = !h.scattered && (h.sigma == 12 || (h.sigma == 32 && waves(h, 24) > 1));
        return three ? spmv_t<float, short, 8>(h, x, y, s) : spmv_t<float, short, 24>(h, x, y, s);
    }
    if (!f32) {
        // 20 warps per SM, but 24 where they save a second or a third wave of chunks: 24 / 20 warps, us,
        // banded 500,000 rows, sigma 24, 3,125 chunks 35.5 / 48.4, dense blocks 300,000 rows, sigma 32,
        // 3,003 chunks 39.4 / 52.0, stencil 110^3, sigma 32, 6,901 chunks 88.6 / 95.7.  Of 38 forms with two
        // waves of 20 warps and one of 24, one was slower with 24 (by 2 %), of 32 with three against two
        // three (by 1 to 3 %), of those with more waves most; with as many waves 20 is 15 % faster.
        const long long w24 = waves(h, 24), w20 = waves(h, 20);
        return w24 <= 2 && w20 > w24 ? spmv_t<double, int, 24>(h, x, y, s)
                                     : spmv_t<double, int, 20>(h, x, y, s);
    }
    // FP32: one CTA of 24, but three of 8 for 32-bit columns that are not scattered (Handle::scattered):
    // stencil 128^3 115 -> 108 us, dense blocks 17 M 41.6 -> 38.6; power law 20 M 88 -> 90
    return h.scattered ? spmv_t<float, int, 24>(h, x, y, s) : spmv_t<float, int, 8>(h, x, y, s);
}

}  // namespace pava
