// Internal declarations shared by the engine's translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include <string>

#include "../../include/pava_gpu.h"
#include "pava_common.cuh"

namespace pava {

// Per-chunk metadata of the GPU CVR form (128 bytes; one chunk = 32 lanes x S steps).
// The row phase needs only the header; the rest describes the chunk's tail, where the rows
// still open when the chunk ran out of rows are spread evenly over the 32 lanes.
struct CvrMeta {
    ChunkHdr h;
    int i_t;       // first tail step (== S when the chunk has no tail)
    int ntail;     // tail slots (rows still open at i_t, in row order), <= 64
    int n_inprog;  // slots [0, n_inprog) hold rows a lane was working on at i_t
    int next_g;    // slot n_inprog + j holds row r_first + next_g + j
    unsigned cont; // bit k: lane k's first tail element continues lane k-1's last row
    unsigned pad[3];
    unsigned char park[32];        // slot of lane k's row in progress at i_t, 0xff if none
    unsigned char first_slot[32];  // slot of lane k's first tail element
    unsigned pad2[4];
};
static_assert(sizeof(CvrMeta) == 128, "CvrMeta layout");

// Per-slice descriptor of the SELL form (32 rows; 4-step blocks of 128 elements).
struct SellSlice {
    int off;         // first element of the slice in the value and column streams
    int nblk;        // 4-step blocks: the slice's longest row, rounded up to 4, over 4
    int colbase;     // DELTA16: base column of the 16-bit offsets
    unsigned flags;  // bit 0: some row of the slice is padded (padding reads no x); bits 1..31:
                     // the first block holding padding (the shortest row / 4)
};
static_assert(sizeof(SellSlice) == 16, "SellSlice layout");

// Engine handle (behind the opaque pava_handle of the C ABI).
struct Handle {
    int format = 0, precision = 0, index_mode = 0;
    int m = 0, n = 0, nnz = 0, n_empty = 0;
    long long n_aug = 0;     // elements after giving every empty row one zero element
    long long nchunks = 0;   // warp chunks
    long long L = 0;         // elements per chunk (padded space = nchunks * L)
    int S = 0;               // CVR: steps per chunk
    int sigma = 0, G = 0;    // CSR5: elements per lane per tile, tiles per chunk
    long long ntiles = 0;
    int scattered = 0;       // CVR, CSR5: neighbouring nonzeros rarely share lines of x
    int longest = 0;         // plain CSR: elements of the longest row
    int lanes_per_row = 0;   // plain CSR: lanes per row group (GL)
    int col_lanes = 1;       //   lanes across the right-hand sides (KC)
    int cols_per_lane = 1;   //   right-hand sides per lane (KPL)
    int rows_per_tile = 0;   //   rows per warp tile of the persistent launch (TR), or per
                             //   CTA tile with x_window
    int x_window = 0;        //   stage each CTA tile's window of X in shared memory
    int device = 0, sm_count = 0;

    int *arp = nullptr;            // augmented row pointer, m + 2 entries (row m = padding)
    void *vals = nullptr;          // format value stream
    void *cols = nullptr;          // format column stream
    unsigned *flags = nullptr;     // CVR row-end bits / CSR5 row-start descriptors
    void *meta = nullptr;          // per-chunk metadata (CvrMeta or ChunkHdr)
    size_t meta_stride = 0;
    int *tile_ptr = nullptr;       // CSR5 tile -> first row
    int *colbase = nullptr;        // DELTA16: per-chunk base column of the 16-bit offsets
    double *carry_head = nullptr;  // per-chunk partial of a first row shared with the left
    double *carry_tail = nullptr;  // per-chunk partial of a last row shared with the right
    int *rp = nullptr, *ci = nullptr;  // plain CSR form
    void *v = nullptr;                 //   values: double, or float for FP32C

    double convert_ms = 0.0;
    size_t device_bytes = 0;
};

// Device memory of handles, conversions and their temporaries: a memory pool per device and
// context that keeps at most POOL_KEEP bytes of what was freed, so that converting a new matrix
// does not pay the driver for its buffers each time.  Large blocks that it would not keep come from
// cudaMalloc (k_support.cu); freeing one waits for the device.  All calls are thread-safe; memory is
// ordered on the stream it is allocated and freed on.
constexpr size_t POOL_KEEP = (size_t)1 << 30;
cudaError_t pool_malloc(void **p, size_t bytes, cudaStream_t s);
template <typename T> cudaError_t pool_malloc(T **p, size_t count, cudaStream_t s) {
    return pool_malloc((void **)p, sizeof(T) * (count ? count : 1), s);
}
// cudaMalloc, once more after giving back what the pool holds unused.
cudaError_t plain_malloc(void **p, size_t bytes);
// Frees memory whose last use is ordered before this point of s (NULL pointers are skipped).
void pool_free(void *p, cudaStream_t s);
// Frees memory that work on any stream may still use: waits for the device first, as cudaFree
// does, and like it leaves a thread-local or relaxed capture elsewhere whole.  Where the wait is not
// possible (a global capture) the memory is kept until a later call can wait.
void pool_free_synced(void *const *ps, int count);
// Bytes the pool holds, and giving back what is unused above `keep`.
size_t pool_reserved();
void pool_trim(size_t keep);
// The same after waiting for the device, with what waits to be freed.
cudaError_t pool_release(size_t keep);

// Launches a product kernel as a programmatic dependent of the kernel before it in the stream.
// All product kernels let their dependents launch early (pdl_trigger: CVR, CSR5, SELL and the fixup at
// once, the row groups of plain CSR after their own wait) and call pdl_wait before they read x or
// write anything, so consecutive products overlap one's launch and first reads of the format, which
// only conversion writes, with the end of the other; behind any other kernel the launch waits as an
// ordinary one does.  x is read by ordinary loads: the kernel before may still be writing it.  512 x 512 Laplacian, CVR (SpMV and fixup): 12.3 ->
// 10.3 us a product in a loop; 128^3 stencil, SELL FP32C: 74.5 -> 71.6 us.
template <typename... KArgs, typename... Args>
cudaError_t launch_product(void (*kernel)(KArgs...), unsigned grid, unsigned threads,
                           size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Sets the message pava_last_error() returns on this thread.
void set_last_error(const std::string &msg);

// Device address of the bounds-check error word (three 64-bit words) on the current device in
// builds with PAVA_BOUNDS_CHECK; nullptr in ordinary builds, whose kernels never test it.
unsigned long long *guard_word();

// Device address of the bounded-wait word (two 64-bit words: waits that gave up, and the first
// one's site + 1) on the current device; in every build.  nullptr when it cannot be resolved.
unsigned long long *wait_word();

// CSR5 tiles per chunk.  The persistent grid keeps `warps` warps resident (24 per SM; FP64 on 32-bit
// columns runs 20 where that takes as many waves, and these rules count 24 for it too unless its
// columns are scattered); each takes chunks in turn, so a chunk count just above a multiple of `warps` leaves a last wave that
// few warps run.
// Default: 4 tiles per chunk, fewer when that leaves fewer chunks than warps.
inline int csr5_default_tiles(long long tiles, long long warps) {
    return tiles >= 4 * warps ? 4 : (tiles >= 2 * warps ? 2 : 1);
}
// Wave-balanced: the G in 1..8 with the fewest tiles on a warp's critical path,
// ceil(tiles / (G * warps)) * G; the largest G among equals.
inline int csr5_wave_tiles(long long tiles, long long warps) {
    int best = 1;
    long long best_t = -1;
    for (int g = 1; g <= 8; ++g) {
        const long long t = (tiles + g * warps - 1) / (g * warps) * g;
        if (best_t < 0 || t <= best_t) { best_t = t; best = g; }
    }
    return best;
}

// Scattered columns, FP64: the G in 1..8 with the smallest cost of a warp's chunks, a chunk costing its
// tiles and a fifth of a tile for its header, carries and start.  Sigma 16, us a product in a
// loop at 1 / 2 / 3 / 4 / 6 / 8 tiles per chunk: 20 M nonzeros (13.5 tiles per resident warp)
// 103 / 100 / 105 / 110 / 115 / 111; 66 M (43.5) 310 / 302 / 304 / 297 / 312 / 321.
inline int csr5_scattered_tiles(long long tiles, long long warps) {
    int best = 1;
    long long best_t = -1;
    for (int g = 1; g <= 8; ++g) {
        const long long t = (tiles + g * warps - 1) / (g * warps) * (5 * g + 1);
        if (best_t < 0 || t <= best_t) { best_t = t; best = g; }
    }
    return best;
}

// Kernel launchers (stream-ordered; return cudaGetLastError()).
// d_err[0]: violations; want_longest: d_err[1] = the length of the longest row, where the row pointer is
// sound.
cudaError_t launch_validate(const int *rp, const int *ci, int m, int n, int nnz, int *d_err,
                            bool want_longest, cudaStream_t s);
// arp[0..m]; arp[m + 1], the padded total, is the caller's (set_int).
cudaError_t build_augmented_rowptr(const int *rp, int m, int *arp, int *d_nempty, cudaStream_t s);
cudaError_t set_int(int *p, int v, cudaStream_t s);
// rows[t] = row of augmented element t*T, t in [0, count) (arp complete).
cudaError_t chunk_rows(const int *arp, int m, long long T, long long count, int *rows,
                       cudaStream_t s);

// DELTA16 base column of every warp chunk (h.colbase): the midpoint of the chunk's smallest
// and largest column; *ovf is set to 1 when a chunk's columns span too much for 16-bit offsets.
// first[c * stride]: row of chunk c's first element.
cudaError_t chunk_colbase(const Handle &h, const int *rp, const int *ci, const int *first,
                          int stride, int *ovf, cudaStream_t s);

// Lines of x (128 bytes of FP64) that LINE_WINDOWS samples of LINE_WINDOW consecutive nonzeros touch,
// summed into *lines (device, zeroed here): a matrix whose samples reuse few lines is scattered.
constexpr int LINE_WINDOW = 1024, LINE_WINDOWS = 32;
cudaError_t sample_lines(const int *ci, int nnz, int *lines, cudaStream_t s);

// Conversions.  With 16-bit offsets they do nothing when *ovf (device) is set.  first: CVR, the
// row of each chunk's first element; CSR5, h.tile_ptr is complete.
cudaError_t cvr_convert(Handle &h, const int *rp, const int *ci, const double *v, const int *first,
                        const int *ovf, cudaStream_t s);
cudaError_t cvr_spmv(const Handle &h, const void *x, void *y, cudaStream_t s);

cudaError_t csr5_convert(Handle &h, const int *rp, const int *ci, const double *v, const int *ovf,
                         cudaStream_t s);
cudaError_t csr5_spmv(const Handle &h, const void *x, void *y, cudaStream_t s);

// fresh: the kernel before it in the stream wrote the headers as well as the carries.
cudaError_t carry_fixup(const Handle &h, void *y, cudaStream_t s, bool fresh = false);

// SELL: sell_plan fills the slice descriptors (h.meta, h.nchunks slices) except their offsets
// and writes the exclusive scan of the slices' block counts to d_blk_off[0..nslices], the total
// to d_res[0], and 1 to d_res[1] when want_base and a slice's columns span too much for 16-bit
// offsets (0 otherwise); sell_fill writes the padded streams and the offsets.
cudaError_t sell_plan(Handle &h, const int *rp, const int *ci, bool want_base, int *d_blk_off,
                      int *d_res, cudaStream_t s);
cudaError_t sell_fill(Handle &h, const int *rp, const int *ci, const double *v,
                      const int *d_blk_off, cudaStream_t s);
cudaError_t sell_spmv(const Handle &h, const void *x, void *y, cudaStream_t s);
// SELL SpMM, Y = A X with X row-major n x k; leading dimensions ldx, ldy in elements.  Lanes per
// row (h.lanes_per_row): 4 (k <= 32), 8 (k <= 64) or 16 (k <= 64); 0 = the engine's choice.
// sell_spmm_lanes gives the lanes it uses for k, 0 when the handle's choice cannot serve k
// (sell_spmm then returns cudaErrorInvalidValue).
constexpr int SELL_SPMM_MAX_K = 64;
// The engine's choice (lanes_per_row 0): four lanes, whose warp reads eight rows' X at once, while the
// sums fit its registers: FP32 up to k = 24, odd k up to 28; FP64 up to k = 12, or 16 where rows are
// short (under 16 elements) or, for even k, long (over 32).  FP64 in a loop, us, 4 / 8 lanes: stencil
// 60^3 k = 13 70 / 63, k = 16 58 / 46, banded 500,000 rows k = 15 167 / 119, dense blocks k = 12 75 / 77,
// 300,000 rows on 16-bit columns k = 16 103 / 122 (32-bit 104 / 108), Laplacian 900^2 k = 13 75 / 93; FP32 banded k = 20
// 116 / 160, k = 27 157 / 186, stencil k = 32 101 / 78.
inline int sell_spmm_lanes(int lanes_per_row, int k, bool f32 = false, bool long_rows = false) {
    const int four = f32 ? (k % 2 ? 28 : 24) : long_rows ? 12 : 16;
    const int g = lanes_per_row ? lanes_per_row : (k <= four ? 4 : 8);
    if (g == 4) return k <= 32 ? 4 : 0;
    if (g == 8 || g == 16) return k <= SELL_SPMM_MAX_K ? g : 0;
    return 0;
}
cudaError_t sell_spmm(const Handle &h, const void *X, long long ldx, void *Y, long long ldy,
                      int k, cudaStream_t s);

// Plain CSR row-group kernel: y = A x, and Y = A X with X row-major n x k (leading
// dimensions ldx, ldy in elements).
cudaError_t csr_spmv(const Handle &h, const void *x, void *y, cudaStream_t s);
cudaError_t csr_spmm(const Handle &h, const void *X, long long ldx, void *Y, long long ldy,
                     int k, cudaStream_t s);
// SpMM with the rows staged per warp (k_csr_spmm.cu), k in 1 .. 128, in its own shape for k (lanes = 0)
// or a named one; csr_spmm runs it too for the shapes csr_staged_shape accepts.
cudaError_t csr_spmm_staged(const Handle &h, const void *X, long long ldx, void *Y, long long ldy,
                            int k, int lanes, int cols, cudaStream_t s);
bool csr_staged_shape(const Handle &shape, int k);
cudaError_t narrow_to_float(const double *src, float *dst, long long n, cudaStream_t s);

}  // namespace pava
