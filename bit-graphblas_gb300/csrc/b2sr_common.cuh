// Shared definitions of the B2SR library: tile word types, the matrix object,
// launch helpers and error plumbing.  Internal header (the public ABI is
// include/b2sr.h).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <climits>
#include <cstddef>
#include <deque>
#include <mutex>
#include <vector>

#include "../../include/b2sr.h"

namespace b2sr {

// Tile word type per tile size.  T = 4 keeps one byte per tile row with the
// row in the low nibble, as the reference's ToBit4Col does
// (bmv_eval/backend/bsrbmv.cu:33-62).
template <int T> struct TileWord;
template <> struct TileWord<4> { using type = uint8_t; };
template <> struct TileWord<8> { using type = uint8_t; };
template <> struct TileWord<16> { using type = uint16_t; };
template <> struct TileWord<32> { using type = uint32_t; };

template <int T> struct Log2;
template <> struct Log2<4> { static constexpr int value = 2; };
template <> struct Log2<8> { static constexpr int value = 3; };
template <> struct Log2<16> { static constexpr int value = 4; };
template <> struct Log2<32> { static constexpr int value = 5; };

inline int word_bytes(int T) { return T <= 8 ? 1 : T / 8; }
inline bool valid_tile(int T) { return T == 4 || T == 8 || T == 16 || T == 32; }

constexpr unsigned FULL_MASK = 0xffffffffu;

// Merge-path coordinate: `row` row-end items and `tile` tiles consumed.
struct Coord {
    int row;
    int tile;
};

// Launch shape of a merge-path multiply.
struct LaunchShape {
    int threads = 256;
    int items = 8;
    int ctas_per_sm = 0;
    int algorithm = 0;  // 0 auto, 1 merge-path, 2 row-binned
    int gather = 0;     // row-binned x gathers: 0 auto, 1 ld.global, 2 texture, 3 set columns only
    int rhs_block = 0;  // dense-RHS columns per warp pass (FP32 count; 0: narrowest covering k)
    int direction = 0;  // bit-vector variants: 0 pull, 1 auto (push for sparse x), 2 push
};

// Row-binned plan of a matrix (b2sr_rowbin.cu): tasks grouped by bin, the
// long rows' segment bookkeeping, and per-bin task/warp offsets.
struct RowBinPlan {
    int4* d_tasks = nullptr;
    int4* d_long = nullptr;
    int ntasks = 0, nlong = 0, nslots = 0;
    int nlong_short = 0;  // long rows with few slots, listed first in d_long
    bool wide = false;    // T = 32: tasks of 128 tiles, for the staged FP32 form
    int task_off[7] = {0, 0, 0, 0, 0, 0, 0};
    int warp_off[7] = {0, 0, 0, 0, 0, 0, 0};
};

// Row-task SpMM plan (b2sr_spmm_rows.cu): one task per tile-row, long ones cut
// into segments with partial slots; larger tasks first.
struct SpmmRowsPlan {
    int4* d_tasks = nullptr;
    int4* d_long = nullptr;      // (tile-row, first slot, slots, 0)
    int ntasks = 0, nlong = 0, nslots = 0;
    int nnarrow = 0;  // long rows of few slots, listed first in d_long
};

// Per-variant cached launch data of a matrix: the grid and the merge-path
// start coordinate of every CTA (grid + 1 entries, device).
struct LaunchPlan {
    LaunchShape shape;
    int grid = 0;
    Coord* d_starts = nullptr;
};

}  // namespace b2sr

// The opaque handle of the C ABI.
struct b2sr_matrix {
    int nrows = 0, ncols = 0, T = 0;
    int nb = 0, nbc = 0, nt = 0;
    long long nnz = 0;
    int* rowptr = nullptr;
    int* colind = nullptr;
    void* tiles = nullptr;
    bool owns = false;
    int device = 0;
    int num_sms = 0;
    b2sr::LaunchShape shapes[4];
    b2sr::LaunchPlan plans[4];
    b2sr::LaunchPlan spmm_plan;  // chunk starts of the SpMM work queue
    b2sr::RowBinPlan rowbin;     // bin_full_full / multi-frontier row-binned plan
    bool rowbin_ready = false;
    b2sr::RowBinPlan rowbin_bits;  // the bit-vector kernels' plan
    bool rowbin_bits_ready = false;
    b2sr::SpmmRowsPlan spmm_rows;  // row-task SpMM plan
    bool spmm_rows_ready = false;
    // Held while a call launches its kernels: they share the stream's scratch, so
    // those of two host threads on one stream must not come in between.
    std::mutex launch_mu;
    // Per-stream scratch (carries, partials, queue counter), grown on demand
    // and reused: calls on one stream are ordered, so they can share it.
    struct StreamScratch {
        cudaStream_t stream;
        void* ptr;
        size_t bytes;
    };
    std::mutex scratch_mu;
    std::vector<StreamScratch> scratch;
    // Per-stream counters of the row-task SpMM kernel's work queue: zeroed when
    // allocated, left zeroed by every launch, and used by nothing else.
    std::vector<StreamScratch> spmm_state;
    // Auto direction outside stream captures: the device's last decision per
    // bit-vector kind (0 none yet, 1 push, 2 pull) in mapped host memory, read
    // by the next call as a hint; and per stream the counters of both sides,
    // zeroed when allocated and left zeroed by every call.
    int* auto_hint = nullptr;
    std::vector<StreamScratch> auto_state;
    // Buffers replaced by larger or rebuilt ones.  A CUDA graph captured
    // earlier may still hold their addresses, so they are freed only when
    // the matrix is freed.
    std::vector<void*> retired;
    b2sr_matrix* transpose = nullptr;
};

namespace b2sr {

// ---- status / allocation helpers (b2sr_api.cu) --------------------------------
void set_cuda_error(cudaError_t e);
void* dev_alloc(size_t bytes);
void* array_alloc(size_t bytes);  // for a matrix's arrays: a block of cudaMalloc (no hook); freed by dev_free
void dev_free(void* p);
void set_launch_count(int n);
void add_launch_count(int n);
// Kernel timer: records an event on `s` before (begin = true) or after the
// dominant kernel of a multiply while b2sr_kernel_timer_start armed it.
void kernel_timer_mark(cudaStream_t s, bool begin);

#define B2SR_CUDA_TRY(expr)                                   \
    do {                                                      \
        cudaError_t _e = (expr);                              \
        if (_e != cudaSuccess) {                              \
            ::b2sr::set_cuda_error(_e);                       \
            return B2SR_ERR_CUDA;                             \
        }                                                     \
    } while (0)

#define B2SR_LAUNCH_CHECK()                                   \
    do {                                                      \
        cudaError_t _e = cudaGetLastError();                  \
        if (_e != cudaSuccess) {                              \
            ::b2sr::set_cuda_error(_e);                       \
            return B2SR_ERR_CUDA;                             \
        }                                                     \
    } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Launch `kernel` behind the previous kernel on `s` with programmatic
// dependent launch: its blocks may be scheduled while that grid drains and
// wait in griddep_wait() until it has completed and its writes are visible.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), unsigned grid, unsigned block, cudaStream_t s,
                                    Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- packing (b2sr_pack.cu) ---------------------------------------------------
// CSR -> B2SR in two passes with shared scratch.  count() validates the CSR,
// writes browptr (nb + 1) and returns the number of tiles and of distinct
// entries; it synchronizes the stream.  B2SR_ERR_INVALID_CSR: nothing is
// packed.  fill() then writes colind (nt) and every tile word (nt * T), on the
// same stream.  The scratch is freed, after the stream has drained, with the
// object.
class PackJob {
public:
    ~PackJob();
    b2sr_status count(const int* rowptr, const int* colind, int nrows, int ncols, int nnz, int T, int* browptr, int* nt,
                      long long* set_bits, cudaStream_t s);
    b2sr_status fill(int* bcolind, void* tiles);
    struct Layout;

private:
    void* scratch = nullptr;
    cudaStream_t s = nullptr;
    int T = 0, nb = 0;
    long long max_chunks = 0, n_entries = 0;
    bool wide = false;  // 64-bit sort keys
};
// In-place exclusive scan of d_vals[0..n) with the total written to d_vals[n]
// (d_vals has n + 1 entries), asynchronous; scratch of exclusive_scan_scratch(n)
// bytes.  *d_err is set to 1 if the total overflows int32, else left alone.
// Returns the kernels that it launched.
size_t exclusive_scan_scratch(long long n);
int exclusive_scan_async(int* d_vals, int n, int* d_err, void* scratch, cudaStream_t s);
b2sr_status launch_pack_vec_bits(const float* x, int n, int T, void* bits, cudaStream_t s);
b2sr_status launch_unpack_vec_bits(const void* bits, int n, int T, float* out, cudaStream_t s);
// Set bits of a B2SR matrix (for the descriptor); result in *d_count (int64).
b2sr_status launch_count_bits(const void* tiles, long long nwords, int T,
                              unsigned long long* d_count, cudaStream_t s);

// ---- transpose (b2sr_transpose.cu) ---------------------------------------------
// A^T's rowptr (nbc + 1 entries), colind and tiles (nt each) from A's, on the
// device (stable radix sort of the tiles by tile-column, then a bit transpose
// of every tile).  Synchronizes `s`.  B2SR_ERR_INVALID_VALUE if a tile-column
// lies outside [0, nbc).
b2sr_status launch_transpose(const int* rowptr, const int* colind, const void* tiles, int nb, int nbc, int nt, int T,
                             int* rowptr_t, int* colind_t, void* tiles_t, cudaStream_t s);

// ---- task lists (b2sr_plan.cu) -----------------------------------------------------
constexpr int PLAN_CLASSES = 64;
// How tile-rows become tasks.  A tile-row of more than `seg` tiles is cut into
// segments: of seg tiles (BINS), or near-equal ones (the others), which with
// row_bits also hold at most about seg_bits set bits each.  Tasks are listed by
// class, tile-rows ascending inside a class:
//   BINS    nbins bins by tile count (bin b: up to unit << b tiles), the last
//           bin first
//   TWO     tasks of at least a quarter of seg, then the rest
//   BITS    most set bits first, in two classes per octave
// Long rows of at most narrow_slots slots are listed before the others.
struct PlanRule {
    enum Kind { BINS, TWO, BITS } kind;
    int seg;
    int classes;
    int unit = 0, nbins = 0, narrow_slots = 0;
    int whole = 0, whole_bits = 0;  // tile-rows with no more tiles / set bits than this are not cut
    const long long* row_bits = nullptr;
    long long seg_bits = 0;
};
struct PlanBounds {
    long long tasks, longs, slots;
};
struct PlanOut {
    int4* tasks;     // (tile-row, first tile, end tile, slot or -1)
    int4* longs;     // (tile-row, first slot, slots, 0)
    int* info;
    int cap_tasks, cap_long;
};
struct PlanTotals {
    int tasks = 0, longs = 0, narrow = 0, slots = 0;
    int first[PLAN_CLASSES + 1] = {0};  // first task of every class, and their number
};
// Array sizes that hold the plan of a matrix with nt tiles and `bits` set bits.
PlanBounds plan_bounds(const PlanRule& r, int nb, long long nt, long long bits);
// Fills the arrays (of those sizes).  Synchronizes `s`, on failure too.
b2sr_status build_plan(const PlanRule& rule, const int* rowptr, int nb, const PlanBounds& cap, int4* tasks, int4* longs,
                       PlanTotals* totals, cudaStream_t s);

// ---- multiply (b2sr_spmv.cu) --------------------------------------------------
struct MatView {
    const int* rowptr;
    const int* colind;
    const void* tiles;
    int nb;
    int ncols;  // x length for bin_full_full (segments past it are read element-wise)
    int T;
};

// Merge-path start coordinates of `grid` equal shares of the nb + nt items.
// nt is read from rowptr[nb] on the device.
b2sr_status launch_partition(const MatView& A, int grid, Coord* d_starts, cudaStream_t s);

// Largest grid the merge-path multiply of (variant, T, shape) uses on this device.
int merge_grid(b2sr_variant v, int T, const LaunchShape& shape, int num_sms);
// Bytes of scratch the merge-path multiply needs for `grid` CTAs.
size_t carry_bytes(b2sr_variant v, int T, int grid);

// One multiply: main merge-path kernel + carry fix-up.  `carries` is scratch of
// carry_bytes(v, T, grid) bytes.  `mask` is used by the masked variant only.
b2sr_status launch_spmv(b2sr_variant v, const MatView& A, const LaunchShape& shape, int grid,
                        const Coord* d_starts, const void* x, void* y, const void* mask,
                        int accumulate, void* carries, cudaStream_t s);

// ---- dense right-hand sides (b2sr_spmm.cu) ---------------------------------------
constexpr int SPMM_CHUNK_ITEMS = 1024;
template <typename V>
b2sr_status spmm_launch(const MatView& A, const V* X, long long ldx, V* Y, long long ldy, int k,
                        int accumulate, const Coord* starts, int nchunks, void* scratch, int grid_warps,
                        cudaStream_t s);
size_t spmm_scratch_bytes(int T, int elem_bytes, int nchunks, int k);
int spmm_grid_warps(int num_sms);

// ---- row-task dense right-hand sides (b2sr_spmm_rows.cu) --------------------------
// Synchronizes `s`.
b2sr_status spmm_rows_plan_create(const int* d_rowptr, const void* d_tiles, int nb, int nt, long long nnz, int T,
                                  int num_sms, SpmmRowsPlan* out, cudaStream_t s);
void spmm_rows_plan_free(SpmmRowsPlan* p);
size_t spmm_rows_scratch_bytes(const SpmmRowsPlan& p, int T, int elem_bytes, int k);
size_t spmm_rows_state_bytes();
template <typename V>
b2sr_status spmm_rows_launch(const MatView& A, const SpmmRowsPlan& p, const V* X, long long ldx, V* Y,
                             long long ldy, int k, int rhs_block, int accumulate, void* scratch, int* state,
                             int num_sms, cudaStream_t s);

// ---- row-binned bin_full_full (b2sr_rowbin.cu) ------------------------------------
// bits: the plan of the bit-vector kernels (longer long-row tasks at T = 4).
b2sr_status rowbin_plan_create(const int* d_rowptr, int nb, int nt, int T, bool bits, RowBinPlan* out, cudaStream_t s);
void rowbin_plan_free(RowBinPlan* p);
size_t rowbin_scratch_bytes(const RowBinPlan& p, int T, int value_bytes);
// Bit-vector variants on the same plan: kind 0 bin_bin_bin, 1 masked, 2 int32
// counts, 3 FP32 counts (bin_bin_full).
size_t rowbin_bits_scratch_bytes(const RowBinPlan& p, int T);
// The push side of an auto-direction product (b2sr_push.cu) as the pull
// kernels see it: they return at once when the push took the product.
struct PushLink {
    int* ctl = nullptr;  // launch_push's counters; null: pull only
    long long nt = 0;
    int pct = 0;  // push when the active tiles are below pct% of nt
    bool gate = false;  // launch the pull from the device, only when chosen, and zero ctl (not in a capture)
};
// Beside a pull: the tiles under x's non-zero words, counted by warps of the
// pull kernel, and from the last of them the direction for the next call (1
// push, 2 pull) into *hint.  state: 2 ints, zeroed, left zeroed.
struct DirectionCount {
    const int* t_rowptr = nullptr;  // A^T's (null: do not count)
    int* state = nullptr;
    int* hint = nullptr;
    long long nt = 0;
    int pct = 0;
};
// timed: kernel timer marks around the main kernel.
b2sr_status rowbin_bits(const RowBinPlan& p, const MatView& A, int kind, const void* x, void* y, const void* mask,
                        int accumulate, void* partials, const PushLink& link, const DirectionCount& count, bool timed,
                        cudaStream_t s);
// sparse_cols: load x only for each tile's set columns (launch option gather = 3,
// the default at T >= 16) instead of the tile-column's whole x segment.
b2sr_status rowbin_spmv(const RowBinPlan& p, const MatView& A, const float* x, float* y, int accumulate,
                        void* scratch, cudaTextureObject_t xtex, bool sparse_cols, cudaStream_t s);
b2sr_status rowbin_multi_bits(const RowBinPlan& p, const MatView& A, const void* x, void* y, const void* mask,
                              int word_bits, int accumulate, void* scratch, cudaTextureObject_t xtex,
                              cudaStream_t s);
// ---- direction-optimised bit-vector products (b2sr_push.cu) -------------------------
// The push form visits only the tile-columns whose x word is non-zero, through
// the transpose At; ctl[1] counts their tiles on the device.  Auto mode takes
// it below push_percent(T, counts)% of nt: about the tile share at which the push
// and the row-binned pull take equal time on R-MAT scale 20 (GB300; push time
// is close to linear in that share).  Where that is depends on how full the
// non-zero x words are, since a push pays an atomic per tile (bits) or per row
// (counts) that it changes: with all bits set 6.6 / 9.6 / 27 / 41% and with one
// bit 39 / 72 / 85+ / 41% for bits at T = 4 / 8 / 16 / 32, 9 / 12 / 12 / 8% and
// 33 / 17 / 12 / 7% for counts; the lines lie between the two.  (One rule of
// 18 / 27 / 45 / 85% for both kinds let counts at 30% of the tiles push in 265
// us at T = 16 and 616 us at T = 32, where the pull takes 115 and 208.)
inline int push_percent(int T, bool counts) {
    return T == 4 ? 18 : T == 8 ? (counts ? 14 : 27) : T == 16 ? (counts ? 12 : 45) : (counts ? 8 : 41);
}
__device__ __forceinline__ bool push_chosen(const int* ctl, int mode, long long nt, int pct) {
    return mode == 2 || (long long)ctl[1] * 100 < nt * pct;
}
// Scratch bytes of launch_push: counters and the work list.
size_t push_scratch_bytes(int nbc, long long nt);
// mode 1 (auto) or 2 (always push); kind as rowbin_bits.  Zeroes y (y_bytes)
// first unless accumulate.  ctl: two zeroed ints, or null for counters in the
// scratch, zeroed first.  Fills *link (counters, threshold) for the pull kernels
// launched after it.
b2sr_status launch_push(const MatView& At, int kind, int mode, const void* x, void* y, const void* mask,
                        int accumulate, size_t y_bytes, long long nt, void* scratch, int* ctl, int num_sms,
                        PushLink* link, int* hint, cudaStream_t s);
// Cached texture object (uint4 texels) over [ptr, ptr + bytes), or 0 when the
// buffer cannot back one (alignment, size).
cudaTextureObject_t vector_texture(const void* ptr, size_t bytes);

}  // namespace b2sr
