// Row-task B2SR x dense multiply: Y = A . X with X [ncols, k] and Y [nb*T, k]
// row-major, FP32 or FP64 (bin_full_full on feature blocks; the adjoint
// dX = A^T . dY is the same kernel on the transposed B2SR).  A work item is one
// group of 4 rows of a task, T/4 items per task and column block.
//
// Plan (once per matrix, b2sr_plan.cu): one task per tile-row.  A tile-row of
// more than rows_whole_tiles() tiles that is longer than spmm_rows_seg() tiles (a
// share of one resident warp's part of all the tiles), or at T >= 8 one of more
// than ROWS_WHOLE_BITS set bits and more than such a share of them, is cut into
// near-equal segments whose partial rows go to slots, which a second kernel adds
// in segment order.  Warps take
// (column block, task, row group) work items from a device queue (an atomic
// counter); long tasks are handed out first, so the queue ends on short ones
// (R-MAT hubs sit all over the vertex range, and in row order the last items
// could be the longest).  The queue's counters live in a zeroed
// per-(matrix, stream) state buffer that the kernel's last warp leaves zeroed
// again, so no launch needs a memset.
//
// Inside a task a warp walks its tiles 32 at a time, one tile per lane.  The
// lanes' set bits are appended to 4 item lists in shared memory, one per row r
// of the group, in tile then column order: the positions come from one warp
// scan of the per-row bit counts (packed several rows to a word).  The lists
// grow over many 32-tile steps (an R-MAT step holds ~8 items per row) and are
// consumed only when one would overflow or the task ends, so a row's items
// come in long runs.  The warp walks each list eight items per lane at a time,
// every lane loading its VEC columns of the eight X rows before adding them
// into acc[r] (a compile-time index), so eight coalesced row loads per lane
// are in flight; the rest of a list goes four (predicated) at a time.  The
// summation order is fixed, so the result does not depend on scheduling.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "b2sr_spmv_impl.cuh"

namespace b2sr {

namespace {

constexpr int ROWS_WARPS = 8;    // warps per block

template <typename V, int VEC> struct RowsVec;
template <> struct RowsVec<float, 1> { using type = float; };
template <> struct RowsVec<float, 2> { using type = float2; };
template <> struct RowsVec<float, 4> { using type = float4; };
template <> struct RowsVec<double, 1> { using type = double; };
template <> struct RowsVec<double, 2> { using type = double2; };

// A lane's VEC columns of an X or Y row.  FULL: neighbouring columns, one
// vector load (all VEC valid and aligned).  Otherwise columns STR apart (STR
// lanes share the row), a coalesced scalar load each, the first nvalid of them
// inside the row: widths and strides that are no multiple of 16 bytes.  SLOTS:
// rows that the launch before this one wrote, by ordinary loads: that launch may
// still run when this kernel starts, and the read-only path (and any load that
// the compiler need not keep behind the wait) is for data that does not change
// while the kernel runs.
template <typename V, int VEC, bool FULL, int STR, bool SLOTS = false>
__device__ __forceinline__ void rows_load(V (&out)[VEC], const V* p, int nvalid) {
    if constexpr (FULL) {
        using VT = typename RowsVec<V, VEC>::type;
        const VT* q = reinterpret_cast<const VT*>(p);
        const VT v = SLOTS ? *q : __ldg(q);
        const V* e = reinterpret_cast<const V*>(&v);
#pragma unroll
        for (int i = 0; i < VEC; ++i) out[i] = e[i];
    } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i) out[i] = i < nvalid ? (SLOTS ? p[i * STR] : __ldg(p + i * STR)) : V(0);
    }
}

// acc += v element-wise; FP32 pairs as one packed two-lane add (add.rn.f32x2:
// two IEEE round-to-nearest adds, bitwise the same as the scalar ones).
template <typename V, int VEC>
__device__ __forceinline__ void rows_add(V (&acc)[VEC], const V (&v)[VEC]) {
    if constexpr (std::is_same<V, float>::value && VEC % 2 == 0) {
#pragma unroll
        for (int i = 0; i < VEC; i += 2) {
            unsigned long long x, y;
            asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(acc[i]), "f"(acc[i + 1]));
            asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(v[i]), "f"(v[i + 1]));
            asm("add.rn.f32x2 %0, %0, %1;" : "+l"(x) : "l"(y));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[i]), "=f"(acc[i + 1]) : "l"(x));
        }
    } else {
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[e] += v[e];
    }
}

// acc += the N loaded rows: one after the other (FULL), or pairwise among
// themselves first (the scalar layouts, which have one X row per load where
// the vector ones have two partial sums per row at the same width).
template <bool FULL, int N, typename V, int VEC>
__device__ __forceinline__ void rows_add_all(V (&acc)[VEC], V (&v)[N][VEC]) {
    if constexpr (!FULL) {
#pragma unroll
        for (int o = 1; o < N; o <<= 1)
#pragma unroll
            for (int u = 0; u < N; u += 2 * o) rows_add<V, VEC>(v[u], v[u + o]);
        rows_add<V, VEC>(acc, v[0]);
    } else {
#pragma unroll
        for (int u = 0; u < N; ++u) rows_add<V, VEC>(acc, v[u]);
    }
}

// STREAM: evict-first, for rows that nothing reads soon.
template <typename V, int VEC, bool FULL, int STR, bool STREAM = false>
__device__ __forceinline__ void rows_store(V* p, const V (&v)[VEC], int nvalid, bool accumulate) {
    if constexpr (FULL) {
        using VT = typename RowsVec<V, VEC>::type;
        VT* q = reinterpret_cast<VT*>(p);
        VT o;
        V* e = reinterpret_cast<V*>(&o);
        if (accumulate) {
            const VT old = *q;
            const V* oe = reinterpret_cast<const V*>(&old);
#pragma unroll
            for (int i = 0; i < VEC; ++i) e[i] = oe[i] + v[i];
        } else {
#pragma unroll
            for (int i = 0; i < VEC; ++i) e[i] = v[i];
        }
        if (STREAM) __stcs(q, o);
        else *q = o;
    } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i)
            if (i < nvalid) p[i * STR] = accumulate ? p[i * STR] + v[i] : v[i];
    }
}

// Rows of a tile-row one task covers: 4, so G = T/4 work items per tile-row.
// A task's accumulators (4 rows x 16 bytes of columns a lane) and loads in
// flight then fit 64 registers at every T, four blocks per SM, and an item's
// rows are few enough for long runs.  With 8 rows (whole tile-rows at T = 8,
// two blocks per SM) each tile was read half as often, but short rows left
// the loads of 16 warps waiting: R-MAT scale 18, k = 64 / 128: T = 8 228 / 407
// -> 197 / 291 us, T = 16 292 / 484 -> 265 / 350 us, T = 32 372 / 544 -> 361 /
// 449 us; 100,003-vertex ER graph of degree 11, k = 50: T = 8 64 -> 46 us,
// T = 32 146 -> 107 us.
constexpr int ROWS_R = 4;
constexpr int ROWS_BLOCKS = 4;   // blocks of ROWS_WARPS warps per SM the register budget is written for
constexpr int ROWS_CAP = 256;    // item capacity of each tile row's region in shared memory; a step adds <= 32*T
constexpr int ROWS_BATCH = 8;    // X-row loads in flight per lane
constexpr int ROWS_REST = 4;     // and of the rest of a list

// Packed per-row bit counts: FIELD bits per row (a row total over 32 lanes
// is at most 32*T: 128 fits 8 bits for T = 4; 256, 512 and 1024 take 16).
template <int T> struct RowsPack {
    static constexpr int FIELD = T == 4 ? 8 : 16;
    static constexpr int PER = 32 / FIELD;        // rows per 32-bit pack
    static constexpr int NP = ROWS_R / PER;    // packs
    static constexpr uint32_t MASK = (1u << FIELD) - 1;
};

// The rows of lane's tile that its task covers: rows 4*g .. 4*g+3 of group g,
// T/8 words read with one load.  bits(r): row r's word, bit T-1-c = column c.
template <int T> struct RowsWord {
    static constexpr int NW = T <= 8 ? 1 : T / 8;
    uint32_t w[NW] = {};
    __device__ __forceinline__ void load(const void* tiles, int j, int g) {
        // byte offset (j*T/4 + g) * NW*4: a multiple of the load's size
        const size_t at = (size_t)j * (T / ROWS_R) + g;
        if constexpr (NW == 4) {
            const uint4 v = __ldg(static_cast<const uint4*>(tiles) + at);
            w[0] = v.x;
            w[1] = v.y;
            w[2] = v.z;
            w[3] = v.w;
        } else if constexpr (NW == 2) {
            const uint2 v = __ldg(static_cast<const uint2*>(tiles) + at);
            w[0] = v.x;
            w[1] = v.y;
        } else {
            w[0] = __ldg(static_cast<const uint32_t*>(tiles) + at);
        }
    }
    __device__ __forceinline__ uint32_t bits(int r) const {
        if constexpr (T == 32) return w[r];
        else if constexpr (T == 16) return (w[r >> 1] >> (16 * (r & 1))) & 0xffffu;
        else return (w[0] >> (8 * r)) & ((1u << T) - 1u);
    }
};

}  // namespace

template <typename V>
struct SpmmRowsArgs {
    const int* colind;
    const void* tiles;
    const V* X;
    V* Y;
    long long ldx, ldy;
    int k;    // total columns
    int ncb;  // column blocks of (32 / IPW) * VEC columns
    const int4* tasks;  // (tile-row, first tile, end tile, slot or -1)
    int ntasks;
    int* state;   // [0] queue counter, [1] warps done
    const int4* long_rows;  // (tile-row, first slot, slots, 0)
    V* partials;  // slot x T x k
    int accumulate;
};

// First column of a lane in column block cb, and how many columns it has there.
template <int VEC, int LPI, bool FULL>
__device__ __forceinline__ int rows_col(int cb, int lane, int k, int& nvalid) {
    const int col = cb * LPI * VEC + (lane % LPI) * (FULL ? VEC : 1);
    nvalid = FULL ? max(0, min(VEC, k - col)) : max(0, min(VEC, (k - col + LPI - 1) / LPI));
    return col;
}

// Long rows: Y row (+)= the row's slots.  A unit is one of a long row's T rows
// and 32 lanes of columns.  Rows of at most NARROW_SLOTS slots (listed first)
// take a warp per unit, slots in segment order; the others a block per unit,
// whose warps add a share of the slots each, in order, and then the shares in
// order.  Launched behind the main kernel.  (The warp that finished a row's last
// segment used to add its slots there, one tile-row at a time and two slots in
// flight beside the main loop's registers: with as many segments as small
// graphs need, hubs waited for it.)
constexpr int NARROW_SLOTS = 32;
template <int T, bool FULL, typename V>
__global__ void __launch_bounds__(ROWS_WARPS * 32, 4)
rows_fixup_kernel(SpmmRowsArgs<V> a, int nnarrow, int narrow_blocks, int ncb) {
    constexpr int VEC = FULL ? 16 / (int)sizeof(V) : 1, SL = 8;
    __shared__ V s_part[ROWS_WARPS][32 * VEC];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool alone = (int)blockIdx.x < narrow_blocks;  // block-uniform
    long long unit = alone ? (long long)blockIdx.x * ROWS_WARPS + warp : (long long)blockIdx.x - narrow_blocks;
    const int cb = (int)(unit % ncb), r = (int)(unit / ncb % T);
    long long lr = unit / ncb / T;
    if (alone && lr >= nnarrow) return;  // a block's last warps: nothing of theirs to wait for
    if (!alone) lr += nnarrow;
    const int4 L = __ldg(a.long_rows + lr);
    int nvalid;
    const int col = rows_col<VEC, 32, FULL>(cb, lane, a.k, nvalid);
    griddep_wait();  // the main kernel's slots
    const V* src = a.partials + ((long long)L.y * T + r) * a.k + col;
    const long long stride = (long long)T * a.k;
    const int end = alone ? L.z : (int)((long long)L.z * (warp + 1) / ROWS_WARPS);
    V tot[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) tot[e] = V(0);
    if (nvalid > 0) {
        int q = alone ? 0 : (int)((long long)L.z * warp / ROWS_WARPS);
        for (; q + SL <= end; q += SL) {
            V v[SL][VEC];
#pragma unroll
            for (int u = 0; u < SL; ++u) rows_load<V, VEC, FULL, 32, true>(v[u], src + (q + u) * stride, nvalid);
#pragma unroll
            for (int u = 0; u < SL; ++u) rows_add<V, VEC>(tot, v[u]);
        }
        if (q < end) {  // the rest, also in flight together
            V v[SL][VEC];
#pragma unroll
            for (int u = 0; u < SL; ++u) rows_load<V, VEC, FULL, 32, true>(v[u], src + (min(q + u, end - 1)) * stride, nvalid);
#pragma unroll
            for (int u = 0; u < SL; ++u)
                if (q + u < end) rows_add<V, VEC>(tot, v[u]);
        }
    }
    if (!alone) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) s_part[warp][e * 32 + lane] = tot[e];
        __syncthreads();
        if (warp != 0) return;
        for (int w = 1; w < ROWS_WARPS; ++w)
#pragma unroll
            for (int e = 0; e < VEC; ++e) tot[e] += s_part[w][e * 32 + lane];
    }
    if (nvalid > 0)
        rows_store<V, VEC, FULL, 32>(a.Y + ((long long)L.x * T + r) * a.ldy + col, tot, nvalid, a.accumulate != 0);
}

// A lane holds VEC columns, LPI = 32/IPW lanes a column block of LPI*VEC
// columns, and a warp loads IPW items (X rows) per instruction (k = 64 FP32:
// two X rows of 16 lanes x 16 bytes).  FULL: 16 bytes of neighbouring columns
// per lane, every vector whole and aligned.  Otherwise rows_width() picks as
// few scalar columns per lane as cover k.
// STREAM (whole-warp vector rows, k > 64 FP32, of a matrix with long rows):
// colind and Y pass through L2 evict-first, which leaves it to the X rows that
// the hubs reuse: R-MAT scale 20, k = 128 2040 -> 2031 us for forward and
// backward, scale 18 517 -> 510.  Others lose by it (256 stacked ER graphs, k =
// 128: 1349 -> 1365 us; 512, k = 64: 2103 -> 2142).
// Work item wi = (column block, task, row group), the group fastest, so the
// G warps of one tile-row read its structure at about the same time.
template <int T, int IPW, int VEC, bool FULL, bool STREAM, typename V>
__global__ void __launch_bounds__(ROWS_WARPS * 32, ROWS_BLOCKS)
spmm_rows_kernel(SpmmRowsArgs<V> a) {
    using P = RowsPack<T>;
    constexpr int R = ROWS_R;  // rows per task
    constexpr int G = T / R;      // row groups per tile-row
    // a step of 32 tiles adds at most 32*T items to a row: more than a region
    // holds only at T >= 16, where such a step is appended in lane ranges
    constexpr bool SPLIT = 32 * T > ROWS_CAP;
    static_assert(T <= ROWS_CAP, "one tile's items of a row must fit an empty region");
    constexpr int LPI = 32 / IPW;
    extern __shared__ int s_items[];  // per warp: R regions of ROWS_CAP items
    const int lane = threadIdx.x & 31;
    const int sub = lane / LPI;  // which item of an instruction this lane loads
    int* items = s_items + (threadIdx.x >> 5) * R * ROWS_CAP;
    const long long nwork = (long long)a.ntasks * a.ncb * G;
    const unsigned ldx = (unsigned)a.ldx;
    while (true) {
        unsigned wi = 0;
        if (lane == 0) wi = atomicAdd(reinterpret_cast<unsigned*>(a.state), 1u);
        wi = __shfl_sync(FULL_MASK, wi, 0);
        if (wi >= nwork) {
            // every warp fetches past the end exactly once; the last one to
            // count itself out leaves the state zeroed for the next launch
            if (lane == 0) {
                __threadfence();
                if (atomicAdd(a.state + 1, 1) == (int)(gridDim.x * ROWS_WARPS) - 1) {
                    a.state[0] = 0;
                    a.state[1] = 0;
                }
            }
            break;
        }
        // column block major: one pass over the tasks per block of X columns
        const int gi = (int)(wi % G);
        const unsigned wt = wi / G;
        const int cb = (int)(wt / (unsigned)a.ntasks), task = (int)(wt - (unsigned)cb * (unsigned)a.ntasks);
        const int4 t = __ldg(a.tasks + task);
        int nvalid;
        const int col = rows_col<VEC, LPI, FULL>(cb, lane, a.k, nvalid);
        const bool active = nvalid > 0;
        const V* xc = a.X + col;
        V acc[R][VEC];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[r][e] = V(0);

        int cnt[R];  // items in each row's region so far (warp-uniform)
#pragma unroll
        for (int r = 0; r < R; ++r) cnt[r] = 0;
        for (int j0 = t.y;; j0 += 32) {
            const bool more = j0 < t.z;  // warp-uniform
            const int j = j0 + lane;
            int tc = 0;
            RowsWord<T> w;
            if (more && j < t.z) {
                tc = STREAM ? __ldcs(a.colind + j) : __ldg(a.colind + j);
                w.load(a.tiles, j, gi);
            }
            // inclusive scan of the packed per-row counts of this step
            uint32_t inc[P::NP], own[P::NP];
#pragma unroll
            for (int p = 0; p < P::NP; ++p) {
                uint32_t c = 0;
#pragma unroll
                for (int q = 0; q < P::PER; ++q) c |= (uint32_t)__popc(w.bits(p * P::PER + q)) << (q * P::FIELD);
                own[p] = c;
                inc[p] = c;
#pragma unroll
                for (int s = 1; s < 32; s <<= 1) {
                    const uint32_t v = __shfl_up_sync(FULL_MASK, inc[p], s);
                    if (lane >= s) inc[p] += v;
                }
            }
            int tot[R];  // this step's items per row (warp-uniform)
            bool flush = !more, split = false;
#pragma unroll
            for (int p = 0; p < P::NP; ++p) {
                const uint32_t all = __shfl_sync(FULL_MASK, inc[p], 31);
#pragma unroll
                for (int q = 0; q < P::PER; ++q) {
                    const int r = p * P::PER + q;
                    tot[r] = (int)((all >> (q * P::FIELD)) & P::MASK);
                    flush |= cnt[r] + tot[r] > ROWS_CAP;
                    split |= tot[r] > ROWS_CAP;
                }
            }
            // the step's lanes in nsub ranges (one unless a row of the step
            // alone would overflow an empty region: then ROWS_CAP / T lanes each)
            int nsub = 1;
            if constexpr (SPLIT) {
                if (split) nsub = 32 * T / ROWS_CAP;
            }
            for (int sb = 0; sb < nsub; ++sb) {
                const int l0 = sb * (32 / nsub), l1 = l0 + 32 / nsub;  // lanes [l0, l1)
                uint32_t base[P::NP];  // packed counts of the lanes before l0
                int rt[R];             // the range's items per row
#pragma unroll
                for (int p = 0; p < P::NP; ++p) base[p] = 0;
#pragma unroll
                for (int r = 0; r < R; ++r) rt[r] = tot[r];
                if constexpr (SPLIT) {
                    if (nsub > 1) {  // warp-uniform
                        flush = false;
#pragma unroll
                        for (int p = 0; p < P::NP; ++p) {
                            base[p] = __shfl_sync(FULL_MASK, inc[p] - own[p], l0);
                            const uint32_t top = __shfl_sync(FULL_MASK, inc[p], l1 - 1) - base[p];
#pragma unroll
                            for (int q = 0; q < P::PER; ++q) {
                                const int r = p * P::PER + q;
                                rt[r] = (int)((top >> (q * P::FIELD)) & P::MASK);
                                flush |= cnt[r] + rt[r] > ROWS_CAP;
                            }
                        }
                    }
                }
                if (flush) {
                    // consume every row's region: sub-group `sub` takes items sub,
                    // sub+IPW, ... with ROWS_BATCH loads in flight per lane
                    if (active) {
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const int* it = items + r * ROWS_CAP;
                            const int qb = cnt[r];
                            int q = sub;
                            for (; q + (ROWS_BATCH - 1) * IPW < qb; q += ROWS_BATCH * IPW) {
                                V xv[ROWS_BATCH][VEC];
#pragma unroll
                                for (int u = 0; u < ROWS_BATCH; ++u) {
                                    const unsigned xr = (unsigned)it[q + u * IPW];
                                    rows_load<V, VEC, FULL, LPI>(xv[u], xc + (size_t)xr * ldx, nvalid);
                                }
                                rows_add_all<FULL, ROWS_BATCH, V, VEC>(acc[r], xv);
                            }
                            for (; q < qb; q += ROWS_REST * IPW) {  // the rest, ROWS_REST loads per lane per round
                                V xv[ROWS_REST][VEC];
#pragma unroll
                                for (int u = 0; u < ROWS_REST; ++u) {
                                    if (q + u * IPW < qb) {
                                        rows_load<V, VEC, FULL, LPI>(
                                            xv[u], xc + (size_t)(unsigned)it[q + u * IPW] * ldx, nvalid);
                                    } else {
#pragma unroll
                                        for (int e = 0; e < VEC; ++e) xv[u][e] = V(0);
                                    }
                                }
                                rows_add_all<FULL, ROWS_REST, V, VEC>(acc[r], xv);
                            }
                        }
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) cnt[r] = 0;
                    __syncwarp();
                }
                if (!more) break;
                // append the range's items to the row regions: X row index of
                // every set bit, in lane then column order
                if (lane >= l0 && lane < l1) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const int p = r / P::PER, q = r % P::PER;
                        int pos = r * ROWS_CAP + cnt[r] +
                                  (int)((((inc[p] - own[p]) - base[p]) >> (q * P::FIELD)) & P::MASK);
                        uint32_t bits = w.bits(r);
                        while (bits) {
                            const int b = 31 - __clz(bits);  // ascending column c = T-1-b
                            bits ^= 1u << b;
                            items[pos++] = tc * T + (T - 1 - b);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < R; ++r) cnt[r] += rt[r];
                __syncwarp();
            }
            if (!more) break;
        }
        // combine the IPW sub-groups (fixed butterfly order)
#pragma unroll
        for (int m = LPI; m < 32; m <<= 1)
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[r][e] += __shfl_xor_sync(FULL_MASK, acc[r][e], m);
        const bool writer = active && sub == 0;
        const int r0 = gi * R;  // first row of the tile-row this task covers
        if (t.w < 0) {
            if (writer) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    rows_store<V, VEC, FULL, LPI, STREAM>(a.Y + ((long long)t.x * T + r0 + r) * a.ldy + col, acc[r], nvalid,
                                                          a.accumulate != 0);
            }
            continue;
        }
        // a segment of a long row: its partial rows to the slot
        V* dst = a.partials + ((long long)t.w * T + r0) * a.k + col;
        if (writer) {
#pragma unroll
            for (int r = 0; r < R; ++r) rows_store<V, VEC, FULL, LPI>(dst + (long long)r * a.k, acc[r], nvalid, false);
        }
    }
}

// ---- plan ---------------------------------------------------------------------------
// Longest task in tiles: 30% of one resident warp's part of the tile visits
// (nt x T/4: a task's tiles are walked once per row group), so that the queue
// stays balanced at every graph size.  The best of 20/30/40% on R-MAT scales
// 16-20 with k = 64 and 128 on GB300; 40% fell off a cliff at T = 4 (the
// queue's end waits on long segments).
// The least segments, for the hubs of small graphs, and the tile-rows that stay
// whole whatever the share: cutting an ordinary tile-row costs more in slots
// and the second kernel than it wins (8140 x 4798 with 29 entries a row, 194
// tiles a tile-row at T = 8, k = 3: 21 us in two segments, 17 whole).  Segments
// of at least 128 tiles and 1024 bits instead: R-MAT scale 12 / 14 at T = 8, k =
// 64 46 / 58 us (31 / 28 with these), scale 14 at T = 4 43 (27), scale 16 at
// T = 16, k = 128 186 (117).
constexpr long long ROWS_MIN_TILES = 32, ROWS_MIN_BITS = 512;
// Whole up to 256 tiles at T <= 8 and 512 above, where a tile-row of the same
// rows has more of them, and a 4-row group takes fewer bits from each (ER, T =
// 16, k = 128: 5678 vertices of degree 28 28.7 us with 256 tiles, 24.5 with 512;
// 10 000 of degree 40 41.5 and 35.0; R-MAT scale 14, T = 16, k = 64 43.5 and
// 46.6; T = 8 27.2 and 39.1).
constexpr int rows_whole_tiles(int T) { return T <= 8 ? 256 : 512; }
constexpr int ROWS_WHOLE_BITS = 1024;
int spmm_rows_seg(int T, long long nt, int num_sms) {
    const long long visits = nt * (T / ROWS_R);
    const long long warps = (long long)std::max(num_sms, 1) * ROWS_BLOCKS * ROWS_WARPS;
    return (int)std::min(8192LL, std::max(ROWS_MIN_TILES, visits * 30 / (100 * warps)));
}

// Set bits of every tile-row, into zeroed bits[nb].  A warp takes 512 tiles in
// a row, 32 at a time (one per lane, its words with the widest loads), finds the
// tile-row of each once and adds up the lanes of one tile-row before it adds to
// bits[]: balanced whatever the row lengths (a warp per tile-row waited 38 us
// for the hubs of R-MAT scale 16; 4 us this way).  rowptr may be anything: a
// tile's row is searched in [0, nb).
constexpr int BITS_TILES = 512;
template <int T>
__global__ void __launch_bounds__(256)
tile_row_bits_kernel(const int* __restrict__ rowptr, const void* __restrict__ tiles, int nb, int nt,
                     unsigned long long* __restrict__ bits) {
    const int lane = threadIdx.x & 31;
    const long long first = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * BITS_TILES;
    if (first >= nt) return;  // warp-uniform
    const int end = (int)min(first + BITS_TILES, (long long)nt);
    auto row_of = [&](int j) {  // the last tile-row that starts at or before tile j
        int lo = 0, hi = nb;
        while (hi - lo > 1) {
            const int mid = lo + ((hi - lo) >> 1);
            if (rowptr[mid] <= j) lo = mid;
            else hi = mid;
        }
        return lo;
    };
    int row = row_of((int)first), next = rowptr[row + 1];  // warp-uniform, and where it ends
    unsigned sum = 0;                                         // this lane's bits of `row`
    for (int j0 = (int)first; j0 < end; j0 += 32) {
        const int j = j0 + lane;
        unsigned c = 0;
        if (j < end) {
            if constexpr (T == 8) {
                const uint2 v = __ldg(static_cast<const uint2*>(tiles) + j);
                c = __popc(v.x) + __popc(v.y);
            } else {
                const uint4* p = static_cast<const uint4*>(tiles) + (size_t)j * (T * T / 128);
#pragma unroll
                for (int q = 0; q < T * T / 128; ++q) {
                    const uint4 v = __ldg(p + q);
                    c += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
                }
            }
        }
        if (min(j0 + 32, end) <= next) {  // all of one tile-row
            sum += c;
            continue;
        }
        // the step crosses tile-rows: the open one, then a tile-row per lane
        sum += j < next ? c : 0u;
        sum = __reduce_add_sync(FULL_MASK, sum);
        if (lane == 0 && sum) atomicAdd(bits + row, (unsigned long long)sum);
        const int mine = j >= next && j < end ? row_of(j) : -1;
        row = row_of(min(j0 + 31, end - 1));
        next = rowptr[row + 1];
        if (mine >= 0 && mine != row && c) atomicAdd(bits + mine, (unsigned long long)c);
        sum = mine == row ? c : 0u;
    }
    sum = __reduce_add_sync(FULL_MASK, sum);
    if (lane == 0 && sum) atomicAdd(bits + row, (unsigned long long)sum);
}

b2sr_status spmm_rows_plan_create(const int* d_rowptr, const void* d_tiles, int nb, int nt, long long nnz, int T,
                                  int num_sms, SpmmRowsPlan* out, cudaStream_t s) {
    // Queue order.  T = 4: tasks of at least a quarter of a segment first,
    // then the rest, each class in tile-row order, so the queue ends on short
    // tasks while tile-rows that share X rows (the blocks of a batched graph)
    // still run together: R-MAT scale 18 / 20 as fast as longest first, and
    // 512 stacked ER graphs 1.86 ms against 2.85 ms longest first (2.61 ms in
    // row order with fixed segments).
    PlanRule rule{T == 4 ? PlanRule::TWO : PlanRule::BITS, spmm_rows_seg(T, nt, num_sms), T == 4 ? 2 : PLAN_CLASSES,
                  0, 0, NARROW_SLOTS, rows_whole_tiles(T), ROWS_WHOLE_BITS};
    // T >= 8: segments also bounded by their set bits, at most 70% of a
    // resident warp's share of all of them, and most set bits first.  A row
    // group holding hub rows carries far more set bits than its tiles suggest
    // (R-MAT scale 18, T = 32: ~9.3 K X-row loads for one warp in a
    // tile-bounded segment of tile-row 0, against 3.1 K set bits per resident
    // warp on average).  R-MAT scale 18, T = 8, k = 64 / 128: 198 / 291 us
    // against 249 / 469 us longest first; 100% instead of 70%: T = 32, k = 128
    // 535 instead of 449 us, 50%: T = 16, k = 33 298 instead of 269 us.
    long long* d_bits = nullptr;
    if (T >= 8 && nb > 0) {
        d_bits = static_cast<long long*>(dev_alloc(sizeof(long long) * (size_t)nb));
        if (!d_bits) return B2SR_ERR_ALLOC;
        const cudaError_t e = cudaMemsetAsync(d_bits, 0, sizeof(long long) * (size_t)nb, s);
        if (e != cudaSuccess) {
            set_cuda_error(e);
            dev_free(d_bits);
            return B2SR_ERR_CUDA;
        }
        const unsigned blocks = (unsigned)(((long long)nt + BITS_TILES * 8 - 1) / (BITS_TILES * 8));
        auto* bits = reinterpret_cast<unsigned long long*>(d_bits);
        if (nt > 0 && T == 8) tile_row_bits_kernel<8><<<blocks, 256, 0, s>>>(d_rowptr, d_tiles, nb, nt, bits);
        if (nt > 0 && T == 16) tile_row_bits_kernel<16><<<blocks, 256, 0, s>>>(d_rowptr, d_tiles, nb, nt, bits);
        if (nt > 0 && T == 32) tile_row_bits_kernel<32><<<blocks, 256, 0, s>>>(d_rowptr, d_tiles, nb, nt, bits);
        rule.row_bits = d_bits;
        const long long warps = (long long)std::max(num_sms, 1) * ROWS_BLOCKS * ROWS_WARPS;
        rule.seg_bits = std::max(ROWS_MIN_BITS, nnz * 7 / (10 * warps));
    }
    const PlanBounds cap = plan_bounds(rule, nb, nt, nnz);
    SpmmRowsPlan p;
    p.d_tasks = static_cast<int4*>(dev_alloc(sizeof(int4) * (size_t)(cap.tasks + cap.longs)));
    b2sr_status st = B2SR_ERR_ALLOC;
    PlanTotals t;
    if (p.d_tasks) {
        p.d_long = p.d_tasks + cap.tasks;
        st = build_plan(rule, d_rowptr, nb, cap, p.d_tasks, p.d_long, &t, s);
    } else {
        cudaStreamSynchronize(s);  // the set-bit count
    }
    dev_free(d_bits);
    if (st != B2SR_SUCCESS) {
        spmm_rows_plan_free(&p);
        return st;
    }
    p.ntasks = t.tasks;
    p.nlong = t.longs;
    p.nnarrow = t.narrow;
    p.nslots = t.slots;
    *out = p;
    return B2SR_SUCCESS;
}

void spmm_rows_plan_free(SpmmRowsPlan* p) {
    dev_free(p->d_tasks);  // d_long is part of it
    p->d_tasks = nullptr;
    p->d_long = nullptr;
}

// Columns of a warp pass (LPI * VEC) and of a lane.  rhs_block > 0 (FP32
// columns; half as many FP64 columns) fixes the block; 0 takes the narrowest
// that covers k.  Vector lanes (FULL): 16 bytes each, 4 to 32 lanes a row.
// Scalar lanes: one column each up to 32 columns (IPW rows per load below
// that), else 32 lanes of 2, 3 or 4 columns (FP64: 2).
struct RowsWidth {
    int ipw, vec;
};
static RowsWidth rows_width(int elem_bytes, int k, int rhs_block, bool full) {
    const int cols = rhs_block > 0 ? rhs_block * 4 / elem_bytes : k;
    RowsWidth w{1, full ? 16 / elem_bytes : 1};
    while (w.ipw < 8 && (32 / (2 * w.ipw)) * w.vec >= cols) w.ipw *= 2;
    const int most = 16 / elem_bytes;
    while (!full && w.vec < most && 32 * w.vec < cols) ++w.vec;
    return w;
}

size_t spmm_rows_scratch_bytes(const SpmmRowsPlan& p, int T, int elem_bytes, int k) {
    return (size_t)std::max(p.nslots, 1) * T * (size_t)k * elem_bytes;
}

size_t spmm_rows_state_bytes() { return 2 * sizeof(int); }

template <int T, int IPW, int VEC, bool FULL, bool STREAM, typename V>
static b2sr_status run_rows(SpmmRowsArgs<V> a, const SpmmRowsPlan& p, int num_sms, cudaStream_t s) {
    constexpr int SMEM = ROWS_WARPS * ROWS_R * ROWS_CAP * (int)sizeof(int);
    // per device: the attribute is set on every launch (cheap), the occupancy once
    cudaError_t e = cudaFuncSetAttribute(spmm_rows_kernel<T, IPW, VEC, FULL, STREAM, V>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return B2SR_ERR_CUDA;
    }
    static int blocks_per_sm = 0;  // per instantiation; the device's SM count scales it
    if (blocks_per_sm == 0) {
        int n = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, spmm_rows_kernel<T, IPW, VEC, FULL, STREAM, V>, ROWS_WARPS * 32,
                                                          SMEM);
        if (e != cudaSuccess) {
            set_cuda_error(e);
            return B2SR_ERR_CUDA;
        }
        blocks_per_sm = std::max(n, 1);
    }
    const long long nwork = (long long)a.ntasks * a.ncb * (T / ROWS_R);
    const long long want = (nwork + ROWS_WARPS - 1) / ROWS_WARPS;
    const int grid = (int)std::max(1LL, std::min<long long>((long long)num_sms * blocks_per_sm, want));
    // the queue counter is 32 bits and ends at nwork + one fetch per warp
    if (nwork + (long long)grid * ROWS_WARPS >= 0xffffffffLL) return B2SR_ERR_NOT_SUPPORTED;
    kernel_timer_mark(s, true);
    spmm_rows_kernel<T, IPW, VEC, FULL, STREAM, V><<<grid, ROWS_WARPS * 32, SMEM, s>>>(a);
    kernel_timer_mark(s, false);
    B2SR_LAUNCH_CHECK();
    add_launch_count(1);
    if (p.nlong > 0) {
        const int fcb = (a.k + 32 * (FULL ? VEC : 1) - 1) / (32 * (FULL ? VEC : 1));
        const long long narrow = ((long long)p.nnarrow * T * fcb + ROWS_WARPS - 1) / ROWS_WARPS;
        const long long blocks = narrow + (long long)(p.nlong - p.nnarrow) * T * fcb;
        if (blocks > 0x7fffffffLL) return B2SR_ERR_NOT_SUPPORTED;
        B2SR_CUDA_TRY(launch_dependent(rows_fixup_kernel<T, FULL, V>, (unsigned)blocks, ROWS_WARPS * 32u, s, a,
                                       p.nnarrow, (int)narrow, fcb));
        add_launch_count(1);
    }
    return B2SR_SUCCESS;
}

template <int T, typename V>
static b2sr_status rows_dispatch(const SpmmRowsArgs<V>& a, RowsWidth w, bool full, const SpmmRowsPlan& p,
                                 int num_sms, cudaStream_t s) {
    constexpr int MOST = 16 / (int)sizeof(V);
    if (full) {
        switch (w.ipw) {
            case 1: return p.nlong > 0 ? run_rows<T, 1, MOST, true, true, V>(a, p, num_sms, s)
                                       : run_rows<T, 1, MOST, true, false, V>(a, p, num_sms, s);
            case 2: return run_rows<T, 2, MOST, true, false, V>(a, p, num_sms, s);
            case 4: return run_rows<T, 4, MOST, true, false, V>(a, p, num_sms, s);
            default: return run_rows<T, 8, MOST, true, false, V>(a, p, num_sms, s);
        }
    }
    if (w.vec == 2) return run_rows<T, 1, 2, false, false, V>(a, p, num_sms, s);
    if constexpr (MOST == 4) {
        if (w.vec == 3) return run_rows<T, 1, 3, false, false, V>(a, p, num_sms, s);
        if (w.vec == 4) return run_rows<T, 1, 4, false, false, V>(a, p, num_sms, s);
    }
    switch (w.ipw) {
        case 1: return run_rows<T, 1, 1, false, false, V>(a, p, num_sms, s);
        case 2: return run_rows<T, 2, 1, false, false, V>(a, p, num_sms, s);
        case 4: return run_rows<T, 4, 1, false, false, V>(a, p, num_sms, s);
        default: return run_rows<T, 8, 1, false, false, V>(a, p, num_sms, s);
    }
}

template <typename V>
b2sr_status spmm_rows_launch(const MatView& A, const SpmmRowsPlan& p, const V* X, long long ldx, V* Y,
                             long long ldy, int k, int rhs_block, int accumulate, void* scratch, int* state,
                             int num_sms, cudaStream_t s) {
    constexpr int VEC = 16 / (int)sizeof(V);
    if (ldx > 0x7fffffffLL) return B2SR_ERR_NOT_SUPPORTED;
    // whole 16-byte column vectors everywhere: X, Y aligned, row strides and k multiples of VEC
    const bool full = ((uintptr_t)X % 16 == 0) && ((uintptr_t)Y % 16 == 0) && (ldx % VEC == 0) &&
                      (ldy % VEC == 0) && (k % VEC == 0);
    const RowsWidth w = rows_width((int)sizeof(V), k, rhs_block, full);
    const int KC = (32 / w.ipw) * w.vec;
    SpmmRowsArgs<V> a;
    a.colind = A.colind;
    a.tiles = A.tiles;
    a.X = X;
    a.Y = Y;
    a.ldx = ldx;
    a.ldy = ldy;
    a.k = k;
    a.ncb = (k + KC - 1) / KC;
    a.tasks = p.d_tasks;
    a.ntasks = p.ntasks;
    a.state = state;
    a.long_rows = p.d_long;
    a.partials = static_cast<V*>(scratch);
    a.accumulate = accumulate;
    if (A.T == 4) return rows_dispatch<4, V>(a, w, full, p, num_sms, s);
    if (A.T == 8) return rows_dispatch<8, V>(a, w, full, p, num_sms, s);
    if (A.T == 16) return rows_dispatch<16, V>(a, w, full, p, num_sms, s);
    if (A.T == 32) return rows_dispatch<32, V>(a, w, full, p, num_sms, s);
    return B2SR_ERR_INVALID_VALUE;
}

template b2sr_status spmm_rows_launch<float>(const MatView&, const SpmmRowsPlan&, const float*, long long, float*,
                                             long long, int, int, int, void*, int*, int, cudaStream_t);
template b2sr_status spmm_rows_launch<double>(const MatView&, const SpmmRowsPlan&, const double*, long long,
                                              double*, long long, int, int, int, void*, int*, int, cudaStream_t);

}  // namespace b2sr
