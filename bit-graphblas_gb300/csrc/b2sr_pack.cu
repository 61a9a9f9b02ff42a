// CSR -> B2SR packing on the device, and dense <-> bit vector conversion.
//
// The reference packs on the host, one tile-row at a time: per non-empty
// tile-row it copies a CSR slab to the device, expands it to dense float tiles
// with cusparseScsr2bsr and bit-packs them with ToBit{T}Col
// (bmv_eval/backend/csr2bsr_batch_bsrbmv.cu:34-133, bmv_eval/backend/bsrbmv.cu:33-203).
// Here the whole matrix is packed on the device with no float expansion:
//
//   1. validate the CSR, an entry per thread (which also counts duplicates, so
//      the number of set bits is known without reading the tiles);
//   2. cut every tile-row into chunks of about 400 (T = 4) or 320 entries;
//   3. a warp per chunk sorts the chunk's entries by (tile-column, row, column),
//      by merging its rows (T <= 8) or in registers, writes the sorted keys and
//      counts the tiles;
//   4. scans give the tile-row pointer and the tile count (the one value the
//      host waits for, to allocate the result);
//   5. a warp per chunk reads its sorted keys back and assembles the tiles in
//      shared memory, in tile-column order: the order cusparseScsr2bsr produces.
//
// R-MAT scale 20 at T = 4 (31.4 M entries, 27.2 M tiles), GB300: a T-way merge
// of the sorted rows by T lanes, counted twice and filled once, took 0.55 +
// 0.55 + 0.75 ms beside 0.36 ms of validation by a warp per row; it advances a
// tile per step and waits on a load in each.  Sorting works on all lanes
// whatever the rows look like.
#include <algorithm>
#include <type_traits>

#include "b2sr_common.cuh"

namespace b2sr {

enum : int { CSR_BAD_ROWPTR = 1, CSR_BAD_COLIND = 2, CSR_UNSORTED = 4 };

// What the host reads back after the count.
struct PackInfo {
    int flag;  // CSR_* bits
    int err;   // a scan overflowed int32
    int nt;
    int pad;
    unsigned long long dups;  // entries equal to the one before them in their row
};

// rowptr[0] == 0, rowptr[nrows] == nnz, 0 <= rowptr[i] <= rowptr[i+1] <= nnz; and
// the entries that start a row, a bit each.  In bounds whatever rowptr holds.
__global__ void __launch_bounds__(256)
validate_rows_kernel(const int* __restrict__ rowptr, int nrows, int nnz, uint32_t* __restrict__ starts,
                     PackInfo* __restrict__ info) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool bad = i == 0 && (rowptr[0] != 0 || rowptr[nrows] != nnz);
    if (i < nrows) {
        const int b = rowptr[i], e = rowptr[i + 1];
        if (b < 0 || e < b || e > nnz) bad = true;
        else if (e > b) atomicOr(starts + (b >> 5), 1u << (b & 31));
    }
    if (__any_sync(FULL_MASK, bad) && (threadIdx.x & 31) == 0) atomicOr(&info->flag, (int)CSR_BAD_ROWPTR);
}

// colind in [0, ncols) and non-decreasing within each row, with the number of
// entries equal to the one before.  Four consecutive entries per thread, as one
// 16-byte load where ALIGNED.  (A warp per row, the rows' own bounds: 357 us
// for R-MAT scale 20; a lookup in rowptr for every entry not above the one
// before: 112 us, issue-bound.)  Only behind a good rowptr: with rowptr[nrows] !=
// nnz the array may be shorter than nnz.
template <bool ALIGNED>
__global__ void __launch_bounds__(256)
validate_entries_kernel(const int* __restrict__ colind, int ncols, int nnz, const uint32_t* __restrict__ starts,
                        PackInfo* __restrict__ info) {
    if (info->flag & CSR_BAD_ROWPTR) return;  // set by validate_rows_kernel only, so uniform
    const long long p = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    const int n = (int)(nnz - p < 4 ? nnz - p : 4);  // <= 0 past the end
    int c[4] = {0, 0, 0, 0};
    if (ALIGNED && n == 4) {
        const int4 v = __ldg(reinterpret_cast<const int4*>(colind + p));
        c[0] = v.x;
        c[1] = v.y;
        c[2] = v.z;
        c[3] = v.w;
    } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (u < n) c[u] = __ldg(colind + p + u);
    }
    int prev = __shfl_up_sync(FULL_MASK, c[3], 1);
    if ((threadIdx.x & 31) == 0 && p > 0 && n > 0) prev = __ldg(colind + p - 1);
    const uint32_t start = n > 0 ? __ldg(starts + (p >> 5)) >> (p & 31) : 0;  // p is a multiple of 4
    int bad = 0, dups = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (u < n) {
            if ((unsigned)c[u] >= (unsigned)ncols) bad |= CSR_BAD_COLIND;
            if (!((start >> u) & 1u) && p + u > 0) {
                if (prev > c[u]) bad |= CSR_UNSORTED;
                if (prev == c[u]) ++dups;
            }
            prev = c[u];
        }
    }
    bad = __reduce_or_sync(FULL_MASK, bad);
    dups = __reduce_add_sync(FULL_MASK, dups);
    if ((threadIdx.x & 31) == 0) {
        if (bad) atomicOr(&info->flag, bad);
        if (dups) atomicAdd(&info->dups, (unsigned long long)dups);
    }
}

// ---- chunks ---------------------------------------------------------------------
// A tile-row of L entries has ceil(L / chunk_entries) chunks (none when empty),
// cut at the tile-columns of every q-th entry of its longest row, so a chunk
// covers a range of tile-columns and holds about chunk_entries entries.  A
// warp sorts up to CHUNK_CAP of them; rows that fill the range unevenly can
// exceed that, and dense tiles or duplicates do: such a chunk is merged by T
// lanes instead, one tile-column at a time, so a few of them set the time.
// 400 at T = 4 and 320 above: packing R-MAT scale 16 at T = 8 takes 213 us with
// 320, 247 with 400 and 286 with 450 (scale 18: 328, 342, 437), scale 20 at
// T = 4 827, 798 and 900.  A tile-row of at most CHUNK_CAP entries is one chunk.
constexpr int CHUNK_CAP = 512;
__host__ __device__ constexpr int chunk_entries(int T) { return T == 4 ? 400 : 320; }
__host__ __device__ __forceinline__ int chunks_of(int entries, int T) {
    const int per = chunk_entries(T);
    return entries == 0 ? 0 : entries <= CHUNK_CAP ? 1 : (entries + per - 1) / per;
}

// Chunks of every tile-row.
__global__ void chunk_plan_kernel(const int* __restrict__ rowptr, int nrows, int nb, int T,
                                  const PackInfo* __restrict__ info, int* __restrict__ nch) {
    const long long tr = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (tr >= nb) return;
    int n = 0;
    if (info->flag == 0) {
        const long long r0 = tr * T, r1 = r0 + T < nrows ? r0 + T : nrows;
        n = chunks_of(rowptr[r1] - rowptr[r0], T);
    }
    nch[tr] = n;
}

// chunk_tr[c] = the tile-row of chunk c; a warp per 32 tile-rows, a tile-row
// with many chunks written by the whole warp.
__global__ void chunk_rows_kernel(const int* __restrict__ choff, int nb, int max_chunks, int* __restrict__ chunk_tr) {
    const int lane = threadIdx.x & 31;
    const long long tr = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int b = tr < nb ? choff[tr] : 0, e = tr < nb ? min(choff[tr + 1], max_chunks) : 0;
    if (e - b <= 4)
        for (int c = b; c < e; ++c) chunk_tr[c] = (int)tr;
    unsigned many = __ballot_sync(FULL_MASK, e - b > 4);
    while (many) {
        const int l = __ffs(many) - 1;
        many &= many - 1;
        const int bb = __shfl_sync(FULL_MASK, b, l), ee = __shfl_sync(FULL_MASK, e, l);
        const int t = __shfl_sync(FULL_MASK, (int)tr, l);
        for (int c = bb + lane; c < ee; c += 32) chunk_tr[c] = t;
    }
}

// Sort key of entry (row r, column col) of a tile-row: tile-column, then row,
// then column inside the tile.  32 bits where they hold it.
template <int T, typename Key>
__device__ __forceinline__ Key pack_key(int r, int col) {
    constexpr int LT = Log2<T>::value;
    return ((Key)(col >> LT) << (2 * LT)) | (Key)((r << LT) | (col & (T - 1)));
}
template <int T> inline bool key_fits_32(int ncols) {
    // below the all-ones key that pads a chunk
    return (((long long)(ncols > 0 ? ncols - 1 : 0) >> Log2<T>::value) + 1) << (2 * Log2<T>::value) <= 0xffffffffLL;
}

// Ascending bitonic sort of 32*K keys, element e = lane*K + k; all indices of
// key[] are compile-time constants.  (A counting sort into 32*K buckets in
// shared memory and odd-even exchanges inside the buckets takes 14% fewer
// instructions on R-MAT scale 20, where the fullest of a chunk's 512 buckets
// holds 13 - 20 keys, and more registers: the same time.)
template <typename Key, int K>
__device__ __forceinline__ void warp_sort(Key (&key)[K], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * K; size <<= 1) {
#pragma unroll
        for (int j = size / 2; j > 0; j >>= 1) {
            if (j >= K) {
                const int d = j / K;
                // the lower partner of an ascending run keeps the smaller key
                const bool keep_min = ((lane & d) == 0) == (((lane * K) & size) == 0);
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const Key o = __shfl_xor_sync(FULL_MASK, key[k], d);
                    key[k] = keep_min ? (o < key[k] ? o : key[k]) : (o > key[k] ? o : key[k]);
                }
            } else {
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    if ((k & j) == 0) {
                        const bool up = size < K ? (k & size) == 0 : ((lane * K) & size) == 0;
                        const Key a = key[k], b = key[k | j];
                        const Key lo = a < b ? a : b, hi = a < b ? b : a;
                        key[k] = up ? lo : hi;
                        key[k | j] = up ? hi : lo;
                    }
                }
            }
        }
    }
}

// Shared memory place of element e: one word of padding per 32, so that both
// e = lane*K + k and e = k*32 + lane are free of bank conflicts.
__device__ __forceinline__ int spread(int e) { return e + (e >> 5); }

// The keys of a chunk lie in buf row after row, each row's ascending, row r's
// from pre[r] to pre[r + 1]: merges neighbouring rows, then neighbouring pairs
// and so on, until key[k] is element lane*K + k of the whole (~0 past the end).
// A lane makes K consecutive elements of a round; a binary search finds where
// they begin in the two runs they come from.
// Packing R-MAT scale 20 by merging instead of sorting: T = 4 806 -> 726 us,
// T = 8 816 -> 768, T = 16 870 -> 878, T = 32 3018 -> 3080 (a round for every
// doubling of T, where the sort's cost does not depend on T); for chunks of at
// most 128 entries too: T = 4 728, T = 8 778.
template <int T, int K> constexpr bool MERGES_ROWS = T <= 8 && K >= 8;
template <int T, typename Key, int K>
__device__ __forceinline__ void merge_rows(Key (&key)[K], Key* buf, const int* pre, int n, int lane) {
    const int o = lane * K;
#pragma unroll 1
    for (int span = 1; span < T; span <<= 1) {
        int r = 0;  // first row of the last pair of runs with pre <= o
#pragma unroll 1
        for (int step = T / 2; step >= 2 * span; step >>= 1)
            if (pre[r + step] <= o) r += step;
        int a = pre[r], b = pre[r + span], aend = b, bend = pre[r + 2 * span];
        const int d = min(o, n) - a;
        int lo = max(0, d - (bend - b)), hi = min(d, aend - a);
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (buf[spread(a + mid)] < buf[spread(b + d - 1 - mid)]) lo = mid + 1;
            else hi = mid;
        }
        a += lo;
        b += d - lo;
        Key ka = a < aend ? buf[spread(a)] : ~Key(0), kb = b < bend ? buf[spread(b)] : ~Key(0);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            while ((ka & kb) == ~Key(0) && r + 2 * span < T) {  // the next pair of runs
                r += 2 * span;
                a = bend;
                b = aend = pre[r + span];
                bend = pre[r + 2 * span];
                ka = a < aend ? buf[spread(a)] : ~Key(0);
                kb = b < bend ? buf[spread(b)] : ~Key(0);
            }
            const bool ta = ka < kb;
            key[k] = ta ? ka : kb;
            const int i = ta ? ++a : ++b;
            const Key v = i < (ta ? aend : bend) ? buf[spread(i)] : ~Key(0);
            if (ta) ka = v;
            else kb = v;
        }
        if (2 * span < T) {
            __syncwarp();
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (o + k < n) buf[spread(o + k)] = key[k];
            __syncwarp();
        }
    }
}

// A chunk as its warp sees it: lane r < T holds row r's first entry in the
// chunk, and how many entries the rows before it have there.
struct ChunkRows {
    int p, pre;
    int n;  // entries of the chunk
};

// Sorts the chunk's n <= 32*K entries, writes them to `sorted` and returns the
// number of distinct tile-columns.  buf: spread(32*K) keys of shared memory.
template <int T, typename Key, int K>
__device__ __forceinline__ int sort_chunk(const int* __restrict__ colind, const ChunkRows& c, Key* __restrict__ sorted,
                                          Key* buf, int* pre, int lane) {
    constexpr int LT = Log2<T>::value;
    Key key[K];
    constexpr int L = K < 8 ? K : 8;  // loads in flight
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += L) {
        int row[L], col[L];
#pragma unroll
        for (int k = 0; k < L; ++k) {
            const int i = (k0 + k) * 32 + lane;
            int r = 0;  // the last row with pre <= i
#pragma unroll
            for (int step = T / 2; step >= 1; step >>= 1) {
                const int before = __shfl_sync(FULL_MASK, c.pre, r + step);
                if (before <= i) r += step;
            }
            const int p = __shfl_sync(FULL_MASK, c.p - c.pre, r) + i;
            row[k] = r;
            col[k] = i < c.n ? __ldg(colind + p) : -1;
        }
#pragma unroll
        for (int k = 0; k < L; ++k) key[k0 + k] = col[k] >= 0 ? pack_key<T, Key>(row[k], col[k]) : ~Key(0);
    }
    if constexpr (MERGES_ROWS<T, K>) {
        if (lane < T) pre[lane] = c.pre;
        if (lane == 0) pre[T] = c.n;
#pragma unroll
        for (int k = 0; k < K; ++k) buf[spread(k * 32 + lane)] = key[k];
        __syncwarp();
        merge_rows<T, Key, K>(key, buf, pre, c.n, lane);
        __syncwarp();
    } else {
        warp_sort<Key, K>(key, lane);
    }
    Key prev = __shfl_up_sync(FULL_MASK, key[K - 1], 1);
    int tiles = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const bool first = k == 0 && lane == 0;
        if (key[k] != ~Key(0) && (first || (key[k] >> (2 * LT)) != (prev >> (2 * LT)))) ++tiles;
        prev = key[k];
    }
    // lane*K + k order -> coalesced stores
#pragma unroll
    for (int k = 0; k < K; ++k) buf[spread(lane * K + k)] = key[k];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = k * 32 + lane;
        if (i < c.n) sorted[i] = buf[spread(i)];
    }
    __syncwarp();
    return __reduce_add_sync(FULL_MASK, tiles);
}

// A chunk of any size: lane r walks its entries, and the smallest pending
// tile-column's entries are written row after row.
template <int T, typename Key>
__device__ __forceinline__ int merge_chunk(const int* __restrict__ colind, int p, int e, Key* __restrict__ sorted, int lane) {
    constexpr int LT = Log2<T>::value;
    int tiles = 0;
    while (true) {
        const int mine = p < e ? colind[p] >> LT : INT_MAX;
        const int m = __reduce_min_sync(FULL_MASK, mine);
        if (m == INT_MAX) break;
        int q = p;
#pragma unroll 1
        while (q < e && (colind[q] >> LT) == m) ++q;
        int inc = q - p;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL_MASK, inc, o);
            if (lane >= o) inc += v;
        }
        Key* dst = sorted + (inc - (q - p));
#pragma unroll 1
        for (; p < q; ++p) *dst++ = pack_key<T, Key>(lane, colind[p]);
        sorted += __shfl_sync(FULL_MASK, inc, 31);
        ++tiles;
    }
    return tiles;
}

constexpr int PACK_WARPS = 8;

// Step 3.  ccount[c] = tiles of chunk c (0 past the last chunk); coff_e[c] =
// its first entry in `sorted` (chunks are in entry order; coff_e[chunks] = nnz).
// Blocks per SM with 32-bit keys, T <= 8 and above: 6 (40 registers) and 5 (48), a
// few bytes spilled: R-MAT scale 20, T = 4, 738 us with 5 and 722 with 6, T =
// 32 the same.
template <int T, typename Key>
__global__ void __launch_bounds__(PACK_WARPS * 32, sizeof(Key) == 4 ? (T <= 8 ? 6 : 5) : 1)
chunk_sort_kernel(const int* __restrict__ rowptr, const int* __restrict__ colind, int nrows, int nb,
                  const int* __restrict__ choff, const int* __restrict__ chunk_tr, int max_chunks,
                  int* __restrict__ ccount, int* __restrict__ coff_e, Key* __restrict__ sorted) {
    constexpr int LT = Log2<T>::value;
    __shared__ Key s_buf[PACK_WARPS][CHUNK_CAP + CHUNK_CAP / 32];
    __shared__ int s_pre[PACK_WARPS][T + 1];
    const int lane = threadIdx.x & 31;
    const long long cl = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (cl > max_chunks) return;
    const int c = (int)cl, nchunks = choff[nb];
    if (c >= nchunks) {
        if (lane == 0) {
            if (c < max_chunks) ccount[c] = 0;
            if (c == nchunks) coff_e[c] = nchunks ? rowptr[nrows] : 0;
        }
        return;
    }
    const int tr = chunk_tr[c], k = c - choff[tr], nk = choff[tr + 1] - choff[tr];
    const long long row = (long long)tr * T + lane;
    int rs = 0, re = 0;
    if (lane < T && row < nrows) {
        rs = rowptr[row];
        re = rowptr[row + 1];
    }
    const int first = __shfl_sync(FULL_MASK, rs, 0);
    int p = rs, e = re;
    if (nk > 1) {  // warp-uniform
        const int len = re - rs, longest = __reduce_max_sync(FULL_MASK, len);
        const int lead = __ffs(__ballot_sync(FULL_MASK, len == longest)) - 1;
        const int lead_rs = __shfl_sync(FULL_MASK, rs, lead);
        const long long q = (longest + nk - 1) / nk, i0 = k * q, i1 = i0 + q;
        // every row's entries from the tile-column of lead entry i0 to that of
        // i1, both searches in step
        const int from = k == 0 ? INT_MIN : i0 < longest ? (colind[lead_rs + i0] >> LT) << LT : INT_MAX;
        const int to = k + 1 < nk && i1 < longest ? (colind[lead_rs + i1] >> LT) << LT : INT_MAX;
        int pe = re, eb = rs;  // p in [p, pe], e in [eb, e]
        while (p < pe || eb < e) {
            const int m0 = p + ((pe - p) >> 1), m1 = eb + ((e - eb) >> 1);
            const int c0 = p < pe ? colind[m0] : 0, c1 = eb < e ? colind[m1] : 0;
            if (p < pe) {
                if (c0 < from) p = m0 + 1;
                else pe = m0;
            }
            if (eb < e) {
                if (c1 < to) eb = m1 + 1;
                else e = m1;
            }
        }
    }
    const int n = e - p;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL_MASK, inc, o);
        if (lane >= o) inc += v;
    }
    ChunkRows rows{p, inc - n, __shfl_sync(FULL_MASK, inc, 31)};
    const int at = first + __reduce_add_sync(FULL_MASK, p - rs);  // entries of the tile-row before the chunk
    Key* buf = s_buf[threadIdx.x >> 5];
    Key* out = sorted + at;
    int tiles;
    if (rows.n > CHUNK_CAP) tiles = merge_chunk<T, Key>(colind, p, e, out, lane);
    else if (rows.n > 256) tiles = sort_chunk<T, Key, 16>(colind, rows, out, buf, s_pre[threadIdx.x >> 5], lane);
    else if (rows.n > 128) tiles = sort_chunk<T, Key, 8>(colind, rows, out, buf, s_pre[threadIdx.x >> 5], lane);
    else if (rows.n > 64) tiles = sort_chunk<T, Key, 4>(colind, rows, out, buf, s_pre[threadIdx.x >> 5], lane);
    else if (rows.n > 32) tiles = sort_chunk<T, Key, 2>(colind, rows, out, buf, s_pre[threadIdx.x >> 5], lane);
    else tiles = sort_chunk<T, Key, 1>(colind, rows, out, buf, s_pre[threadIdx.x >> 5], lane);
    if (lane == 0) {
        ccount[c] = tiles;
        coff_e[c] = at;
    }
}

// Step 4: rowptr of the tiles, and the tile count, from the scanned chunk
// offsets (coff[c] = tiles before chunk c, also for c past the last chunk).
__global__ void tile_rowptr_kernel(const int* __restrict__ choff, const int* __restrict__ coff, int nb,
                                   int* __restrict__ browptr, PackInfo* __restrict__ info) {
    const long long tr = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (tr > nb) return;
    const int v = coff[choff[tr]];
    browptr[tr] = v;
    if (tr == nb) info->nt = v;
}

// Step 5: the tiles of chunk c from its sorted keys, 32 entries at a time.  A
// batch touches at most 32 tiles, one of them perhaps begun by the batch
// before; they are assembled in a ring of 32 tiles in shared memory and leave
// in whole 16-byte words (T = 16, 32) or whole tiles once finished.  ALIGNED:
// `tiles` is 16-byte aligned (else word by word).
template <int T, typename Key, bool ALIGNED>
__global__ void __launch_bounds__(PACK_WARPS * 32)
chunk_fill_kernel(const int* __restrict__ choff, int nb, const int* __restrict__ coff, const int* __restrict__ coff_e,
                  const Key* __restrict__ sorted, int* __restrict__ bcolind, typename TileWord<T>::type* tiles) {
    using W = typename TileWord<T>::type;
    constexpr int LT = Log2<T>::value;
    constexpr int RB = T == 4 ? 8 : T;    // bits from one row to the next
    constexpr int TW = T * RB / 32;       // 32-bit words of a tile
    __shared__ __align__(16) uint32_t s_ring[PACK_WARPS][32 * TW];
    const int lane = threadIdx.x & 31;
    const long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= choff[nb]) return;
    uint32_t* ring = s_ring[threadIdx.x >> 5];
    for (int i = lane; i < 32 * TW; i += 32) ring[i] = 0;
    __syncwarp();
    const int b = coff_e[c], e = coff_e[c + 1];
    int cur = coff[c], done = cur;  // tiles begun / written
    Key last = 0;                   // tile-column of the batch before
    // writes tiles [done, upto) and clears their places
    auto flush = [&](int upto) {
        if constexpr (ALIGNED) {
            using U = typename std::conditional<T == 4, uint32_t, typename std::conditional<T == 8, uint2, uint4>::type>::type;
            constexpr int PER = TW * 4 / (int)sizeof(U);  // units of a tile
            U* dst = reinterpret_cast<U*>(tiles) + (size_t)done * PER;
            U* src = reinterpret_cast<U*>(ring);
            const int n = (upto - done) * PER;
            for (int u = lane; u < n; u += 32) {
                U& v = src[((done + u / PER) & 31) * PER + u % PER];
                dst[u] = v;
                v = U{};
            }
        } else {
            W* dst = tiles + (size_t)done * T;
            W* src = reinterpret_cast<W*>(ring);
            const int n = (upto - done) * T;
            for (int u = lane; u < n; u += 32) {
                W& v = src[((done + u / T) & 31) * T + u % T];
                dst[u] = v;
                v = 0;
            }
        }
        done = upto;
        __syncwarp();
    };
    for (int i0 = b; i0 < e; i0 += 32) {
        const bool on = i0 + lane < e;
        const Key key = on ? __ldcs(sorted + i0 + lane) : Key(0);
        const Key m = key >> (2 * LT);
        Key before = __shfl_up_sync(FULL_MASK, m, 1);
        if (lane == 0) before = last;
        const bool head = on && ((lane == 0 && i0 == b) || m != before);
        const unsigned heads = __ballot_sync(FULL_MASK, head);
        if (heads & 1u) flush(cur);  // the open tile is finished
        const int t = cur - 1 + __popc(heads & (0xffffffffu >> (31 - lane)));
        if (on) {
            const int bit = (int)((key >> LT) & (T - 1)) * RB + T - 1 - (int)(key & (T - 1));
            atomicOr(ring + (t & 31) * TW + bit / 32, 1u << (bit & 31));
        }
        if (head) bcolind[t] = (int)m;
        cur += __popc(heads);
        __syncwarp();
        flush(cur - 1);
        last = __shfl_sync(FULL_MASK, m, 31);
    }
    flush(cur);
}

// ---- exclusive scan -------------------------------------------------------------
// Per-block sums, a scan of the block sums in one CTA where they are many, and
// the per-block scan with the block offset.  Sums are kept in 64 bits so an int32
// overflow of the total is detected instead of wrapping.
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ long long block_sum_ll(long long v, long long* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL_MASK, v, o);
    if (lane == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL_MASK, v, o);
    }
    __syncthreads();
    return v;  // valid in thread 0
}

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and stores the block total in *total.
__device__ __forceinline__ long long block_exscan_ll(long long v, long long* sh, long long* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        long long u = __shfl_up_sync(FULL_MASK, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        long long s = lane < nw ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            long long u = __shfl_up_sync(FULL_MASK, s, o);
            if (lane >= o) s += u;
        }
        if (lane < nw) sh[lane] = s;  // inclusive warp totals
    }
    __syncthreads();
    const long long warp_off = w > 0 ? sh[w - 1] : 0;
    *total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warp_off + inc - v;
}

__global__ void __launch_bounds__(SCAN_THREADS)
scan_reduce_kernel(const int* __restrict__ vals, int n, long long* __restrict__ partial) {
    __shared__ long long sh[32];
    const long long base = (long long)blockIdx.x * SCAN_TILE;
    long long v = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        long long i = base + (long long)k * SCAN_THREADS + threadIdx.x;
        if (i < n) v += vals[i];
    }
    v = block_sum_ll(v, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
}

__global__ void __launch_bounds__(SCAN_THREADS)
scan_partials_kernel(long long* __restrict__ partial, int nblocks) {
    __shared__ long long sh[32];
    long long carry = 0;
    for (int base = 0; base < nblocks; base += SCAN_THREADS) {
        const int i = base + threadIdx.x;
        long long v = i < nblocks ? partial[i] : 0;
        long long total;
        long long ex = block_exscan_ll(v, sh, &total);
        if (i < nblocks) partial[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) partial[nblocks] = carry;
}

// partial: the block sums (SUMS: every block adds up those before it), or
// their exclusive scan.
template <bool SUMS>
__global__ void __launch_bounds__(SCAN_THREADS)
scan_apply_kernel(int* __restrict__ vals, int n, const long long* __restrict__ partial,
                  int nblocks, int* __restrict__ err) {
    __shared__ long long sh[32], s_before;
    const long long base = (long long)blockIdx.x * SCAN_TILE;
    // Each thread owns SCAN_ITEMS consecutive elements.
    const long long first = base + (long long)threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    long long local = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = (first + k < n) ? vals[first + k] : 0;
        local += v[k];
    }
    long long before = 0;
    if (SUMS) {
        for (int i = threadIdx.x; i < (int)blockIdx.x; i += SCAN_THREADS) before += partial[i];
        before = block_sum_ll(before, sh);
        if (threadIdx.x == 0) s_before = before;
        __syncthreads();
        before = s_before;
    } else {
        before = partial[blockIdx.x];
    }
    long long total;
    long long ex = block_exscan_ll(local, sh, &total) + before;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (first + k < n) {
            if (ex > INT_MAX) *err = 1;
            vals[first + k] = (int)ex;
        }
        ex += v[k];
    }
    if ((int)blockIdx.x == nblocks - 1 && threadIdx.x == 0) {
        const long long all = before + total;
        if (all > INT_MAX) *err = 1;
        vals[n] = (int)(all > INT_MAX ? INT_MAX : all);
    }
}

size_t exclusive_scan_scratch(long long n) {
    return sizeof(long long) * (size_t)((n > 0 ? (n + SCAN_TILE - 1) / SCAN_TILE : 1) + 1);
}

int exclusive_scan_async(int* vals, int n, int* err, void* scratch, cudaStream_t s) {
    const int nblocks = n > 0 ? (n + SCAN_TILE - 1) / SCAN_TILE : 1;
    long long* partial = static_cast<long long*>(scratch);
    // one launch up to SCAN_TILE values, two while a block can add up the sums
    // before it in a step, else three
    if (nblocks > 1) scan_reduce_kernel<<<nblocks, SCAN_THREADS, 0, s>>>(vals, n, partial);
    if (nblocks > SCAN_THREADS) {
        scan_partials_kernel<<<1, SCAN_THREADS, 0, s>>>(partial, nblocks);
        scan_apply_kernel<false><<<nblocks, SCAN_THREADS, 0, s>>>(vals, n, partial, nblocks, err);
    } else {
        scan_apply_kernel<true><<<nblocks, SCAN_THREADS, 0, s>>>(vals, n, partial, nblocks, err);
    }
    return nblocks > SCAN_THREADS ? 3 : nblocks > 1 ? 2 : 1;
}

// ---- host side --------------------------------------------------------------------
// One scratch allocation holds everything the two passes share.
struct PackJob::Layout {
    PackInfo* info;
    uint32_t* starts;
    size_t zeroed;  // info and starts, from the beginning on
    void* scan;
    int *choff, *chunk_tr, *coff, *coff_e;
    void* sorted;
    size_t bytes;
    Layout(char* base, int nb, long long max_chunks, long long nnz, size_t key) {
        size_t at = 0;
        auto take = [&](size_t n) {
            char* p = base + at;
            at += (n + 255) / 256 * 256;
            return p;
        };
        info = reinterpret_cast<PackInfo*>(take(sizeof(PackInfo)));
        starts = reinterpret_cast<uint32_t*>(take(sizeof(uint32_t) * (size_t)(nnz / 32 + 1)));
        zeroed = at;
        scan = take(exclusive_scan_scratch(std::max<long long>(nb, max_chunks)));
        choff = reinterpret_cast<int*>(take(sizeof(int) * ((size_t)nb + 1)));
        chunk_tr = reinterpret_cast<int*>(take(sizeof(int) * (size_t)max_chunks));
        coff = reinterpret_cast<int*>(take(sizeof(int) * ((size_t)max_chunks + 1)));
        coff_e = reinterpret_cast<int*>(take(sizeof(int) * ((size_t)max_chunks + 1)));
        sorted = take(key * (size_t)nnz);
        bytes = at;
    }
};

PackJob::~PackJob() {
    if (!scratch) return;
    cudaStreamSynchronize(s);
    dev_free(scratch);
}

template <int T>
static void launch_sort(bool wide, int blocks, const int* rowptr, const int* colind, int nrows, int nb,
                        const PackJob::Layout& l, int max_chunks, cudaStream_t s) {
    if (wide)
        chunk_sort_kernel<T, unsigned long long><<<blocks, PACK_WARPS * 32, 0, s>>>(
            rowptr, colind, nrows, nb, l.choff, l.chunk_tr, max_chunks, l.coff, l.coff_e,
            static_cast<unsigned long long*>(l.sorted));
    else
        chunk_sort_kernel<T, uint32_t><<<blocks, PACK_WARPS * 32, 0, s>>>(
            rowptr, colind, nrows, nb, l.choff, l.chunk_tr, max_chunks, l.coff, l.coff_e,
            static_cast<uint32_t*>(l.sorted));
}

template <int T, typename Key>
static void launch_fill_key(int blocks, int nb, const PackJob::Layout& l, int* bcolind, void* tiles, cudaStream_t s) {
    using W = typename TileWord<T>::type;
    const Key* keys = static_cast<const Key*>(l.sorted);
    if ((uintptr_t)tiles % 16 == 0)
        chunk_fill_kernel<T, Key, true><<<blocks, PACK_WARPS * 32, 0, s>>>(l.choff, nb, l.coff, l.coff_e, keys, bcolind,
                                                                           static_cast<W*>(tiles));
    else
        chunk_fill_kernel<T, Key, false><<<blocks, PACK_WARPS * 32, 0, s>>>(l.choff, nb, l.coff, l.coff_e, keys,
                                                                            bcolind, static_cast<W*>(tiles));
}

b2sr_status PackJob::count(const int* rowptr, const int* colind, int nrows, int ncols, int nnz, int T_, int* browptr,
                           int* nt, long long* set_bits, cudaStream_t stream) {
    s = stream;
    T = T_;
    nb = (int)(((long long)nrows + T - 1) / T);
    *nt = 0;
    if (set_bits) *set_bits = 0;
    if (nrows == 0) {
        B2SR_CUDA_TRY(cudaMemsetAsync(browptr, 0, sizeof(int), s));
        B2SR_CUDA_TRY(cudaStreamSynchronize(s));
        return B2SR_SUCCESS;
    }
    wide = !(T == 4 ? key_fits_32<4>(ncols) : T == 8 ? key_fits_32<8>(ncols) : T == 16 ? key_fits_32<16>(ncols)
                                                                                   : key_fits_32<32>(ncols));
    max_chunks = nb + nnz / chunk_entries(T) + 1;  // sum over tile-rows of ceil(entries / chunk_entries)
    n_entries = nnz;
    const size_t key = wide ? 8 : 4;
    scratch = dev_alloc(Layout(nullptr, nb, max_chunks, nnz, key).bytes);
    if (!scratch) return B2SR_ERR_ALLOC;
    const Layout l(static_cast<char*>(scratch), nb, max_chunks, nnz, key);
    B2SR_CUDA_TRY(cudaMemsetAsync(scratch, 0, l.zeroed, s));
    validate_rows_kernel<<<(unsigned)(((long long)nrows + 255) / 256), 256, 0, s>>>(rowptr, nrows, nnz, l.starts, l.info);
    if (nnz > 0) {
        const unsigned blocks = (unsigned)(((long long)nnz + 1023) / 1024);
        if ((uintptr_t)colind % 16 == 0)
            validate_entries_kernel<true><<<blocks, 256, 0, s>>>(colind, ncols, nnz, l.starts, l.info);
        else
            validate_entries_kernel<false><<<blocks, 256, 0, s>>>(colind, ncols, nnz, l.starts, l.info);
    }
    chunk_plan_kernel<<<(nb + 255) / 256, 256, 0, s>>>(rowptr, nrows, nb, T, l.info, l.choff);
    exclusive_scan_async(l.choff, nb, &l.info->err, l.scan, s);
    chunk_rows_kernel<<<(nb + 255) / 256, 256, 0, s>>>(l.choff, nb, (int)max_chunks, l.chunk_tr);
    const int blocks = (int)((max_chunks + 1 + PACK_WARPS - 1) / PACK_WARPS);
    switch (T) {
        case 4: launch_sort<4>(wide, blocks, rowptr, colind, nrows, nb, l, (int)max_chunks, s); break;
        case 8: launch_sort<8>(wide, blocks, rowptr, colind, nrows, nb, l, (int)max_chunks, s); break;
        case 16: launch_sort<16>(wide, blocks, rowptr, colind, nrows, nb, l, (int)max_chunks, s); break;
        default: launch_sort<32>(wide, blocks, rowptr, colind, nrows, nb, l, (int)max_chunks, s); break;
    }
    exclusive_scan_async(l.coff, (int)max_chunks, &l.info->err, l.scan, s);
    tile_rowptr_kernel<<<(nb + 1 + 255) / 256, 256, 0, s>>>(l.choff, l.coff, nb, browptr, l.info);
    B2SR_LAUNCH_CHECK();
    PackInfo h;
    B2SR_CUDA_TRY(cudaMemcpyAsync(&h, l.info, sizeof h, cudaMemcpyDeviceToHost, s));
    B2SR_CUDA_TRY(cudaStreamSynchronize(s));
    if (h.flag != 0) return B2SR_ERR_INVALID_CSR;
    if (h.err != 0) return B2SR_ERR_OVERFLOW;
    *nt = h.nt;
    if (set_bits) *set_bits = (long long)nnz - (long long)h.dups;
    return B2SR_SUCCESS;
}

b2sr_status PackJob::fill(int* bcolind, void* tiles) {
    const Layout l(static_cast<char*>(scratch), nb, max_chunks, n_entries, wide ? 8 : 4);
    const int blocks = (int)((max_chunks + PACK_WARPS - 1) / PACK_WARPS);
#define B2SR_FILL_T(TT)                                                                       \
    if (T == TT) {                                                                            \
        if (wide) launch_fill_key<TT, unsigned long long>(blocks, nb, l, bcolind, tiles, s);  \
        else launch_fill_key<TT, uint32_t>(blocks, nb, l, bcolind, tiles, s);                 \
    }
    B2SR_FILL_T(4) B2SR_FILL_T(8) B2SR_FILL_T(16) B2SR_FILL_T(32)
#undef B2SR_FILL_T
    B2SR_LAUNCH_CHECK();
    return B2SR_SUCCESS;
}

// ---- dense <-> bits ---------------------------------------------------------------
// A warp votes on 32 consecutive elements; the bit-reversed ballot holds
// element 32k + l at bit 31 - l, i.e. 32/T words of the MSB-first layout side
// by side (ToBit{T}Row order, bmv_eval/backend/bsrbmv.cu:64-222).
template <int T>
__global__ void pack_vec_bits_kernel(const float* __restrict__ x, long long n,
                                     typename TileWord<T>::type* __restrict__ bits,
                                     long long nwords) {
    using W = typename TileWord<T>::type;
    constexpr int PER = 32 / T;  // words per ballot
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long chunk = warp; chunk * 32 < n; chunk += nwarps) {
        const long long i = chunk * 32 + lane;
        const bool v = i < n && x[i] > 0.0f;
        const uint32_t word32 = __brev(__ballot_sync(FULL_MASK, v));
        if (lane < PER) {
            const long long wi = chunk * PER + lane;
            if (wi < nwords) {
                const uint32_t w = (T == 32) ? word32 : (word32 >> (32 - T * (lane + 1))) & ((1u << T) - 1u);
                bits[wi] = (W)w;
            }
        }
    }
}

template <int T>
__global__ void unpack_vec_bits_kernel(const typename TileWord<T>::type* __restrict__ bits,
                                       long long n, float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t w = bits[i / T];
    out[i] = ((w >> (T - 1 - (int)(i % T))) & 1u) ? 1.0f : 0.0f;
}

b2sr_status launch_pack_vec_bits(const float* x, int n, int T, void* bits, cudaStream_t s) {
    if (n <= 0) return B2SR_SUCCESS;
    const long long nwords = ((long long)n + T - 1) / T;
    const int threads = 256;
    long long blocks = (((long long)n + 31) / 32 * 32 + threads - 1) / threads;
    if (blocks > 65535LL * 8) blocks = 65535LL * 8;
    switch (T) {
        case 4: pack_vec_bits_kernel<4><<<(unsigned)blocks, threads, 0, s>>>(x, n, (uint8_t*)bits, nwords); break;
        case 8: pack_vec_bits_kernel<8><<<(unsigned)blocks, threads, 0, s>>>(x, n, (uint8_t*)bits, nwords); break;
        case 16: pack_vec_bits_kernel<16><<<(unsigned)blocks, threads, 0, s>>>(x, n, (uint16_t*)bits, nwords); break;
        case 32: pack_vec_bits_kernel<32><<<(unsigned)blocks, threads, 0, s>>>(x, n, (uint32_t*)bits, nwords); break;
        default: return B2SR_ERR_INVALID_VALUE;
    }
    B2SR_LAUNCH_CHECK();
    return B2SR_SUCCESS;
}

b2sr_status launch_unpack_vec_bits(const void* bits, int n, int T, float* out, cudaStream_t s) {
    if (n <= 0) return B2SR_SUCCESS;
    const int threads = 256;
    const unsigned blocks = (unsigned)(((long long)n + threads - 1) / threads);
    switch (T) {
        case 4: unpack_vec_bits_kernel<4><<<blocks, threads, 0, s>>>((const uint8_t*)bits, n, out); break;
        case 8: unpack_vec_bits_kernel<8><<<blocks, threads, 0, s>>>((const uint8_t*)bits, n, out); break;
        case 16: unpack_vec_bits_kernel<16><<<blocks, threads, 0, s>>>((const uint16_t*)bits, n, out); break;
        case 32: unpack_vec_bits_kernel<32><<<blocks, threads, 0, s>>>((const uint32_t*)bits, n, out); break;
        default: return B2SR_ERR_INVALID_VALUE;
    }
    B2SR_LAUNCH_CHECK();
    return B2SR_SUCCESS;
}

// ---- set-bit count ----------------------------------------------------------------
__global__ void count_bits_kernel(const uint8_t* __restrict__ bytes, long long nbytes,
                                  unsigned long long* __restrict__ out) {
    unsigned long long c = 0;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nbytes; i += stride)
        c += __popc((unsigned)bytes[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(FULL_MASK, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

b2sr_status launch_count_bits(const void* tiles, long long nwords, int T,
                              unsigned long long* d_count, cudaStream_t s) {
    B2SR_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), s));
    const long long nbytes = nwords * word_bytes(T);
    if (nbytes == 0) return B2SR_SUCCESS;
    const int threads = 256;
    long long blocks = (nbytes + threads - 1) / threads;
    if (blocks > 4096) blocks = 4096;
    count_bits_kernel<<<(unsigned)blocks, threads, 0, s>>>((const uint8_t*)tiles, nbytes, d_count);
    B2SR_LAUNCH_CHECK();
    return B2SR_SUCCESS;
}

}  // namespace b2sr
