// Transposed B2SR built on the device.
//
// The tiles of A^T, in storage order, are the tiles of A ordered by
// (tile-column, tile-row).  A's tiles are stored in tile-row order, so a
// stable sort by tile-column gives that order: a least-significant-digit radix
// sort over digits of up to 9 bits (two passes for the 262,144 tile-columns of
// R-MAT scale 20 at T = 4).  Each pass counts the digits of every 4096-tile
// block, scans the per-(digit, block) counts (digit-major, so equal digits keep
// block order), and scatters.  A warp ranks its 256 consecutive tiles 32 at a
// time with __match_any_sync and a per-warp counter array, so the output order
// is the input order inside every digit; the block then orders its tiles by
// digit in shared memory and writes each digit's run at once.
//
// What travels with the tile-column: the tile-row, and at T = 4 and 8 the tile
// itself, bit-transposed in the first pass while A's tiles are read in order, so
// the last pass writes A^T's arrays and nothing is gathered.  At T = 16 and 32
// the tile's index travels, and one more kernel gathers the 32- or 128-byte
// tiles and transposes them across lanes.
//
// R-MAT scale 20 at T = 4, GB300: 1.82 ms of kernels with three 8-bit passes
// that moved (tile-column, index) one scattered word at a time and a gather by
// index (0.69 ms: a 32-byte sector per 4-byte tile), 2.8 ms a call; now
// 0.80 ms of kernels (scatters 0.30 and 0.28, counts 0.06 each) and 0.93 ms.
//
// Every index a kernel forms stays inside its buffers whatever the column
// values are (digits are masked; the lower bounds are clamped; the sorted
// values are a permutation of the tile indices), and a tile-column outside
// [0, nbc) is reported, not sorted.
#include <algorithm>
#include <type_traits>

#include "b2sr_common.cuh"

namespace b2sr {

namespace {

// 16 warps of 8 rounds each, three blocks per SM (R-MAT scale 20 at T = 4: 0.92
// ms a call; 8 warps of 16 rounds 1.00, 32 of 4 1.03, 8 of 8 0.99).
constexpr int TR_WARPS = 16;                     // warps per block
constexpr int TR_THREADS = TR_WARPS * 32;
constexpr int TR_ROUNDS = 8;                     // 32-tile rounds per warp
constexpr int TR_BLOCK = TR_THREADS * TR_ROUNDS;           // tiles per block
constexpr int TR_BITS = 9;                                 // digit bits at most
constexpr int TR_RADIX = 1 << TR_BITS;

// Digit of a key: `shift`, and `mask` = digits - 1.
__device__ __forceinline__ int tr_digit(int key, int shift, int mask) { return (int)((unsigned)key >> shift) & mask; }

// hist[d * nblocks + b] = tiles of block b whose digit is d; the first pass
// also flags tile-columns outside [0, nbc).
__global__ void __launch_bounds__(TR_THREADS)
radix_count_kernel(const int* __restrict__ keys, int n, int shift, int mask, int nblocks, int* __restrict__ hist,
                   int nbc, int* __restrict__ bad) {
    __shared__ int cnt[TR_RADIX];
    for (int i = threadIdx.x; i <= mask; i += TR_THREADS) cnt[i] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * TR_BLOCK;
    int flag = 0;
#pragma unroll 8
    for (int k = threadIdx.x; k < TR_BLOCK; k += TR_THREADS) {
        const long long i = base + k;
        if (i < n) {
            const int key = keys[i];
            if (bad && (unsigned)key >= (unsigned)nbc) flag = 1;
            atomicAdd(&cnt[tr_digit(key, shift, mask)], 1);
        }
    }
    if (flag) atomicOr(bad, 1);
    __syncthreads();
    for (int d = threadIdx.x; d <= mask; d += TR_THREADS) hist[(long long)d * nblocks + blockIdx.x] = cnt[d];
}

// What a tile carries beside its tile-column and tile-row: its transposed
// words (T = 4, 8) or its index in A.
template <int T> struct TrLoad { using type = int; };
template <> struct TrLoad<4> { using type = uint32_t; };
template <> struct TrLoad<8> { using type = unsigned long long; };

// Exchanges, for j = T/2 .. 1, the elements (r, c|j) and (r|j, c): bits 9j apart
// in a tile of one byte per row.
__device__ __forceinline__ uint32_t transpose_tile(uint32_t w) {  // T = 4
    w &= 0x0f0f0f0fu;
    uint32_t t = (w ^ (w >> 18)) & 0x00000303u;
    w ^= t ^ (t << 18);
    t = (w ^ (w >> 9)) & 0x00050005u;
    return w ^ t ^ (t << 9);
}
__device__ __forceinline__ unsigned long long transpose_tile(unsigned long long w) {  // T = 8
    unsigned long long t = (w ^ (w >> 36)) & 0x0f0f0f0full;
    w ^= t ^ (t << 36);
    t = (w ^ (w >> 18)) & 0x0000333300003333ull;
    w ^= t ^ (t << 18);
    t = (w ^ (w >> 9)) & 0x0055005500550055ull;
    return w ^ t ^ (t << 9);
}

// A's tile i (T = 4, 8), also from an array that is only byte-aligned.
template <typename P>
__device__ __forceinline__ P load_tile(const P* tiles, long long i) {
    if ((reinterpret_cast<uintptr_t>(tiles) & (sizeof(P) - 1)) == 0) return __ldg(tiles + i);
    const uint8_t* b = reinterpret_cast<const uint8_t*>(tiles + i);
    P w = 0;
#pragma unroll
    for (int k = 0; k < (int)sizeof(P); ++k) w |= (P)b[k] << (8 * k);
    return w;
}

// One stable scatter pass.  FIRST: the loads come from A (transposed tiles, or
// indices) instead of load_in.  keys_out / rows_out / load_out: the next
// pass's input, or in the last pass the sorted tile-columns, A^T's colind and
// A^T's tiles (T = 16 / 32: the order of the tiles).  offs = scanned hist.
template <int T, bool FIRST>
__global__ void __launch_bounds__(TR_THREADS, 3)
radix_scatter_kernel(const int* __restrict__ keys_in, const int* __restrict__ rows_in,
                     const typename TrLoad<T>::type* __restrict__ load_in, int n, int shift, int mask, int nblocks,
                     const int* __restrict__ offs, int* __restrict__ keys_out, int* __restrict__ rows_out,
                     typename TrLoad<T>::type* __restrict__ load_out) {
    using P = typename TrLoad<T>::type;
    extern __shared__ __align__(16) char s_mem[];
    P* s_load = reinterpret_cast<P*>(s_mem);                 // TR_BLOCK each, in digit order
    int* s_key = reinterpret_cast<int*>(s_load + TR_BLOCK);
    int* s_row = s_key + TR_BLOCK;
    uint16_t* wcnt = reinterpret_cast<uint16_t*>(s_row + TR_BLOCK);  // [warp][digit]
    __shared__ int s_base[TR_RADIX];   // where the block's digit d goes, minus its place in the block
    __shared__ int s_start[TR_RADIX];  // its place in the block
    __shared__ int s_sum[TR_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, digits = mask + 1;
    for (int i = threadIdx.x; i < TR_WARPS * TR_RADIX; i += TR_THREADS) wcnt[i] = 0;
    __syncthreads();
    const long long bbase = (long long)blockIdx.x * TR_BLOCK;
    const int count = (int)(n - bbase < TR_BLOCK ? n - bbase : TR_BLOCK);
    const int first = warp * 32 * TR_ROUNDS + lane;  // this lane's tiles: first + 32 q
    const unsigned below = (1u << lane) - 1u;
    uint16_t* mine = wcnt + warp * TR_RADIX;
    int key[TR_ROUNDS], rank[TR_ROUNDS];
#pragma unroll
    for (int q = 0; q < TR_ROUNDS; ++q) key[q] = first + 32 * q < count ? keys_in[bbase + first + 32 * q] : 0;
#pragma unroll
    for (int q = 0; q < TR_ROUNDS; ++q) {
        const bool ok = first + 32 * q < count;
        // lanes past the end form their own group and count nowhere
        const int d = ok ? tr_digit(key[q], shift, mask) : TR_RADIX;
        const unsigned peers = __match_any_sync(FULL_MASK, d);
        rank[q] = ok ? mine[d] + __popc(peers & below) : 0;
        __syncwarp();
        if (ok && (peers & below) == 0) mine[d] = (uint16_t)(mine[d] + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // per digit: the tiles of the warps before this one come first; then the
    // digits' places in the block (an exclusive scan, a digit per thread)
    static_assert(TR_THREADS == TR_RADIX, "a digit per thread");
    const int dg = threadIdx.x;
    int sum = 0;
    for (int w = 0; w < TR_WARPS; ++w) {
        const int c = wcnt[w * TR_RADIX + dg];
        wcnt[w * TR_RADIX + dg] = (uint16_t)sum;
        sum += c;
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL_MASK, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) s_sum[warp] = inc;
    __syncthreads();
    int at = inc - sum;
    for (int w = 0; w < warp; ++w) at += s_sum[w];
    s_start[dg] = at;
    s_base[dg] = (dg < digits ? offs[(long long)dg * nblocks + blockIdx.x] : 0) - at;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < TR_ROUNDS; ++q) {
        const int k = first + 32 * q;
        if (k < count) {
            const int d = tr_digit(key[q], shift, mask);
            const int to = s_start[d] + mine[d] + rank[q];
            const long long i = bbase + k;
            s_key[to] = key[q];
            s_row[to] = rows_in[i];
            if constexpr (!FIRST) s_load[to] = load_in[i];
            else if constexpr (T <= 8) s_load[to] = transpose_tile(load_tile(load_in, i));
            else s_load[to] = (int)i;
        }
    }
    __syncthreads();
#pragma unroll 4
    for (int k = threadIdx.x; k < count; k += TR_THREADS) {
        const int v = s_key[k];
        const int pos = s_base[tr_digit(v, shift, mask)] + k;
        keys_out[pos] = v;
        rows_out[pos] = s_row[k];
        load_out[pos] = s_load[k];
    }
}

// rowptr_t[c] = first position of tile-column c in the sorted keys (c <= nbc).
__global__ void transpose_rowptr_kernel(const int* __restrict__ keys, int n, int nbc, int* __restrict__ rowptr_t) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c > nbc) return;
    int lo = 0, hi = n;  // first index with keys[idx] >= c
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if (keys[mid] < c) lo = mid + 1;
        else hi = mid;
    }
    rowptr_t[c] = lo;
}

// tile_row[k] = the tile-row of tile k: one warp per tile-row (grid-stride;
// ranges clamped to [0, nt)).
__global__ void tile_row_kernel(const int* __restrict__ rowptr, int nb, int nt, int* __restrict__ tile_row) {
    const int lane = threadIdx.x & 31;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nb; r += nwarps) {
        const int b = max(rowptr[r], 0), e = min(rowptr[r + 1], nt);
        for (int k = b + lane; k < e; k += 32) tile_row[k] = (int)r;
    }
}

// Output tile d of A^T (T = 16, 32) from source tile order[d] of A.  T lanes
// per tile, one row word each; U tiles per lane group, all loaded before the
// first is transposed.  A step j of the transpose exchanges the blocks
// (row & j == 0, column & j) and (row & j, column & j == 0) between lanes j
// apart (T ballots and selects per tile took three times as long at T = 32).
template <int T>
__global__ void __launch_bounds__(256)
transpose_gather_kernel(const typename TileWord<T>::type* __restrict__ src, const int* __restrict__ order, int nt,
                        typename TileWord<T>::type* __restrict__ dst) {
    using W = typename TileWord<T>::type;
    constexpr int U = 4;
    const int r = threadIdx.x % T;
    const long long d0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / T * U;
    uint32_t w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) w[u] = d0 + u < nt ? (uint32_t)__ldg(src + (long long)__ldg(order + d0 + u) * T + r) : 0u;
#pragma unroll
    for (int j = T / 2; j >= 1; j >>= 1) {
        // columns with c & j == 0 (column c is bit T-1-c)
        const uint32_t m = (j == 16 ? 0xffff0000u : j == 8 ? 0xff00ff00u : j == 4 ? 0xf0f0f0f0u : j == 2 ? 0xccccccccu : 0xaaaaaaaau) &
                           (uint32_t)(0xffffffffu >> (32 - T));
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t o = __shfl_xor_sync(FULL_MASK, w[u], j);
            w[u] = (r & j) ? (w[u] & ~m) | ((o & ~m) << j) : (w[u] & m) | ((o & m) >> j);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (d0 + u < nt) dst[(d0 + u) * T + r] = (W)w[u];
}

template <int T>
size_t scatter_smem() {
    return (sizeof(typename TrLoad<T>::type) + 2 * sizeof(int)) * TR_BLOCK + sizeof(uint16_t) * TR_WARPS * TR_RADIX;
}

template <int T, bool FIRST>
cudaError_t launch_scatter(const int* keys, const int* rows, const void* load, int nt, int shift, int mask, int nblocks,
                           const int* offs, int* keys_out, int* rows_out, void* load_out, cudaStream_t s) {
    using P = typename TrLoad<T>::type;
    const cudaError_t e = cudaFuncSetAttribute(radix_scatter_kernel<T, FIRST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)scatter_smem<T>());
    if (e != cudaSuccess) return e;
    radix_scatter_kernel<T, FIRST><<<nblocks, TR_THREADS, scatter_smem<T>(), s>>>(
        keys, rows, static_cast<const P*>(load), nt, shift, mask, nblocks, offs, keys_out, rows_out,
        static_cast<P*>(load_out));
    return cudaGetLastError();
}

// The passes over one scratch block: [flags | hist | scan | keys, rows, loads x 2].
template <int T>
b2sr_status run_transpose(const int* rowptr, const int* colind, const void* tiles, int nb, int nbc, int nt,
                          int* rowptr_t, int* colind_t, void* tiles_t, cudaStream_t s) {
    using P = typename TrLoad<T>::type;
    int bits = 0;
    while (bits < 31 && (1LL << bits) < (long long)nbc) ++bits;  // keys < nbc <= 2^bits
    // at least one pass: it also checks every tile-column against nbc
    const int passes = std::max(1, (bits + TR_BITS - 1) / TR_BITS);
    const int per = std::max(1, (bits + passes - 1) / passes), mask = (1 << per) - 1;
    const int nblocks = (int)(((long long)nt + TR_BLOCK - 1) / TR_BLOCK);
    const long long nhist = (long long)(mask + 1) * nblocks;
    if (nhist > INT_MAX) return B2SR_ERR_OVERFLOW;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t p = at;
        at += (bytes + 255) / 256 * 256;
        return p;
    };
    const size_t words = sizeof(int) * (size_t)nt, loads = sizeof(P) * (size_t)nt;
    const size_t o_flags = take(2 * sizeof(int)), o_hist = take(sizeof(int) * ((size_t)nhist + 1)),
                 o_scan = take(exclusive_scan_scratch(nhist));
    const size_t o_key[2] = {take(words), take(passes > 1 ? words : 0)};
    const size_t o_row[2] = {take(words), take(passes > 1 ? words : 0)};
    // the last pass writes its loads to tiles_t (or, as the order, to the set
    // that it does not read)
    const size_t o_load[2] = {take(T >= 16 || passes > 1 ? loads : 0), take(T >= 16 ? (passes > 1 ? loads : 0) : (passes > 2 ? loads : 0))};
    char* mem = static_cast<char*>(dev_alloc(at));
    if (!mem) return B2SR_ERR_ALLOC;
    int* flags = reinterpret_cast<int*>(mem + o_flags);  // [0] scan overflow, [1] tile-column out of range
    int* hist = reinterpret_cast<int*>(mem + o_hist);
    int* key[2] = {reinterpret_cast<int*>(mem + o_key[0]), reinterpret_cast<int*>(mem + o_key[1])};
    int* row[2] = {reinterpret_cast<int*>(mem + o_row[0]), reinterpret_cast<int*>(mem + o_row[1])};
    void* load[2] = {mem + o_load[0], mem + o_load[1]};
    cudaError_t e = cudaMemsetAsync(flags, 0, 2 * sizeof(int), s);
    // the tile-rows of A's tiles, where the first pass does not write rows
    int* tile_row = passes > 1 ? row[1] : row[0];
    const long long row_blocks = std::min<long long>(((long long)nb * 32 + 255) / 256, 65535LL * 8);
    if (e == cudaSuccess) {
        tile_row_kernel<<<(unsigned)row_blocks, 256, 0, s>>>(rowptr, nb, nt, tile_row);
        e = cudaGetLastError();
    }
    const int* keys = colind;
    const int* rows = tile_row;
    const void* in = tiles;
    void* order = nullptr;
    for (int p = 0; p < passes && e == cudaSuccess; ++p) {
        const int shift = per * p, to = p & 1;
        const bool last = p + 1 == passes;
        radix_count_kernel<<<nblocks, TR_THREADS, 0, s>>>(keys, nt, shift, mask, nblocks, hist, nbc,
                                                          p == 0 ? flags + 1 : nullptr);
        const int scans = exclusive_scan_async(hist, (int)nhist, flags, mem + o_scan, s);
        int* rows_out = last ? colind_t : row[to];
        void* load_out = last && T <= 8 ? tiles_t : load[to];
        e = p == 0 ? launch_scatter<T, true>(keys, rows, in, nt, shift, mask, nblocks, hist, key[to], rows_out, load_out, s)
                   : launch_scatter<T, false>(keys, rows, in, nt, shift, mask, nblocks, hist, key[to], rows_out, load_out, s);
        keys = key[to];
        rows = rows_out;
        in = order = load_out;
        add_launch_count(2 + scans);
    }
    if (e == cudaSuccess) {
        transpose_rowptr_kernel<<<(unsigned)(((long long)nbc + 1 + 255) / 256), 256, 0, s>>>(keys, nt, nbc, rowptr_t);
        add_launch_count(2);
        if constexpr (T >= 16) {
            using W = typename TileWord<T>::type;
            const long long threads = ((long long)nt + 3) / 4 * T;
            transpose_gather_kernel<T><<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(
                static_cast<const W*>(tiles), static_cast<const int*>(order), nt, static_cast<W*>(tiles_t));
            add_launch_count(1);
        }
        e = cudaGetLastError();
    }
    int h[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, flags, sizeof(h), cudaMemcpyDeviceToHost, s);
    const cudaError_t drained = cudaStreamSynchronize(s);
    dev_free(mem);
    if (e == cudaSuccess) e = drained;
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return B2SR_ERR_CUDA;
    }
    if (h[1] != 0) return B2SR_ERR_INVALID_VALUE;  // a tile-column outside the matrix
    return h[0] != 0 ? B2SR_ERR_OVERFLOW : B2SR_SUCCESS;
}

}  // namespace

b2sr_status launch_transpose(const int* rowptr, const int* colind, const void* tiles, int nb, int nbc, int nt, int T,
                             int* rowptr_t, int* colind_t, void* tiles_t, cudaStream_t s) {
    if (nt < 0 || nb < 0 || nbc < 0) return B2SR_ERR_INVALID_VALUE;
    if (nt == 0) {
        B2SR_CUDA_TRY(cudaMemsetAsync(rowptr_t, 0, sizeof(int) * ((size_t)nbc + 1), s));
        // as below: the transpose may be used on any stream, or freed, from here on
        B2SR_CUDA_TRY(cudaStreamSynchronize(s));
        return B2SR_SUCCESS;
    }
    if (nb == 0 || nbc == 0) return B2SR_ERR_INVALID_VALUE;  // tiles need a tile-row and a tile-column
    switch (T) {
        case 4: return run_transpose<4>(rowptr, colind, tiles, nb, nbc, nt, rowptr_t, colind_t, tiles_t, s);
        case 8: return run_transpose<8>(rowptr, colind, tiles, nb, nbc, nt, rowptr_t, colind_t, tiles_t, s);
        case 16: return run_transpose<16>(rowptr, colind, tiles, nb, nbc, nt, rowptr_t, colind_t, tiles_t, s);
        case 32: return run_transpose<32>(rowptr, colind, tiles, nb, nbc, nt, rowptr_t, colind_t, tiles_t, s);
    }
    return B2SR_ERR_INVALID_VALUE;
}

}  // namespace b2sr
