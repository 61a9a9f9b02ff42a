// Row-binned multiplies with a tile spread over T/4 lanes: bit vectors at
// T = 32, 32- / 64-bit OR at T = 16 and 32, FP32 sums at T = 32 on matrices
// whose tiles do not fit in L2.
//
// A 16 x 16 tile is 32 bytes, a 32 x 32 tile 128.  With a lane per tile a warp
// load touches 32 separate lines and a lane needs T row accumulators; here
// neighbouring lanes share a tile, each with four of its rows (8 bytes at
// T = 16, 16 at T = 32), so a warp load covers 8 / 4 whole tiles back to back
// and a lane keeps four accumulators.
//
// A pass is four such loads, so 32 / 16 tile slots.  The rows of plan bins
// 0..4 (at most 2 * 2^b tiles at T = 16, 2^b at T = 32) share passes; bin 5,
// longer rows and the segments of rows cut up, has a warp per task.
//
// Sums visit a row's tiles in a fixed order, so they are reproducible.
//
// GB300, R-MAT scale 20 unless said otherwise, lane per tile -> this form:
//   T = 32 bin_bin_bin 1% / 30% frontier   419 / 419 -> 194 / 276 us
//   T = 32 int32 counts, 30%               525 -> 292 us
//   T = 32 FP32 sums                       673 -> 505 us (2.9 -> 3.9 TB/s of
//     tiles); 300,000-vertex ER graph of degree 16: 178 -> 135 us
//   64 frontiers, R-MAT scale 18: T = 32 723 -> 174 us, T = 16 287 -> 144 us;
//   32 frontiers: 403 -> 130 us, 148 -> 91 us
// Bit vectors at T = 16 stay with a lane per tile (112 us when this was 138; 105
// now: a lane's two 16-byte loads already use every sector they touch).
#pragma once

#include "b2sr_spmv_impl.cuh"

namespace b2sr {

constexpr int WIDE_STEPS = 4;  // tile loads of a pass
template <int T> constexpr int WIDE_LPT = T / 4;                        // lanes per tile
template <int T> constexpr int WIDE_TPS = 32 / WIDE_LPT<T>;             // tiles per load
template <int T> constexpr int WIDE_PASS = WIDE_STEPS * WIDE_TPS<T>;    // tile slots of a pass

// Four rows of a tile.  Column c is bit T-1-c of every row.
template <int T> struct WideRows;
template <> struct WideRows<32> {
    uint4 w;
    __device__ __forceinline__ void clear() { w = make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ void load(const void* tiles, int j, int sub) {
        w = __ldcs(static_cast<const uint4*>(tiles) + (size_t)j * 8 + sub);
    }
    __device__ __forceinline__ uint32_t columns() const { return w.x | w.y | w.z | w.w; }
    __device__ __forceinline__ uint32_t row(int k) const { return k == 0 ? w.x : k == 1 ? w.y : k == 2 ? w.z : w.w; }
    // row k has the column of bit b (a single bit, or 0)
    __device__ __forceinline__ bool has(int k, uint32_t b) const {
        return ((k == 0 ? w.x : k == 1 ? w.y : k == 2 ? w.z : w.w) & b) != 0;
    }
    // rows with a bit in common with the x word, row k at bit 3-k; and counts
    __device__ __forceinline__ uint32_t hits(uint32_t x) const {
        return ((w.x & x) ? 8u : 0u) | ((w.y & x) ? 4u : 0u) | ((w.z & x) ? 2u : 0u) | ((w.w & x) ? 1u : 0u);
    }
    __device__ __forceinline__ void add_counts(int (&acc)[4], uint32_t x) const {
        acc[0] += __popc(w.x & x);
        acc[1] += __popc(w.y & x);
        acc[2] += __popc(w.z & x);
        acc[3] += __popc(w.w & x);
    }
};
template <> struct WideRows<16> {
    uint2 w;  // row 0 in the low half of w.x
    __device__ __forceinline__ void clear() { w = make_uint2(0, 0); }
    __device__ __forceinline__ void load(const void* tiles, int j, int sub) {
        w = __ldcs(static_cast<const uint2*>(tiles) + (size_t)j * 4 + sub);
    }
    __device__ __forceinline__ uint32_t columns() const {
        const uint32_t v = w.x | w.y;
        return (v | (v >> 16)) & 0xffffu;
    }
    __device__ __forceinline__ uint32_t row(int k) const { return ((k < 2 ? w.x : w.y) >> (16 * (k & 1))) & 0xffffu; }
    __device__ __forceinline__ bool has(int k, uint32_t b) const {
        return ((k < 2 ? w.x : w.y) & ((k & 1) ? b << 16 : b)) != 0;
    }
};

// The tile slots of one pass: which tile this lane's group has in step s.
// G slots per task; ty / tz: lane i holds task i's tile range.
template <int T, int G>
__device__ __forceinline__ void wide_slots(int ty, int tz, int q, int (&j)[WIDE_STEPS]) {
#pragma unroll
    for (int s = 0; s < WIDE_STEPS; ++s) {
        const int slot = s * WIDE_TPS<T> + q;
        const int b = __shfl_sync(FULL_MASK, ty, slot / G), e = __shfl_sync(FULL_MASK, tz, slot / G);
        j[s] = b + slot % G < e ? b + slot % G : -1;
    }
}

// ---- value semirings: FP32 sums, 32- / 64-bit OR ------------------------------------------
// x element of column c of tile-column tc (columns at or past ncols read as zero)
template <class Sem>
__device__ __forceinline__ typename Sem::V wide_x(const typename Sem::V* __restrict__ x, long long base, int c,
                                                  int ncols) {
    return base + c < ncols ? __ldg(x + base + c) : Sem::zero();
}

// Four rows k[] of a tile through its whole x segment (all lanes of the warp
// at once): every lane of a tile loads four elements of the segment, and the
// lanes pass each other the columns.
template <int T, class Sem>
__device__ __forceinline__ void wide_add_dense(typename Sem::V (&acc)[4], const uint32_t (&k)[4], long long base,
                                               const typename Sem::V* __restrict__ x, int ncols, int lane) {
    using V = typename Sem::V;
    constexpr int LPT = WIDE_LPT<T>, PER = 16 / (int)sizeof(V);
    const long long c0 = base + 4 * (lane % LPT);
    V seg[4];
    if (c0 + 4 <= ncols) {
#pragma unroll
        for (int p = 0; p < 4 / PER; ++p)
            *reinterpret_cast<uint4*>(seg + p * PER) = __ldg(reinterpret_cast<const uint4*>(x + c0) + p);
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) seg[e] = c0 + e < ncols ? __ldg(x + c0 + e) : Sem::zero();
    }
#pragma unroll 1
    for (int l = 0; l < LPT; ++l) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const V v = __shfl_sync(FULL_MASK, seg[e], l, LPT);
            const uint32_t b = 1u << (T - 1 - e - 4 * l);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (k[i] & b) acc[i] = Sem::add(acc[i], v);
        }
    }
}

// Adds a pass's tiles into NACC accumulator sets: WIDE_STEPS / NACC
// neighbouring steps belong to the same tile-row.  The first K set columns of
// every tile (found once for its lanes) have their x elements in flight
// together; the rest follow one by one, or, from WIDE_DENSE<T> on, through
// the whole segment.
template <int T> constexpr int WIDE_K = T == 32 ? 2 : 1;
template <int T> constexpr int WIDE_DENSE = 8;
template <int T, class Sem, int NACC>
__device__ __forceinline__ void wide_add(typename Sem::V (&acc)[NACC][4], const WideRows<T> (&w)[WIDE_STEPS],
                                         const int (&tc)[WIDE_STEPS], const typename Sem::V* __restrict__ x,
                                         int ncols, int lane) {
    using V = typename Sem::V;
    constexpr int K = WIDE_K<T>, PER = WIDE_STEPS / NACC;
    uint32_t cm[WIDE_STEPS], bit[WIDE_STEPS][K];
    V v[WIDE_STEPS][K];
#pragma unroll
    for (int s = 0; s < WIDE_STEPS; ++s) {
        cm[s] = w[s].columns();
#pragma unroll
        for (int o = 1; o < WIDE_LPT<T>; o <<= 1) cm[s] |= __shfl_xor_sync(FULL_MASK, cm[s], o);
    }
#pragma unroll
    for (int s = 0; s < WIDE_STEPS; ++s) {
        const long long base = (long long)tc[s] * T;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t b = cm[s] ? 0x80000000u >> __clz(cm[s]) : 0u;  // the lowest column left
            const int c = T - 32 + __clz(b);
            bit[s][k] = b;
            v[s][k] = b ? wide_x<Sem>(x, base, c, ncols) : Sem::zero();
            cm[s] ^= b;
        }
    }
#pragma unroll
    for (int s = 0; s < WIDE_STEPS; ++s) {
        V(&a)[4] = acc[s / PER];
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (w[s].has(i, bit[s][k])) a[i] = Sem::add(a[i], v[s][k]);
    }
    int most = 0;
#pragma unroll
    for (int s = 0; s < WIDE_STEPS; ++s) most = max(most, __popc(cm[s]));
    most = __reduce_max_sync(FULL_MASK, most);
    if (most > WIDE_DENSE<T>) {
#pragma unroll
        for (int s = 0; s < WIDE_STEPS; ++s) {
            if (!__any_sync(FULL_MASK, __popc(cm[s]) > WIDE_DENSE<T>)) continue;
            uint32_t r[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] = w[s].row(i) & cm[s];
            wide_add_dense<T, Sem>(acc[s / PER], r, (long long)tc[s] * T, x, ncols, lane);
            cm[s] = 0;
        }
        most = WIDE_DENSE<T>;
    }
#pragma unroll 1
    for (; most > 0; --most) {
        uint32_t b[WIDE_STEPS];
        V xv[WIDE_STEPS];
#pragma unroll
        for (int s = 0; s < WIDE_STEPS; ++s) {
            b[s] = cm[s] ? 0x80000000u >> __clz(cm[s]) : 0u;
            xv[s] = b[s] ? wide_x<Sem>(x, (long long)tc[s] * T, T - 32 + __clz(b[s]), ncols) : Sem::zero();
            cm[s] ^= b[s];
        }
#pragma unroll
        for (int s = 0; s < WIDE_STEPS; ++s) {
            V(&a)[4] = acc[s / PER];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (w[s].has(i, b[s])) a[i] = Sem::add(a[i], xv[s]);
        }
    }
}

// acc over the tiles of `n` neighbouring lane groups (lanes WIDE_LPT apart)
template <int T, class Sem, int N>
__device__ __forceinline__ void wide_reduce(typename Sem::V (&acc)[4]) {
#pragma unroll
    for (int o = N / 2; o >= 1; o >>= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            acc[i] = Sem::add(acc[i], __shfl_xor_sync(FULL_MASK, acc[i], o * WIDE_LPT<T>));
}

// Writes four rows of a task (t: row, -, -, out slot or -1).
template <int T, class Sem, class Args>
__device__ __forceinline__ void wide_store(const Args& a, int row, int out, int sub, typename Sem::V (&acc)[4]) {
    using V = typename Sem::V;
    const size_t off = (size_t)(out < 0 ? row : out) * T + 4 * sub;
    V* dst = static_cast<V*>(out < 0 ? a.y : a.partials) + off;
    if (out < 0 && a.mask) {
        const V* mk = static_cast<const V*>(a.mask) + off;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = Sem::clear(acc[i], mk[i]);
    }
    const bool add = out < 0 && a.accumulate;
    constexpr int PER = 16 / sizeof(V);
#pragma unroll
    for (int p = 0; p < 4 / PER; ++p) {
        uint4* d = reinterpret_cast<uint4*>(dst) + p;
        V o[PER];
#pragma unroll
        for (int e = 0; e < PER; ++e) o[e] = acc[p * PER + e];
        if (add) {
            const uint4 old = *d;
            const V* ov = reinterpret_cast<const V*>(&old);
#pragma unroll
            for (int e = 0; e < PER; ++e) o[e] = Sem::add(ov[e], o[e]);
        }
        *d = *reinterpret_cast<const uint4*>(o);
    }
}

template <int T, class Sem, int G, class Args>
__device__ __forceinline__ void wide_group(const Args& a, int task0, int tend) {
    using V = typename Sem::V;
    constexpr int LPT = WIDE_LPT<T>, TPS = WIDE_TPS<T>, NT = WIDE_PASS<T> / G;  // NT tasks per warp
    const int lane = threadIdx.x & 31, q = lane / LPT, sub = lane % LPT;
    const V* x = static_cast<const V*>(a.x);
    const int4 t = lane < NT && task0 + lane < tend ? __ldg(a.tasks + task0 + lane) : make_int4(0, 0, 0, -2);
    int j[WIDE_STEPS], tc[WIDE_STEPS];
    WideRows<T> w[WIDE_STEPS];
    wide_slots<T, G>(t.y, t.z, q, j);
#pragma unroll
    for (int s = 0; s < WIDE_STEPS; ++s) {
        tc[s] = 0;
        w[s].clear();
        if (j[s] >= 0) {
            tc[s] = __ldcs(a.colind + j[s]);
            w[s].load(a.tiles, j[s], sub);
        }
    }
    // a task's steps share an accumulator set when a task is longer than a step
    constexpr int NACC = G > TPS ? WIDE_PASS<T> / G : WIDE_STEPS;
    V acc[NACC][4];
#pragma unroll
    for (int n = 0; n < NACC; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = Sem::zero();
    wide_add<T, Sem, NACC>(acc, w, tc, x, a.ncols, lane);
#pragma unroll
    for (int n = 0; n < NACC; ++n) {
        constexpr int RED = G < TPS ? G : TPS;  // lane groups holding tiles of one task
        wide_reduce<T, Sem, RED>(acc[n]);
        const int ti = n * (NT / NACC) + q / RED;
        const int row = __shfl_sync(FULL_MASK, t.x, ti), out = __shfl_sync(FULL_MASK, t.w, ti);
        if (q % RED == 0 && out != -2) wide_store<T, Sem>(a, row, out, sub, acc[n]);
    }
}

// ---- long rows: the non-zero words of staged tiles, one per lane ------------------------------
// A stage is 2 KB of consecutive tiles (64 at T = 16, 16 at T = 32), 512 words,
// and their tile-columns, copied to shared memory by cp.async while the stage
// before it is worked on.  On R-MAT graphs some 30 (T = 32) to 90 (T = 16) of
// the words are non-zero, unevenly spread: rows of a tile-row differ in degree
// by up to 300x.  So the warp first lists the non-zero words (a 16-bit mask per
// lane, one scan), and then every lane takes words from the list in turn, finds
// their bits and loads their x elements: all lanes are busy whatever rows the
// bits are in.  A lane adds into its own copy of the T row sums in shared
// memory (bank = lane, so no conflicts, no atomics and a fixed order); the
// copies are summed when the task ends.
// From here on a stage goes column by column instead (wide_add_dense): more
// than DENSE_BITS set bits, counted when more than DENSE_WORDS words are
// non-zero.  (2000 instead of 1024: R-MAT scale 18 at T = 32 137 us, not 129.)
constexpr int DENSE_WORDS = 160, DENSE_BITS = 1024;
constexpr int STAGE_BYTES = 2048;
constexpr int STAGE_WORDS = STAGE_BYTES / 4;
template <int T> constexpr int STAGE_TILES = STAGE_BYTES * 8 / (T * T);
template <int T, class V> struct WideStage {
    uint4 tiles[2][STAGE_BYTES / 16];
    V sum[T * 32];  // row r, lane l at r * 32 + l
    int tc[2][STAGE_TILES<T>];
    uint16_t list[STAGE_WORDS];
};

__device__ __forceinline__ void cp_async16(void* s, const void* g, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
                 "r"(on ? 16 : 0));
}
__device__ __forceinline__ void cp_async4(void* s, const void* g, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g),
                 "r"(on ? 4 : 0));
}

// Starts the copy of tiles [j0, end) (at most a stage; past the end: zeros,
// with the source address kept inside the arrays).
template <int T, class V, class Args>
__device__ __forceinline__ void stage_start(const Args& a, WideStage<T, V>& st, int buf, int j0, int end, int lane) {
    constexpr int PER_TILE = T * T / 128;  // 16-byte units of a tile
#pragma unroll
    for (int u = 0; u < STAGE_BYTES / 16 / 32; ++u) {
        const int unit = u * 32 + lane;
        const bool on = j0 + unit / PER_TILE < end;
        cp_async16(&st.tiles[buf][unit],
                   static_cast<const uint4*>(a.tiles) + (on ? (size_t)j0 * PER_TILE + unit : (size_t)0), on);
    }
#pragma unroll
    for (int u = 0; u < (STAGE_TILES<T> + 31) / 32; ++u) {
        const int k = u * 32 + lane;
        const bool on = j0 + k < end;
        if (k < STAGE_TILES<T>) cp_async4(&st.tc[buf][k], a.colind + (on ? j0 + k : 0), on);
    }
    asm volatile("cp.async.commit_group;");
}

// A long row or segment: one task per warp, a stage after the other.
template <int T, class Sem, class Args>
__device__ __forceinline__ void wide_long(const Args& a, int task, WideStage<T, typename Sem::V>& st) {
    using V = typename Sem::V;
    constexpr int ST = STAGE_TILES<T>, TW = T * T / 32;  // words of a tile
    constexpr int LPT = WIDE_LPT<T>, TPS = WIDE_TPS<T>;
    const int lane = threadIdx.x & 31, q = lane / LPT, sub = lane % LPT;
    const V* __restrict__ x = static_cast<const V*>(a.x);
    const int4 t = __ldg(a.tasks + task);
    stage_start<T>(a, st, 0, t.y, t.z, lane);
#pragma unroll
    for (int r = 0; r < T; ++r) st.sum[r * 32 + lane] = Sem::zero();
    V acc[4];  // dense stages: rows 4*sub .. 4*sub+3 of every TPS-th tile
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = Sem::zero();
    int buf = 0;
#pragma unroll 1
    for (int j0 = t.y; j0 < t.z; j0 += ST, buf ^= 1) {
        stage_start<T>(a, st, buf ^ 1, j0 + ST, t.z, lane);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        uint32_t mask = 0;  // bit 4*u + e: word e of unit u*32 + lane
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint4 w = st.tiles[buf][u * 32 + lane];
            mask |= ((w.x ? 1u : 0u) | (w.y ? 2u : 0u) | (w.z ? 4u : 0u) | (w.w ? 8u : 0u)) << (4 * u);
        }
        const int own = __popc(mask);
        int inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL_MASK, inc, o);
            if (lane >= o) inc += v;
        }
        const int total = __shfl_sync(FULL_MASK, inc, 31);
        const uint32_t* words = reinterpret_cast<const uint32_t*>(st.tiles[buf]);
        if (total > DENSE_WORDS) {  // warp-uniform; so is the count below
            int bits = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint4 w = st.tiles[buf][u * 32 + lane];
                bits += __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
            }
            if (__reduce_add_sync(FULL_MASK, bits) > DENSE_BITS) {
#pragma unroll 1
                for (int tile = q; tile < ST; tile += TPS) {
                    uint32_t k[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        k[i] = T == 32 ? words[tile * 32 + 4 * sub + i]
                                       : reinterpret_cast<const uint16_t*>(words)[tile * 16 + 4 * sub + i];
                    wide_add_dense<T, Sem>(acc, k, (long long)st.tc[buf][tile] * T, x, a.ncols, lane);
                }
                __syncwarp();
                continue;
            }
        }
        uint16_t* out = st.list + (inc - own);
        while (mask) {
            const int b = __ffs(mask) - 1;
            mask &= mask - 1;
            *out++ = (uint16_t)((b >> 2) * 128 + lane * 4 + (b & 3));
        }
        __syncwarp();
#pragma unroll 1
        for (int i = lane; i < total; i += 32) {
            const int w = st.list[i];
            uint32_t bits = words[w];
            const int base = st.tc[buf][w / TW] * T;
            V* sum = st.sum + (T == 32 ? w % 32 : 2 * (w % TW)) * 32 + lane;
            // bit b: T = 32: column 31 - b; T = 16: row 2*(w % 8) + b/16, column 15 - b%16
            while (bits) {
                const int b0 = __ffs(bits) - 1;
                bits &= bits - 1;
                const int b1 = bits ? __ffs(bits) - 1 : b0;
                const bool two = bits != 0;
                bits &= bits - 1;
                const int c0 = base + T - 1 - (b0 & (T - 1)), c1 = base + T - 1 - (b1 & (T - 1));
                const V v0 = c0 < a.ncols ? __ldg(x + c0) : Sem::zero();
                const V v1 = two && c1 < a.ncols ? __ldg(x + c1) : Sem::zero();
                V* s0 = sum + (T == 32 ? 0 : (b0 >> 4) * 32);
                *s0 = Sem::add(*s0, v0);
                if (two) {
                    V* s1 = sum + (T == 32 ? 0 : (b1 >> 4) * 32);
                    *s1 = Sem::add(*s1, v1);
                }
            }
        }
        __syncwarp();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        V& mine = st.sum[(4 * sub + i) * 32 + lane];
        mine = Sem::add(mine, acc[i]);
    }
    __syncwarp();
    // row r: its 32 lane sums, from copy r on so that the lanes read 32 banks;
    // at T = 16 two lanes share a row
    const int r = lane % T, l0 = T == 32 ? 0 : (lane / T) * T;
    V p[4] = {Sem::zero(), Sem::zero(), Sem::zero(), Sem::zero()};
#pragma unroll
    for (int l = 0; l < T; ++l) p[l & 3] = Sem::add(p[l & 3], st.sum[r * 32 + l0 + ((l + r) & (T - 1))]);
    V s = Sem::add(Sem::add(p[0], p[1]), Sem::add(p[2], p[3]));
    if (T == 16) s = Sem::add(s, __shfl_xor_sync(FULL_MASK, s, 16));
    __syncwarp();
    if (lane >= T) return;
    const size_t off = (size_t)(t.w < 0 ? t.x : t.w) * T + r;
    if (t.w >= 0) {
        static_cast<V*>(a.partials)[off] = s;
        return;
    }
    if (a.mask) s = Sem::clear(s, static_cast<const V*>(a.mask)[off]);
    V* y = static_cast<V*>(a.y) + off;
    *y = a.accumulate ? Sem::add(*y, s) : s;
}

// ---- bit vectors ------------------------------------------------------------------------
// Whether most x words are zero, judged on 32 words spread over x (the same
// for every warp, so they stay in L1): then a tile is loaded only after its x
// word is known not to be zero.  That costs a dependent load, and saves the
// tile's bytes: either choice gives the same words and counts.
template <typename W>
__device__ __forceinline__ bool mostly_zero(const W* __restrict__ x, int nbc) {
    const int lane = threadIdx.x & 31;
    const bool on = nbc > 0 && __ldg(x + (int)((long long)lane * nbc >> 5)) != 0;
    return __popc(__ballot_sync(FULL_MASK, on)) <= 16;
}

template <int T>
__device__ __forceinline__ void wide_bits_load(const int* colind, const void* tiles, const void* x, bool skip,
                                               const int (&j)[WIDE_STEPS], int sub, WideRows<T> (&w)[WIDE_STEPS],
                                               uint32_t (&xw)[WIDE_STEPS]) {
    using W = typename TileWord<T>::type;
    int tc[WIDE_STEPS];
#pragma unroll
    for (int s = 0; s < WIDE_STEPS; ++s) {
        tc[s] = j[s] >= 0 ? __ldcs(colind + j[s]) : -1;
        w[s].clear();
        if (!skip && j[s] >= 0) w[s].load(tiles, j[s], sub);
    }
#pragma unroll
    for (int s = 0; s < WIDE_STEPS; ++s) xw[s] = tc[s] >= 0 ? (uint32_t)__ldg(static_cast<const W*>(x) + tc[s]) : 0u;
    if (skip) {
#pragma unroll
        for (int s = 0; s < WIDE_STEPS; ++s)
            if (xw[s]) w[s].load(tiles, j[s], sub);
    }
}

// Combines and writes one task's words or counts; RED lane groups hold its tiles.
template <int T, int KIND, int RED, class Args>
__device__ __forceinline__ void wide_bits_store(const Args& a, int row, int out, int q, int sub, uint32_t m,
                                                int (&acc)[4]) {
    using W = typename TileWord<T>::type;
    constexpr int LPT = WIDE_LPT<T>;
    const bool writer = q % RED == 0 && out != -2;
    if constexpr (KIND <= 1) {
        m <<= T - 4 - 4 * sub;  // row 4*sub + k at bit T-1-4*sub-k
#pragma unroll
        for (int o = RED * LPT / 2; o >= 1; o >>= 1) m |= __shfl_xor_sync(FULL_MASK, m, o);
        if (!writer || sub != 0) return;
        if (out >= 0) {
            static_cast<uint32_t*>(a.partials)[out] = m;
            return;
        }
        W* y = static_cast<W*>(a.y) + row;
        if (KIND == 1) m &= ~(uint32_t)__ldg(static_cast<const W*>(a.mask) + row);
        *y = (W)(a.accumulate ? ((uint32_t)*y | m) : m);
    } else {
#pragma unroll
        for (int o = RED / 2; o >= 1; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(FULL_MASK, acc[i], o * LPT);
        if (!writer) return;
        const size_t off = (size_t)(out < 0 ? row : out) * T + 4 * sub;
        // y is only known to be 4-byte aligned here
        if (out >= 0) {
            *reinterpret_cast<int4*>(static_cast<int*>(a.partials) + off) = make_int4(acc[0], acc[1], acc[2], acc[3]);
        } else if constexpr (KIND == 2) {
            int* dst = static_cast<int*>(a.y) + off;
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = a.accumulate ? dst[i] + acc[i] : acc[i];
        } else {
            float* dst = static_cast<float*>(a.y) + off;
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = a.accumulate ? dst[i] + (float)acc[i] : (float)acc[i];
        }
    }
}

template <int T, int KIND, int G, class Args>
__device__ __forceinline__ void wide_bits_group(const Args& a, int task0, int tend, bool skip) {
    constexpr int LPT = WIDE_LPT<T>, TPS = WIDE_TPS<T>, NT = WIDE_PASS<T> / G;
    const int lane = threadIdx.x & 31, q = lane / LPT, sub = lane % LPT;
    const int4 t = lane < NT && task0 + lane < tend ? __ldg(a.tasks + task0 + lane) : make_int4(0, 0, 0, -2);
    int j[WIDE_STEPS];
    uint32_t xw[WIDE_STEPS];
    WideRows<T> w[WIDE_STEPS];
    wide_slots<T, G>(t.y, t.z, q, j);
    wide_bits_load<T>(a.colind, a.tiles, a.x, skip, j, sub, w, xw);
    constexpr int PER = G > TPS ? G / TPS : 1;  // steps of one task
    constexpr int RED = G < TPS ? G : TPS;
#pragma unroll
    for (int n = 0; n < WIDE_STEPS / PER; ++n) {
        uint32_t m = 0;
        int acc[4] = {0, 0, 0, 0};
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            const int s = n * PER + p;
            if constexpr (KIND <= 1) m |= w[s].hits(xw[s]);
            else w[s].add_counts(acc, xw[s]);
        }
        const int ti = (n * PER * TPS + q) / G;
        const int row = __shfl_sync(FULL_MASK, t.x, ti), out = __shfl_sync(FULL_MASK, t.w, ti);
        wide_bits_store<T, KIND, RED>(a, row, out, q, sub, m, acc);
    }
}

template <int T, int KIND, class Args>
__device__ __forceinline__ void wide_bits_long(const Args& a, int task, bool skip) {
    constexpr int LPT = WIDE_LPT<T>, TPS = WIDE_TPS<T>;
    const int lane = threadIdx.x & 31, q = lane / LPT, sub = lane % LPT;
    const int4 t = __ldg(a.tasks + task);
    uint32_t m = 0;
    int acc[4] = {0, 0, 0, 0};
#pragma unroll 1
    for (int j0 = t.y; j0 < t.z; j0 += WIDE_PASS<T>) {
        int j[WIDE_STEPS];
        uint32_t xw[WIDE_STEPS];
        WideRows<T> w[WIDE_STEPS];
#pragma unroll
        for (int s = 0; s < WIDE_STEPS; ++s) {
            j[s] = j0 + s * TPS + q;
            if (j[s] >= t.z) j[s] = -1;
        }
        wide_bits_load<T>(a.colind, a.tiles, a.x, skip, j, sub, w, xw);
#pragma unroll
        for (int s = 0; s < WIDE_STEPS; ++s) {
            if constexpr (KIND <= 1) m |= w[s].hits(xw[s]);
            else w[s].add_counts(acc, xw[s]);
        }
    }
    wide_bits_store<T, KIND, TPS>(a, t.x, t.w, q, sub, m, acc);
}

}  // namespace b2sr
