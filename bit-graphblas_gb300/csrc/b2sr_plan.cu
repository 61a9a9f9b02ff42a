// Task lists of the row-binned and the row-task kernels, built on the device
// from the tile-row pointer.
//
// A tile-row becomes one task, or several segments when it is long; tasks are
// listed by class (bin, or size), tile-rows ascending inside a class.  That is a
// stable multi-way split of the tile-rows with a weight each: counts per
// (class, block of 256 tile-rows), one exclusive scan over all of them, and a
// second pass in which every tile-row adds its rank inside the block.  The same
// scan places the segments' slots and the list of long rows, so a plan costs
// one wait, for its totals.
//
// On the host (a download of rowptr, vectors per class, an upload) R-MAT scale
// 20 at T = 4 took 2.2 ms for the row-binned plan and 2.3 ms for the dense-RHS
// one; here 0.09 and 0.10 ms on GB300.
#include <algorithm>

#include "b2sr_common.cuh"

namespace b2sr {

namespace {

constexpr int PLAN_ROWS = 256;  // tile-rows per block, one per thread
constexpr int PLAN_WARPS = PLAN_ROWS / 32;

// What becomes of one tile-row.
struct RowTasks {
    int b0, m;   // its tiles
    int nseg;    // tasks; more than one: segments with a slot each
    int cls;     // class of its tasks
    bool narrow; // long row listed before the others
};

// Size classes, largest first: two per octave.
__device__ __forceinline__ int size_class(long long v) {
    if (v <= 0) return PLAN_CLASSES - 1;
    const int e = 63 - __clzll(v);
    const int sub = e >= 1 ? (int)(v >> (e - 1)) & 1 : 0;
    return max(PLAN_CLASSES - 1 - (2 * e + sub), 0);
}

__device__ __forceinline__ RowTasks row_tasks(const PlanRule& r, const int* __restrict__ rowptr, int i, int nb) {
    RowTasks t{0, 0, 0, 0, false};
    if (i >= nb) return t;
    t.b0 = rowptr[i];
    t.m = rowptr[i + 1] - t.b0;
    t.nseg = t.m > max(r.seg, r.whole) ? (t.m - 1) / r.seg + 1 : 1;
    if (r.kind == PlanRule::BINS) {
        int b = 0;
        while (b < r.nbins - 1 && t.m > (r.unit << b)) ++b;
        t.cls = r.nbins - 1 - b;
        t.narrow = t.nseg <= r.narrow_slots;
        return t;
    }
    long long bits = 0;
    if (r.row_bits) {
        bits = r.row_bits[i];
        const long long by_bits = bits > r.whole_bits ? (bits + r.seg_bits - 1) / r.seg_bits : 1;
        t.nseg = (int)min((long long)max(t.m, 1), max((long long)t.nseg, by_bits));
    }
    t.narrow = t.nseg <= r.narrow_slots;
    const int len = (t.m + t.nseg - 1) / t.nseg;  // of a segment
    if (r.kind == PlanRule::TWO) t.cls = 4LL * len >= r.seg ? 0 : 1;
    else t.cls = size_class(bits / t.nseg);
    return t;
}

// Counters after the classes: slots, narrow long rows, other long rows.
enum { C_SLOTS = 0, C_NARROW = 1, C_LONG = 2, C_EXTRA = 3 };

__global__ void __launch_bounds__(PLAN_ROWS)
plan_count_kernel(PlanRule rule, const int* __restrict__ rowptr, int nb, int nblocks, int* __restrict__ hist) {
    __shared__ int cnt[PLAN_CLASSES + C_EXTRA];
    for (int k = threadIdx.x; k < rule.classes + C_EXTRA; k += blockDim.x) cnt[k] = 0;
    __syncthreads();
    const int i = blockIdx.x * PLAN_ROWS + threadIdx.x;
    const RowTasks t = row_tasks(rule, rowptr, i, nb);
    if (i < nb) {
        atomicAdd(&cnt[t.cls], t.nseg);
        if (t.nseg > 1) {
            atomicAdd(&cnt[rule.classes + C_SLOTS], t.nseg);
            atomicAdd(&cnt[rule.classes + (t.narrow ? C_NARROW : C_LONG)], 1);
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < rule.classes + C_EXTRA; k += blockDim.x)
        hist[(long long)k * nblocks + blockIdx.x] = cnt[k];
}

__global__ void __launch_bounds__(PLAN_ROWS)
plan_emit_kernel(PlanRule rule, const int* __restrict__ rowptr, int nb, int nblocks, const int* __restrict__ offs,
                 PlanOut out) {
    __shared__ int wcnt[PLAN_WARPS][PLAN_CLASSES];  // tasks of a class in the warps before
    __shared__ int wextra[PLAN_WARPS][C_EXTRA];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = lane; k < rule.classes; k += 32) wcnt[warp][k] = 0;
    __syncwarp();
    const int i = blockIdx.x * PLAN_ROWS + threadIdx.x;
    const RowTasks t = row_tasks(rule, rowptr, i, nb);
    const bool on = i < nb, cut = on && t.nseg > 1;
    // rank among the warp's tile-rows of the class: one task each, plus the
    // further segments of the long ones
    const unsigned below = (1u << lane) - 1u;
    const unsigned peers = __match_any_sync(FULL_MASK, on ? t.cls : -1);
    int rank = __popc(peers & below), more = 0;
    for (unsigned c = __ballot_sync(FULL_MASK, cut); c; c &= c - 1) {
        const int l = __ffs(c) - 1, extra = __shfl_sync(FULL_MASK, t.nseg, l) - 1;
        if ((peers >> l) & 1u) {
            if (l < lane) rank += extra;
            more += extra;
        }
    }
    if (on && (peers & below) == 0) wcnt[warp][t.cls] = __popc(peers) + more;
    int pre[C_EXTRA] = {cut ? t.nseg : 0, cut && t.narrow ? 1 : 0, cut && !t.narrow ? 1 : 0};
#pragma unroll
    for (int x = 0; x < C_EXTRA; ++x) {
        const int own = pre[x];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL_MASK, pre[x], o);
            if (lane >= o) pre[x] += v;
        }
        if (lane == 31) wextra[warp][x] = pre[x];
        pre[x] -= own;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < rule.classes + C_EXTRA; k += blockDim.x) {
        int* col = k < rule.classes ? &wcnt[0][k] : &wextra[0][k - rule.classes];
        const int stride = k < rule.classes ? PLAN_CLASSES : C_EXTRA;
        int s = 0;
        for (int w = 0; w < PLAN_WARPS; ++w) {
            const int v = col[w * stride];
            col[w * stride] = s;
            s += v;
        }
    }
    __syncthreads();
    // totals for the host: first task of every class, then the extra counters' starts, then the end
    if (blockIdx.x == 0)
        for (int k = threadIdx.x; k <= rule.classes + C_EXTRA; k += blockDim.x) out.info[k] = offs[(long long)k * nblocks];
    auto at = [&](int k) { return offs[(long long)k * nblocks + blockIdx.x]; };
    const int first_slot = offs[(long long)(rule.classes + C_SLOTS) * nblocks];
    const int first_long = offs[(long long)(rule.classes + C_NARROW) * nblocks];
    int task = 0, slot = -1;
    if (on) task = at(t.cls) + wcnt[warp][t.cls] + rank;
    if (cut) {
        slot = at(rule.classes + C_SLOTS) - first_slot + wextra[warp][C_SLOTS] + pre[C_SLOTS];
        const int x = t.narrow ? C_NARROW : C_LONG;
        const int lr = at(rule.classes + x) - first_long + wextra[warp][x] + pre[x];
        if (lr < out.cap_long) out.longs[lr] = make_int4(i, slot, t.nseg, 0);
    }
    auto emit = [&](int row, int b0, int m, int nseg, int task, int slot, int q) {
        int t0, t1;
        if (rule.kind == PlanRule::BINS) {  // whole segments, the last one shorter
            t0 = b0 + q * rule.seg;
            t1 = min(t0 + rule.seg, b0 + m);
        } else {  // near-equal segments
            t0 = b0 + (int)((long long)m * q / nseg);
            t1 = b0 + (int)((long long)m * (q + 1) / nseg);
        }
        if (task + q < out.cap_tasks) out.tasks[task + q] = make_int4(row, t0, t1, slot < 0 ? -1 : slot + q);
    };
    if (on && t.nseg <= 4)
        for (int q = 0; q < t.nseg; ++q) emit(i, t.b0, t.m, t.nseg, task, slot, q);
    // long rows by the whole warp
    for (unsigned c = __ballot_sync(FULL_MASK, on && t.nseg > 4); c; c &= c - 1) {
        const int l = __ffs(c) - 1;
        const int row = __shfl_sync(FULL_MASK, i, l), b0 = __shfl_sync(FULL_MASK, t.b0, l),
                  m = __shfl_sync(FULL_MASK, t.m, l), nseg = __shfl_sync(FULL_MASK, t.nseg, l),
                  tk = __shfl_sync(FULL_MASK, task, l), sl = __shfl_sync(FULL_MASK, slot, l);
        for (int q = lane; q < nseg; q += 32) emit(row, b0, m, nseg, tk, sl, q);
    }
}

}  // namespace

// Upper bounds of a valid matrix; a rowptr that is not monotone (wrapped
// arrays are not checked) can ask for more, which the kernels do not write and
// which is reported.
PlanBounds plan_bounds(const PlanRule& r, int nb, long long nt, long long bits) {
    const long long cuts = nt / r.seg + (r.row_bits ? bits / r.seg_bits : 0);
    return {nb + cuts, std::min<long long>(nb, cuts), 2 * cuts};
}

b2sr_status build_plan(const PlanRule& rule, const int* rowptr, int nb, const PlanBounds& cap, int4* tasks, int4* longs,
                       PlanTotals* totals, cudaStream_t s) {
    const int nblocks = (nb + PLAN_ROWS - 1) / PLAN_ROWS;
    const long long n = (long long)(rule.classes + C_EXTRA) * nblocks;
    // every return waits for `s`: the caller frees row_bits, which kernels that
    // it has queued may still be writing
    if (n > INT_MAX || cap.tasks > INT_MAX || cap.slots > INT_MAX) {
        cudaStreamSynchronize(s);
        return B2SR_ERR_OVERFLOW;
    }
    int* info = nullptr;
    const size_t info_ints = 128;
    static_assert(PLAN_CLASSES + C_EXTRA + 2 <= 128, "totals and the overflow flag");
    const size_t hist_bytes = (sizeof(int) * ((size_t)n + 1) + 255) / 256 * 256;
    char* scratch = static_cast<char*>(dev_alloc(sizeof(int) * info_ints + hist_bytes + exclusive_scan_scratch(n)));
    if (!scratch) {
        cudaStreamSynchronize(s);
        return B2SR_ERR_ALLOC;
    }
    info = reinterpret_cast<int*>(scratch);
    int* hist = reinterpret_cast<int*>(scratch + sizeof(int) * info_ints);
    int* err = info + info_ints - 1;
    int h[info_ints] = {0};
    cudaError_t e = cudaMemsetAsync(info, 0, sizeof(int) * info_ints, s);
    if (e == cudaSuccess && nb > 0) {
        plan_count_kernel<<<nblocks, PLAN_ROWS, 0, s>>>(rule, rowptr, nb, nblocks, hist);
        exclusive_scan_async(hist, (int)n, err, scratch + sizeof(int) * info_ints + hist_bytes, s);
        const PlanOut out{tasks, longs, info, (int)cap.tasks, (int)cap.longs};
        plan_emit_kernel<<<nblocks, PLAN_ROWS, 0, s>>>(rule, rowptr, nb, nblocks, hist, out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, info, sizeof h, cudaMemcpyDeviceToHost, s);
    const cudaError_t drained = cudaStreamSynchronize(s);
    dev_free(scratch);
    if (e == cudaSuccess) e = drained;
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return B2SR_ERR_CUDA;
    }
    for (int k = 0; k <= rule.classes; ++k) totals->first[k] = h[k];
    totals->tasks = h[rule.classes];
    totals->slots = h[rule.classes + C_NARROW] - h[rule.classes + C_SLOTS];
    totals->narrow = h[rule.classes + C_LONG] - h[rule.classes + C_NARROW];
    totals->longs = h[rule.classes + C_EXTRA] - h[rule.classes + C_NARROW];
    if (h[info_ints - 1] != 0 || totals->tasks > cap.tasks || totals->longs > cap.longs || totals->slots > cap.slots)
        return B2SR_ERR_INVALID_VALUE;
    return B2SR_SUCCESS;
}

}  // namespace b2sr
