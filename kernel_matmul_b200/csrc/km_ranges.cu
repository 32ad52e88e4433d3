// Band construction on the device: start/end column per 128-row block.
//
// The reference computes these with sequential scans on one CPU thread after copying x to the
// host (native/ranges/ranges.cpp:8-150), which puts a device synchronisation into every kernel
// forward.  Here nothing leaves the device and nothing synchronises.
//
// Parallel formulation.  Every scan of the reference has the form "first grid position
// j >= j0 for which pred_i(j) holds, else n", where the grid is {0, step, 2 step, ..} below n
// and j0 is the result of the previous row block.  When x2 is non-decreasing, pred_i is
// monotone in j (fp32 subtraction and comparison are monotone), so that position is
// max(j0, first_i) with first_i found by binary search over the grid, and the recurrences
// over row blocks turn into prefix maxima:
//   make_ranges:            start[i] = max_{i' <= i} lb_i' ;  end[i] = max(start[i], max_{i' <= i} ub_i')
//   make_ranges_symmetric:  end[i] = max(block, max_{i' <= i} ub_i') ;
//                           start[k] = block * (first i <= k with ceil(end[i] / block) > k), else n
// with every predicate evaluated in fp32 exactly as the reference writes it.  Monotonicity
// is checked per batch row (NaNs count as unsorted); batch rows that fail it are processed by a
// sequential scan that restates the reference loop, so the int32 results are bit-identical to the
// reference for every input.
#include "km_common.cuh"

namespace km {

// First grid index t in [0, G) with pred(t * step), else G.  pred monotone (false.. true..).
template <typename Pred>
__device__ __forceinline__ int64_t first_true(int64_t G, Pred pred) {
    int64_t lo = 0, hi = G;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (pred(mid)) hi = mid; else lo = mid + 1;
    }
    return lo;
}

// One band construction.  mode 0 = make_ranges, mode 1 = symmetric (only upper bounds, predicate
// with >=).  `cutoffs` (device, B values) overrides the scalar when not null; x1s / x2s: elements
// between batch rows of x (0: one row shared by all).
struct RangesArgs {
    int64_t B, m, n, R;
    const float *x1, *x2;
    int64_t x1s, x2s;
    float cutoff_scalar;
    const float *cutoffs;
    int block, step, mode;
    int32_t *start, *end;
    int32_t *unsorted;  // per batch row: non-zero if x2 is not non-decreasing
};

// lb (first grid column within cutoff below the block's first row) and ub (first grid column beyond
// cutoff above the block's last row) of row block i, written to start / end as scratch.
__device__ __forceinline__ void row_block_bounds(const RangesArgs &q, int64_t b, int64_t i) {
    const float cutoff = q.cutoffs ? q.cutoffs[b] : q.cutoff_scalar;
    const float *a = q.x1 + b * q.x1s;
    const float *c = q.x2 + b * q.x2s;
    const int64_t idx = b * q.R + i, step = q.step;
    const int64_t G = (q.n + step - 1) / step;
    const float last = a[min((i + 1) * (int64_t)q.block, q.m) - 1];
    if (q.mode == 0) {
        const float first = a[i * q.block];
        const int64_t tl = first_true(G, [&](int64_t t) { return first - c[t * step] <= cutoff; });
        const int64_t tu = first_true(G, [&](int64_t t) { return c[t * step] - last > cutoff; });
        q.start[idx] = (int32_t)min(tl * step, q.n);
        q.end[idx] = (int32_t)min(tu * step, q.n);
    } else {
        const int64_t tu = first_true(G, [&](int64_t t) { return c[t * step] - last >= cutoff; });
        q.end[idx] = (int32_t)min(tu * step, q.n);
    }
}

// Inclusive-to-exclusive prefix maxima over the 1024 threads of the CTA of two values at once.
__device__ __forceinline__ void block_exclusive_max2(int &v, int &w, int *warp_v, int *warp_w) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int yv = __shfl_up_sync(0xffffffffu, v, o), yw = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) v = max(v, yv), w = max(w, yw);
    }
    if (lane == 31) warp_v[warp] = v, warp_w[warp] = w;
    v = __shfl_up_sync(0xffffffffu, v, 1), w = __shfl_up_sync(0xffffffffu, w, 1);
    if (lane == 0) v = w = INT_MIN;
    __syncthreads();
    for (int p = 0; p < warp; p++) v = max(v, warp_v[p]), w = max(w, warp_w[p]);
}

// Prefix maxima of a batch row and, in the symmetric mode, the starts, by one CTA of 1024 threads:
// every thread owns R / 1024 consecutive row blocks.  The symmetric start of column block k is the
// first row block whose end reaches past k: row block i therefore WRITES the starts of the column
// blocks its end adds to those reached before, R writes altogether (a binary search per column
// block over the finished ends took a launch of its own).
__device__ __forceinline__ void finish_row(const RangesArgs &q, int64_t b, int *warp_v, int *warp_w) {
    const int64_t R = q.R, chunk = (R + blockDim.x - 1) / blockDim.x;
    const int64_t i0 = min(R, threadIdx.x * chunk), i1 = min(R, i0 + chunk);
    int32_t *S = q.start + b * R, *E = q.end + b * R;
    int v = INT_MIN, w = INT_MIN;
    for (int64_t i = i0; i < i1; i++) {
        w = max(w, E[i]);
        if (q.mode == 0) v = max(v, S[i]);
    }
    block_exclusive_max2(v, w, warp_v, warp_w);
    if (q.mode == 0) {
        for (int64_t i = i0; i < i1; i++) {
            v = max(v, S[i]);
            w = max(w, E[i]);
            S[i] = v;
            E[i] = max(v, w);
        }
        return;
    }
    w = max(w, q.block);
    const auto reach_of = [&](int e) { return ((int64_t)e + q.block - 1) / q.block; };
    int64_t reach = i0 == 0 ? 0 : reach_of(w);
    for (int64_t i = i0; i < i1; i++) {
        w = max(w, E[i]);
        E[i] = w;
        const int64_t next = reach_of(w);
        for (int64_t k = reach; k < min(next, R); k++) S[k] = k == 0 ? 0 : (i <= k ? (int32_t)(i * q.block) : (int32_t)q.n);
        reach = next;
    }
    if (i0 < i1 && i1 == R)  // column blocks that no row block reaches
        for (int64_t k = reach; k < R; k++) S[k] = k == 0 ? 0 : (int32_t)q.n;
}

// Sequential restatement of the reference scans for a batch row whose x2 is not sorted
// (native/ranges/ranges.cpp:24-59 and :76-97).  One thread.
__device__ void sequential_row(const RangesArgs &q, int64_t b) {
    const float cutoff = q.cutoffs ? q.cutoffs[b] : q.cutoff_scalar;
    const float *a = q.x1 + b * q.x1s;
    const float *c = q.x2 + b * q.x2s;
    const int64_t R = q.R, m = q.m, n = q.n, block = q.block, step = q.step;
    int32_t *S = q.start + b * R, *E = q.end + b * R;
    if (q.mode == 0) {
        int64_t ps = 0, pe = 0;
        for (int64_t i = 0; i < R; i++) {
            const float first = a[i * block];
            const float last = a[min((i + 1) * block, m) - 1];
            int64_t j = ps;
            while (j < n && !(first - c[j] <= cutoff)) j = min(j + step, n);
            int64_t t = max(pe, j);
            while (t < n && !(c[t] - last > cutoff)) t = min(t + step, n);
            S[i] = (int32_t)j;
            E[i] = (int32_t)t;
            ps = j;
            pe = t;
        }
    } else {
        for (int64_t i = 0; i < R; i++) S[i] = (int32_t)n;
        if (R > 0) S[0] = 0;
        int64_t j = block;
        for (int64_t i = 0; i < R; i++) {
            const float last = a[min((i + 1) * block, n) - 1];
            while (j < n && !(c[j] - last >= cutoff)) j = min(j + block, n);
            E[i] = (int32_t)j;
            const int64_t reach = (j + block - 1) / block;
            for (int64_t t = i; t < reach && t < R; t++) S[t] = min(S[t], (int32_t)(i * block));
        }
    }
}

// The whole construction of one batch row by one CTA: what a training step on up to RANGES_ONE_CTA_N
// points pays is launches, not work (five of them, 11 us of device time and as much host time,
// before; one, about 5 us, now).
__global__ void __launch_bounds__(1024) ranges_one_cta_kernel(const RangesArgs q) {
    __shared__ int warp_v[32], warp_w[32];
    const int64_t b = blockIdx.x;
    const float *c = q.x2 + b * q.x2s;
    int unsorted = 0;
#pragma unroll 4
    for (int64_t j = threadIdx.x; j + 1 < q.n; j += 1024) unsorted |= !(c[j] <= c[j + 1]);
    for (int64_t i = threadIdx.x; i < q.R; i += 1024) row_block_bounds(q, b, i);
    if (__syncthreads_or(unsorted)) {
        if (threadIdx.x == 0) sequential_row(q, b);
        return;
    }
    finish_row(q, b, warp_v, warp_w);
}

// Larger batch rows: sorted check and bounds by the whole GPU (q.unsorted is zero on entry), ...
__global__ void __launch_bounds__(256) ranges_bounds_kernel(const RangesArgs q) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t w = first; w < q.B * q.R; w += stride) row_block_bounds(q, w / q.R, w % q.R);
    const int64_t rows = q.x2s == 0 ? 1 : q.B;  // a shared x2 is checked once, for all batch rows
    for (int64_t b = 0; b < rows; b++) {
        const float *c = q.x2 + b * q.x2s;
        int unsorted = 0;
        for (int64_t j = first; j + 1 < q.n; j += stride) unsorted |= !(c[j] <= c[j + 1]);
        if (unsorted) q.unsorted[b] = 1;
    }
}

// ... then one CTA per batch row.
__global__ void __launch_bounds__(1024) ranges_finish_kernel(const RangesArgs q) {
    __shared__ int warp_v[32], warp_w[32];
    const int64_t b = blockIdx.x;
    if (q.unsorted[q.x2s == 0 ? 0 : b]) {
        if (threadIdx.x == 0) sequential_row(q, b);
        return;
    }
    finish_row(q, b, warp_v, warp_w);
}

// transpose: every row block marks the column blocks it touches (integer atomic min / max
// commute, so the result does not depend on the order).
__global__ void transpose_mark_kernel(int64_t B, int64_t R, int64_t C, const int32_t *start, const int32_t *end,
                                      int x1_size, int block, int32_t *start_t, int32_t *end_t) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= B * R) return;
    const int64_t b = idx / R, r = idx % R;
    const int s = start[idx], e = end[idx];
    if (s == e) return;
    const int64_t c0 = s / block;
    const int64_t c1 = ((int64_t)e + block - 1) / block;
    const int row0 = (int)(r * block);
    const int row1 = min(row0 + block, x1_size);
    for (int64_t c = max(c0, (int64_t)0); c < c1 && c < C; c++) {
        atomicMin(start_t + b * C + c, row0);
        atomicMax(end_t + b * C + c, row1);
    }
}

__global__ void transpose_init_kernel(int64_t total, int x1_size, int32_t *start_t, int32_t *end_t) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx < total) {
        start_t[idx] = x1_size;
        end_t[idx] = 0;
    }
}

// Untouched column blocks take the start of the nearest touched block to their left (0 if
// none) as an empty range (native/ranges/ranges.cpp:136-146).  One CTA per batch; a chunked
// scan carries the last touched start.
__global__ void __launch_bounds__(1024) transpose_fix_kernel(int64_t C, int x1_size, int32_t *start_t,
                                                              int32_t *end_t) {
    __shared__ int warp_last[32];
    __shared__ int carry;
    int32_t *S = start_t + blockIdx.x * C, *E = end_t + blockIdx.x * C;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = -1;  // index of the last touched block seen so far
    __syncthreads();
    for (int64_t base = 0; base < C; base += 1024) {
        const int64_t c = base + threadIdx.x;
        const int sv = c < C ? S[c] : x1_size;
        const bool touched = c < C && sv != x1_size;
        int last = touched ? (int)c : -1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, last, o);
            if (lane >= o) last = max(last, y);
        }
        if (lane == 31) warp_last[warp] = last;
        __syncthreads();
        int pre = carry;
        for (int q = 0; q < warp; q++) pre = max(pre, warp_last[q]);
        last = max(last, pre);
        __syncthreads();
        if (threadIdx.x == 1023) carry = last;
        // S[last] for last < c is a touched block and is never rewritten, so reading it here is safe
        if (c < C && !touched) {
            const int v = last >= 0 ? S[last] : 0;
            S[c] = v;
            E[c] = v;
        }
        __syncthreads();
    }
}

// One CTA reads 65 536 points in about 3 us; from there on the whole GPU is the faster way.
constexpr int64_t RANGES_ONE_CTA_N = 1 << 16;

// One thread per item on at most 2^20 blocks of 256 threads: callers refuse more items.
constexpr int64_t KM_RANGES_MAX_ITEMS = (1LL << 20) * 256;
static inline unsigned grid_for(int64_t total, int threads) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(total, threads), 1 << 20));
}

static int make_ranges_common(const char *name, int64_t B, int64_t m, int64_t n, const float *x1, int64_t x1s,
                              const float *x2, int64_t x2s, float cutoff, const float *cutoffs, int block, int step,
                              int mode, int32_t *start, int32_t *end, int32_t *flags, cudaStream_t s) {
    KM_REQUIRE(B >= 0 && m >= 0 && n >= 0 && n <= 0x7fffffffLL - 2 * (int64_t)block && m <= 0x7fffffffLL,
               KM_ERR_INVALID_ARGUMENT, "%s: bad sizes", name);
    KM_REQUIRE(block >= 1, KM_ERR_INVALID_ARGUMENT, "%s: block_size must be >= 1", name);
    const int64_t R = ceil_div(m, block);
    if (B == 0 || R == 0) return KM_OK;
    KM_REQUIRE(x1 && x2 && start && end && flags, KM_ERR_INVALID_ARGUMENT, "%s: null pointer", name);
    KM_REQUIRE(B <= 0x7fffffffLL, KM_ERR_UNSUPPORTED, "%s: too many batch rows", name);
    // (the per-element kernels run one thread per (batch row, row block) on grids of at most 2^20 blocks)
    KM_REQUIRE(B <= KM_RANGES_MAX_ITEMS / R, KM_ERR_UNSUPPORTED, "%s: more than %lld (batch row, row block) pairs", name,
               (long long)KM_RANGES_MAX_ITEMS);
    const RangesArgs q = {B, m, n, R, x1, x2, x1s, x2s, cutoff, cutoffs, block, step, mode, start, end, flags};
    if (n <= RANGES_ONE_CTA_N && R <= RANGES_ONE_CTA_N) {
        ranges_one_cta_kernel<<<(unsigned)B, 1024, 0, s>>>(q);
    } else {
        const cudaError_t err = cudaMemsetAsync(flags, 0, (size_t)B * sizeof(int32_t), s);
        if (err != cudaSuccess) return cuda_fail(err, name);
        const int64_t threads = std::max<int64_t>(B * R, n);
        ranges_bounds_kernel<<<(unsigned)std::min<int64_t>(ceil_div(threads, 256), 148 * 8), 256, 0, s>>>(q);
        ranges_finish_kernel<<<(unsigned)B, 1024, 0, s>>>(q);
    }
    KM_CHECK_LAUNCH(name);
    return KM_OK;
}

}  // namespace km

extern "C" int km_make_ranges_f32(int64_t B, int64_t m, int64_t n, const float *x1, const float *x2, float cutoff,
                                  int32_t block_size, int32_t align, int32_t *start, int32_t *end, int32_t *flags,
                                  void *stream) {
    return km::make_ranges_common("km_make_ranges_f32", B, m, n, x1, m, x2, n, cutoff, nullptr, block_size,
                                  align ? block_size : 1, 0, start, end, flags, static_cast<cudaStream_t>(stream));
}

extern "C" int km_make_ranges_symmetric_f32(int64_t B, int64_t n, const float *x, float cutoff, int32_t block_size,
                                            int32_t *start, int32_t *end, int32_t *flags, void *stream) {
    return km::make_ranges_common("km_make_ranges_symmetric_f32", B, n, n, x, n, x, n, cutoff, nullptr, block_size,
                                  block_size, 1, start, end, flags, static_cast<cudaStream_t>(stream));
}

extern "C" int km_make_ranges_symmetric_cutoffs_f32(int64_t B, int64_t n, const float *x, int64_t x_batch_stride,
                                                    const float *cutoffs, int32_t block_size, int32_t *start,
                                                    int32_t *end, int32_t *flags, void *stream) {
    KM_REQUIRE(cutoffs != nullptr || B == 0, KM_ERR_INVALID_ARGUMENT, "km_make_ranges_symmetric_cutoffs_f32: null cutoffs");
    KM_REQUIRE(x_batch_stride == 0 || x_batch_stride >= n, KM_ERR_INVALID_ARGUMENT,
               "km_make_ranges_symmetric_cutoffs_f32: x_batch_stride must be 0 (shared x) or at least n");
    return km::make_ranges_common("km_make_ranges_symmetric_cutoffs_f32", B, n, n, x, x_batch_stride, x, x_batch_stride,
                                  0.0f, cutoffs, block_size, block_size, 1, start, end, flags,
                                  static_cast<cudaStream_t>(stream));
}

extern "C" int km_transpose_ranges_i32(int64_t B, int64_t R, const int32_t *start, const int32_t *end,
                                       int64_t x1_size, int64_t x2_size, int32_t block_size, int32_t *start_t,
                                       int32_t *end_t, void *stream) {
    using namespace km;
    KM_REQUIRE(B >= 0 && R >= 0 && x1_size >= 0 && x2_size >= 0 && x1_size <= 0x7fffffffLL - block_size &&
                   x2_size <= 0x7fffffffLL - block_size,
               KM_ERR_INVALID_ARGUMENT, "km_transpose_ranges_i32: bad sizes");
    KM_REQUIRE(block_size >= 1, KM_ERR_INVALID_ARGUMENT, "km_transpose_ranges_i32: block_size must be >= 1");
    const int64_t C = ceil_div(x2_size, block_size);
    if (B == 0 || C == 0) return KM_OK;
    KM_REQUIRE(start_t && end_t && (R == 0 || (start && end)), KM_ERR_INVALID_ARGUMENT,
               "km_transpose_ranges_i32: null pointer");
    KM_REQUIRE(B <= 0x7fffffffLL, KM_ERR_UNSUPPORTED, "km_transpose_ranges_i32: too many batch rows");
    KM_REQUIRE(B <= KM_RANGES_MAX_ITEMS / C && (R == 0 || B <= KM_RANGES_MAX_ITEMS / R), KM_ERR_UNSUPPORTED,
               "km_transpose_ranges_i32: more than %lld (batch row, block) pairs", (long long)KM_RANGES_MAX_ITEMS);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    transpose_init_kernel<<<grid_for(B * C, 256), 256, 0, s>>>(B * C, (int)x1_size, start_t, end_t);
    if (R > 0)
        transpose_mark_kernel<<<grid_for(B * R, 256), 256, 0, s>>>(B, R, C, start, end, (int)x1_size, block_size,
                                                                   start_t, end_t);
    transpose_fix_kernel<<<(unsigned)B, 1024, 0, s>>>(C, (int)x1_size, start_t, end_t);
    KM_CHECK_LAUNCH("km_transpose_ranges_i32");
    return KM_OK;
}
