// Gather single kernel-matrix entries (index) and the gradient of the gather (index_bwd).
//
// A lookup reads two or more indices and, at random, its block's range and two points: what bounds
// both ops is the rate of those scattered reads (a tag each in L1, most points a sector from L2), not
// the index streams.  So a thread takes four consecutive lookups at a time, all their reads in flight; large calls
// keep the ranges in shared memory; and a forward call that a backward one will follow writes the
// distances x1[row] - x2[col] it found (4 bytes a lookup, coalesced), from which the gradient is a plain
// stream.  (2^24 lookups of 131 072 points in both directions: 308 -> 188 us.)  Out-of-band (and out-of-range) lookups give 0 and every output element is written, so no
// zero fill is needed (reference: zero fill + one 64-thread block per 64 lookups,
// native/index/index.cu:12-101).
//
// index_bwd: every thread accumulates the raw gradient sums of the lookups it visits in registers -- for
// up to IDX_BATCHES kernels side by side, else for as long as they belong to one batch --, CTAs reduce,
// and one fp64 atomic per CTA and sum lands in a [batch][4] fp64 workspace; the common finish kernel
// applies the chain rule.  The reference writes one slot per lookup and batch into a (B, P, ib, L/64, 64)
// temporary and sums it (native/index_bwd/index_bwd.cu:12-112).
#include <type_traits>

#include "km_common.cuh"

namespace km {

struct IndexArgs {
    Batch batch;
    int64_t m, n, L;
    int64_t row_blocks;
    int staged;  // ranges of all batches in shared memory
    int vec;     // index streams, distances and values may be accessed 16 bytes at a time
    View<const float> x1, x2, params;
    View<const int> start, end;
    const int32_t *bidx[KM_MAX_BATCH_DIMS];
    const int32_t *row, *col;
    const float *out_grad;
    float *out;
    float *distances;  // written by the gather (may be null), read by the gradient from distances
    double *sums;      // index_bwd: [batch.count][KM_MAX_PARAMS]
};

constexpr int IDX_UNROLL = 4;    // lookups of a thread at a time
constexpr int IDX_BATCHES = 8;   // most kernels whose parameters and sums are kept in shared memory and registers
constexpr int IDX_STAGED = 4096; // most ranges kept in shared memory (32 KB)
// "Distance" of a lookup without an entry: a NaN that no subtraction gives (those have an empty payload).
constexpr unsigned IDX_NO_ENTRY = 0x7fabcdefu;

// Four values of a stream from l on, zeros past the end.
template <typename T>
__device__ __forceinline__ void load_lookups(const T *p, int64_t l, int count, bool vec, T (&v)[IDX_UNROLL]) {
    if (vec && count == IDX_UNROLL) {
        const int4 w = *reinterpret_cast<const int4 *>(p + l);
        memcpy(v, &w, sizeof(w));
    } else {
#pragma unroll
        for (int u = 0; u < IDX_UNROLL; u++) v[u] = u < count ? p[l + u] : T(0);
    }
}
__device__ __forceinline__ void store_lookups(float *p, int64_t l, int count, bool vec, const float (&v)[IDX_UNROLL]) {
    if (vec && count == IDX_UNROLL) {
        *reinterpret_cast<float4 *>(p + l) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int u = 0; u < IDX_UNROLL; u++)
            if (u < count) p[l + u] = v[u];
    }
}

// Flat batch index of lookups l .. l + count - 1; -1: out of range.
__device__ __forceinline__ void load_batches(const IndexArgs &a, int64_t l, int count, BatchIndex (&bi)[IDX_UNROLL],
                                             int64_t (&flat)[IDX_UNROLL]) {
#pragma unroll
    for (int u = 0; u < IDX_UNROLL; u++) flat[u] = u < count ? 0 : -1;
#pragma unroll
    for (int d = 0; d < KM_MAX_BATCH_DIMS; d++) {
        if (d < a.batch.ndim) {
            int v[IDX_UNROLL];
            load_lookups(a.bidx[d], l, count, a.vec, v);
#pragma unroll
            for (int u = 0; u < IDX_UNROLL; u++) {
                const bool ok = flat[u] >= 0 && v[u] >= 0 && v[u] < a.batch.size[d];
                flat[u] = ok ? flat[u] * a.batch.size[d] + v[u] : -1;
                bi[u].i[d] = ok ? v[u] : 0;
            }
        } else {
#pragma unroll
            for (int u = 0; u < IDX_UNROLL; u++) bi[u].i[d] = 0;
        }
    }
}

// Ranges of all row blocks and batches into shared memory.
__device__ __forceinline__ void stage_ranges(const IndexArgs &a, int2 *ranges) {
    if (!a.staged) return;
    for (int i = threadIdx.x; i < (int)(a.batch.count * a.row_blocks); i += 256) {
        const BatchIndex bi = decompose(a.batch, i / a.row_blocks);
        const int64_t r = i % a.row_blocks;
        ranges[i] = make_int2(batch_ptr(a.start, bi)[r * a.start.s0], batch_ptr(a.end, bi)[r * a.end.s0]);
    }
    __syncthreads();
}

// Distances of lookups l .. l + count - 1; ok: the lookup has an entry.
__device__ __forceinline__ void resolve_lookups(const IndexArgs &a, const int2 *ranges, int64_t l, int count,
                                                BatchIndex (&bi)[IDX_UNROLL], int64_t (&flat)[IDX_UNROLL], bool (&ok)[IDX_UNROLL],
                                                float (&tau)[IDX_UNROLL]) {
    int row[IDX_UNROLL], col[IDX_UNROLL], lo[IDX_UNROLL], hi[IDX_UNROLL];
    load_batches(a, l, count, bi, flat);
    load_lookups(a.row, l, count, a.vec, row);
    load_lookups(a.col, l, count, a.vec, col);
#pragma unroll
    for (int u = 0; u < IDX_UNROLL; u++) {
        ok[u] = flat[u] >= 0 && row[u] >= 0 && row[u] < a.m && col[u] >= 0 && col[u] < a.n;
        lo[u] = hi[u] = 0;
        if (ok[u]) {
            const int64_t r = row[u] / KM_BLOCK_SIZE;
            if (a.staged) {
                const int2 range = ranges[flat[u] * a.row_blocks + r];
                lo[u] = range.x, hi[u] = range.y;
            } else {
                lo[u] = batch_ptr(a.start, bi[u])[r * a.start.s0];
                hi[u] = batch_ptr(a.end, bi[u])[r * a.end.s0];
            }
        }
    }
    float p1[IDX_UNROLL], p2[IDX_UNROLL];
#pragma unroll
    for (int u = 0; u < IDX_UNROLL; u++) {
        ok[u] = ok[u] && lo[u] <= col[u] && col[u] < hi[u];
        p1[u] = ok[u] ? batch_ptr(a.x1, bi[u])[(int64_t)row[u] * a.x1.s0] : 0.0f;
        p2[u] = ok[u] ? batch_ptr(a.x2, bi[u])[(int64_t)col[u] * a.x2.s0] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < IDX_UNROLL; u++) tau[u] = p1[u] - p2[u];
}

// The kernels of a call: one, up to IDX_BATCHES in shared memory, or (NB 0) read for every lookup.
template <int KT, int NB>
struct IndexKernels {
    static constexpr int SHARED = NB > 1 ? NB : 1;
    KernelFn<KT> one;
    KernelFn<KT> *table;
    __device__ __forceinline__ void init(const IndexArgs &a, KernelFn<KT> *shared) {
        table = shared;
        if (NB == 1) one.init(a.params.data, a.params.s0);
        if (NB > 1) {
            if (threadIdx.x < a.batch.count) shared[threadIdx.x].init(batch_ptr(a.params, decompose(a.batch, threadIdx.x)), a.params.s0);
            __syncthreads();
        }
    }
    __device__ __forceinline__ KernelFn<KT> of(const IndexArgs &a, int64_t flat, const BatchIndex &bi) const {
        if (NB == 1) return one;
        if (NB > 1) return table[flat];
        KernelFn<KT> fn;
        fn.init(batch_ptr(a.params, bi), a.params.s0);
        return fn;
    }
};

template <int KT, int NB>
__global__ void __launch_bounds__(256, 4) index_kernel(const IndexArgs a) {
    extern __shared__ __align__(16) int2 ranges[];
    __shared__ KernelFn<KT> shared_fns[IndexKernels<KT, NB>::SHARED];
    IndexKernels<KT, NB> fns;
    fns.init(a, shared_fns);
    stage_ranges(a, ranges);
    for (int64_t l = (blockIdx.x * 256LL + threadIdx.x) * IDX_UNROLL; l < a.L; l += (int64_t)gridDim.x * 256 * IDX_UNROLL) {
        const int count = (int)min((int64_t)IDX_UNROLL, a.L - l);
        BatchIndex bi[IDX_UNROLL];
        int64_t flat[IDX_UNROLL];
        bool ok[IDX_UNROLL];
        float tau[IDX_UNROLL], v[IDX_UNROLL];
        resolve_lookups(a, ranges, l, count, bi, flat, ok, tau);
#pragma unroll
        for (int u = 0; u < IDX_UNROLL; u++) {
            v[u] = 0.0f;
            if (ok[u]) {
                const KernelFn<KT> fn = fns.of(a, flat[u], bi[u]);
                v[u] = fn.scale * fn.unscaled(tau[u]);
            } else {
                tau[u] = __uint_as_float(IDX_NO_ENTRY);
            }
        }
        store_lookups(a.out, l, count, a.vec, v);
        if (a.distances != nullptr) store_lookups(a.distances, l, count, a.vec, tau);
    }
}

// NB: 1, up to IDX_BATCHES, or 0 for more.  SAVED: from the distances of the gather.
template <int KT, int NB, bool SAVED>
__global__ void __launch_bounds__(256, NB > 1 ? 2 : 4) index_bwd_kernel(const IndexArgs a) {
    constexpr int NS = KernelFn<KT>::NSUMS, SLOTS = NB > 1 ? NB : 1;
    extern __shared__ __align__(16) int2 ranges[];
    __shared__ KernelFn<KT> shared_fns[IndexKernels<KT, NB>::SHARED];
    __shared__ float warp_sums[8][SLOTS * KM_MAX_PARAMS];
    IndexKernels<KT, NB> fns;
    fns.init(a, shared_fns);
    if (!SAVED) stage_ranges(a, ranges);

    float sums[SLOTS][NS];
#pragma unroll
    for (int b = 0; b < SLOTS; b++)
#pragma unroll
        for (int q = 0; q < NS; q++) sums[b][q] = 0.0f;
    int64_t cur = -1;
    const auto flush = [&]() {
        if (cur < 0) return;
#pragma unroll
        for (int q = 0; q < NS; q++) {
            if (sums[0][q] != 0.0f) atomicAdd(a.sums + cur * KM_MAX_PARAMS + q, (double)sums[0][q]);
            sums[0][q] = 0.0f;
        }
    };

    for (int64_t l = (blockIdx.x * 256LL + threadIdx.x) * IDX_UNROLL; l < a.L; l += (int64_t)gridDim.x * 256 * IDX_UNROLL) {
        const int count = (int)min((int64_t)IDX_UNROLL, a.L - l);
        BatchIndex bi[IDX_UNROLL];
        int64_t flat[IDX_UNROLL];
        bool ok[IDX_UNROLL];
        float tau[IDX_UNROLL], g[IDX_UNROLL];
        load_lookups(a.out_grad, l, count, a.vec, g);
        if (SAVED) {
            load_lookups(const_cast<const float *>(a.distances), l, count, a.vec, tau);
            load_batches(a, l, count, bi, flat);
#pragma unroll
            for (int u = 0; u < IDX_UNROLL; u++) ok[u] = flat[u] >= 0 && __float_as_uint(tau[u]) != IDX_NO_ENTRY;
        } else {
            resolve_lookups(a, ranges, l, count, bi, flat, ok, tau);
        }
#pragma unroll
        for (int u = 0; u < IDX_UNROLL; u++) {
            if (!ok[u]) continue;
            const KernelFn<KT> fn = fns.of(a, flat[u], bi[u]);
            if (NB == 1) {
                fn.accumulate_precise(tau[u], g[u], sums[0]);
            } else if (NB > 1) {
                float term[NS];
#pragma unroll
                for (int q = 0; q < NS; q++) term[q] = 0.0f;
                fn.accumulate_precise(tau[u], g[u], term);
#pragma unroll
                for (int b = 0; b < SLOTS; b++)
#pragma unroll
                    for (int q = 0; q < NS; q++) sums[b][q] += flat[u] == b ? term[q] : 0.0f;
            } else {
                if (flat[u] != cur) flush(), cur = flat[u];
                fn.accumulate_precise(tau[u], g[u], sums[0]);
            }
        }
    }

    if (NB == 0) {  // every thread adds what it still holds
        flush();
        return;
    }
    // reduce over the CTA first, then one atomic per sum
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int b = 0; b < SLOTS; b++)
#pragma unroll
        for (int q = 0; q < NS; q++) {
            float v = sums[b][q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) warp_sums[warp][b * KM_MAX_PARAMS + q] = v;
        }
    __syncthreads();
    const int b = threadIdx.x / KM_MAX_PARAMS, q = threadIdx.x % KM_MAX_PARAMS;
    if (b < a.batch.count && b < SLOTS && q < NS) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; w++) v += warp_sums[w][threadIdx.x];
        if (v != 0.0f) atomicAdd(a.sums + threadIdx.x, (double)v);
    }
}

template <typename F>
static int index_dispatch(int kernel_type, int64_t batches, F f) {
    const auto kernels = [&](auto kt) {
        if (batches == 1) return f(kt, std::integral_constant<int, 1>());
        if (batches <= IDX_BATCHES) return f(kt, std::integral_constant<int, IDX_BATCHES>());
        return f(kt, std::integral_constant<int, 0>());
    };
    switch (kernel_type) {
    case KM_KERNEL_RBF: return kernels(std::integral_constant<int, KM_KERNEL_RBF>());
    case KM_KERNEL_SPECTRAL: return kernels(std::integral_constant<int, KM_KERNEL_SPECTRAL>());
    default: return kernels(std::integral_constant<int, KM_KERNEL_LOCALLY_PERIODIC>());
    }
}

// (a whole number of times the CTAs that fit: 2 or 4 per SM)
static unsigned index_grid(int64_t L) { return (unsigned)std::min<int64_t>(ceil_div(L, 256 * IDX_UNROLL), 148 * 8); }

// Vector accesses and staged ranges, once the streams are known.  Ranges are staged where that is little
// against the scattered reads it saves: every CTA reads all of them, 32 at a time.
static size_t index_plan(IndexArgs &a, bool uses_ranges) {
    const auto aligned = [](const void *p) { return (uintptr_t)p % 16 == 0; };
    a.vec = aligned(a.row) && aligned(a.col) && aligned(a.out) && aligned(a.out_grad) && aligned(a.distances);
    for (int d = 0; d < a.batch.ndim; d++) a.vec = a.vec && aligned(a.bidx[d]);
    const int64_t ranges = a.batch.count * a.row_blocks;
    a.staged = uses_ranges && ranges <= IDX_STAGED && a.L >= 64 * ranges;
    return a.staged ? (size_t)ranges * sizeof(int2) : 0;
}

static int fill_index_args(const char *name, IndexArgs &a, int kernel_type, const km_batch *batch, int64_t m,
                           int64_t n, int64_t L, const km_view *x1, const km_view *x2, const km_view *params,
                           const km_view *start, const km_view *end, const int32_t *const *batch_indices,
                           const int32_t *row, const int32_t *col) {
    KM_REQUIRE(valid_kernel_type(kernel_type), KM_ERR_INVALID_ARGUMENT, "%s: unknown kernel type %d", name, kernel_type);
    KM_REQUIRE(batch && x1 && x2 && params && start && end, KM_ERR_INVALID_ARGUMENT, "%s: null argument", name);
    KM_REQUIRE(m >= 0 && n >= 0 && L >= 0 && n <= 0x7fffffffLL && m <= 0x7fffffffLL, KM_ERR_INVALID_ARGUMENT,
               "%s: bad sizes", name);
    int rc = make_batch(batch, &a.batch);
    if (rc != KM_OK) return rc;
    a.m = m;
    a.n = n;
    a.L = L;
    a.x1 = make_view<const float>(x1, a.batch);
    a.x2 = make_view<const float>(x2, a.batch);
    a.params = make_view<const float>(params, a.batch);
    a.start = make_view<const int>(start, a.batch);
    a.end = make_view<const int>(end, a.batch);
    for (int d = 0; d < KM_MAX_BATCH_DIMS; d++) a.bidx[d] = nullptr;
    if (L > 0) {
        KM_REQUIRE(row && col, KM_ERR_INVALID_ARGUMENT, "%s: null index pointer", name);
        KM_REQUIRE(a.batch.ndim == 0 || batch_indices != nullptr, KM_ERR_INVALID_ARGUMENT, "%s: null batch_indices", name);
        for (int d = 0; d < a.batch.ndim; d++) {
            KM_REQUIRE(batch_indices[d] != nullptr, KM_ERR_INVALID_ARGUMENT, "%s: null batch index array %d", name, d);
            a.bidx[d] = batch_indices[d];
        }
    }
    a.row = row;
    a.col = col;
    a.row_blocks = ceil_div(m, KM_BLOCK_SIZE);
    a.out_grad = nullptr;
    a.out = nullptr;
    a.distances = nullptr;
    a.sums = nullptr;
    return KM_OK;
}

static int index_forward(const char *name, IndexArgs &a, int kernel_type, float *out, float *distances, cudaStream_t s) {
    if (a.L == 0) return KM_OK;
    KM_REQUIRE(out != nullptr, KM_ERR_INVALID_ARGUMENT, "%s: null output", name);
    a.out = out, a.distances = distances;
    const size_t smem = index_plan(a, true);
    return index_dispatch(kernel_type, a.batch.count, [&](auto kt, auto nb) {
        index_kernel<decltype(kt)::value, decltype(nb)::value><<<index_grid(a.L), 256, smem, s>>>(a);
        KM_CHECK_LAUNCH("gather launch");
        return (int)KM_OK;
    });
}

template <bool SAVED>
static int index_backward(const char *name, IndexArgs &a, int kernel_type, const km_batch *batch, const float *out_grad,
                          const km_view *grad, void *workspace, size_t workspace_bytes, cudaStream_t s) {
    KM_REQUIRE(grad != nullptr, KM_ERR_INVALID_ARGUMENT, "%s: null argument", name);
    if (a.batch.count == 0) return KM_OK;
    const size_t need = km_index_bwd_workspace_bytes(kernel_type, batch);
    KM_REQUIRE(workspace_bytes >= need && workspace != nullptr, KM_ERR_WORKSPACE, "%s: workspace of %zu bytes needed, %zu given", name,
               need, workspace_bytes);
    KM_REQUIRE(a.L == 0 || out_grad != nullptr, KM_ERR_INVALID_ARGUMENT, "%s: null out_grad", name);
    a.out_grad = out_grad;
    a.sums = static_cast<double *>(workspace);
    const cudaError_t err = cudaMemsetAsync(workspace, 0, need, s);
    if (err != cudaSuccess) return cuda_fail(err, "gather gradient memset");
    if (a.L > 0) {
        const size_t smem = index_plan(a, !SAVED);
        const int rc = index_dispatch(kernel_type, a.batch.count, [&](auto kt, auto nb) {
            index_bwd_kernel<decltype(kt)::value, decltype(nb)::value, SAVED><<<index_grid(a.L), 256, smem, s>>>(a);
            KM_CHECK_LAUNCH("gather gradient launch");
            return (int)KM_OK;
        });
        if (rc != KM_OK) return rc;
    }
    return launch_grad_finish(kernel_type, a.batch, 1, a.sums, true, a.params, make_view<float>(grad, a.batch), s);
}

}  // namespace km

extern "C" int km_index_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t L,
                            const km_view *x1, const km_view *x2, const km_view *params, const km_view *start,
                            const km_view *end, const int32_t *const *batch_indices, const int32_t *row,
                            const int32_t *col, float *out, void *stream) {
    using namespace km;
    IndexArgs a;
    const int rc = fill_index_args("km_index_f32", a, kernel_type, batch, m, n, L, x1, x2, params, start, end,
                                   batch_indices, row, col);
    if (rc != KM_OK) return rc;
    return index_forward("km_index_f32", a, kernel_type, out, nullptr, static_cast<cudaStream_t>(stream));
}

extern "C" int km_index_distances_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t L,
                                      const km_view *x1, const km_view *x2, const km_view *params, const km_view *start,
                                      const km_view *end, const int32_t *const *batch_indices, const int32_t *row,
                                      const int32_t *col, float *out, float *distances, void *stream) {
    using namespace km;
    IndexArgs a;
    const int rc = fill_index_args("km_index_distances_f32", a, kernel_type, batch, m, n, L, x1, x2, params, start, end,
                                   batch_indices, row, col);
    if (rc != KM_OK) return rc;
    KM_REQUIRE(L == 0 || distances != nullptr, KM_ERR_INVALID_ARGUMENT, "km_index_distances_f32: null distances");
    return index_forward("km_index_distances_f32", a, kernel_type, out, distances, static_cast<cudaStream_t>(stream));
}

extern "C" size_t km_index_bwd_workspace_bytes(int kernel_type, const km_batch *batch) {
    (void)kernel_type;
    km::Batch b;
    if (batch == nullptr || km::make_batch(batch, &b) != KM_OK) return 0;
    return (size_t)b.count * KM_MAX_PARAMS * sizeof(double);
}

extern "C" int km_index_bwd_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t L,
                                const km_view *x1, const km_view *x2, const km_view *params,
                                const km_view *start, const km_view *end, const int32_t *const *batch_indices,
                                const int32_t *row, const int32_t *col, const float *out_grad,
                                const km_view *grad, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace km;
    IndexArgs a;
    const int rc = fill_index_args("km_index_bwd_f32", a, kernel_type, batch, m, n, L, x1, x2, params, start, end,
                                   batch_indices, row, col);
    if (rc != KM_OK) return rc;
    return index_backward<false>("km_index_bwd_f32", a, kernel_type, batch, out_grad, grad, workspace, workspace_bytes,
                                 static_cast<cudaStream_t>(stream));
}

extern "C" int km_index_bwd_distances_f32(int kernel_type, const km_batch *batch, int64_t L, const km_view *params,
                                          const int32_t *const *batch_indices, const float *distances, const float *out_grad,
                                          const km_view *grad, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace km;
    KM_REQUIRE(valid_kernel_type(kernel_type) && batch && params && L >= 0, KM_ERR_INVALID_ARGUMENT,
               "km_index_bwd_distances_f32: bad arguments");
    IndexArgs a = {};
    const int rc = make_batch(batch, &a.batch);
    if (rc != KM_OK) return rc;
    KM_REQUIRE(L == 0 || distances, KM_ERR_INVALID_ARGUMENT, "km_index_bwd_distances_f32: null distances");
    KM_REQUIRE(L == 0 || a.batch.ndim == 0 || batch_indices, KM_ERR_INVALID_ARGUMENT, "km_index_bwd_distances_f32: null batch_indices");
    a.L = L;
    a.params = make_view<const float>(params, a.batch);
    for (int d = 0; L > 0 && d < a.batch.ndim; d++) {
        KM_REQUIRE(batch_indices[d] != nullptr, KM_ERR_INVALID_ARGUMENT, "km_index_bwd_distances_f32: null batch index array %d", d);
        a.bidx[d] = batch_indices[d];
    }
    a.distances = const_cast<float *>(distances);  // (only read)
    return index_backward<true>("km_index_bwd_distances_f32", a, kernel_type, batch, out_grad, grad, workspace, workspace_bytes,
                                static_cast<cudaStream_t>(stream));
}
