// Materialise the masked kernel matrix (dense) and its hyper-parameter gradient (dense_bwd).
//
// dense: HBM-write bound.  One CTA writes a 32-row x 512-column tile of out; threads run
// along the columns so that every row is written as one contiguous 2 KB segment of aligned 128-bit
// stores, and tiles outside the band are written as zeros by the same kernel -- no separate zero fill.
// 32 rows a tile: with 128, three kernels of 6007 x 6007 were 1.4 waves of CTAs.  (433 MB in 104 us,
// 4.2 TB/s.)  The reference stores with threadIdx.x along the ROW dimension (stride-n writes) after a
// full torch::zeros pass (native/dense/dense.cu:12-98).
//
// dense_bwd: HBM-read bound on the band part of out_grad.  A cluster of CTAs per (batch, row block) walks
// the band, lanes along the columns, rows streamed: 56 us for the 76 MB of that example's band, where one
// CTA per row block (141 CTAs) took about 200; partial sums go through the same fixed-order fp64 finish
// as the other gradient ops (native/dense_bwd/dense_bwd.cu:12-116).
#include <cooperative_groups.h>

#include <type_traits>

#include "km_common.cuh"

namespace km {

struct DenseArgs {
    Batch batch;
    int64_t m, n;
    int64_t row_strips, col_tiles;
    View<const float> x1, x2, params;
    View<const int> start, end;
    View<float> out;
};

constexpr int DENSE_TILE_COLS = 512;
constexpr int DENSE_TILE_ROWS = 32;

// VEC: columns are contiguous.  A row then starts 0 .. 3 floats past a 16-byte boundary, and its tiles
// that much earlier, so that a thread's four columns are always one aligned store.
template <int KT, bool VEC>
__global__ void __launch_bounds__(256) dense_kernel(const DenseArgs a) {
    __shared__ float x1s[DENSE_TILE_ROWS];

    int64_t item = blockIdx.x;
    const int64_t ct = item % a.col_tiles;
    item /= a.col_tiles;
    const int64_t strip = item % a.row_strips;
    const int64_t b = item / a.row_strips;
    const int64_t row0 = strip * DENSE_TILE_ROWS, r = row0 / KM_BLOCK_SIZE;

    const BatchIndex bi = decompose(a.batch, b);
    const float *x1 = batch_ptr(a.x1, bi);
    const float *x2 = batch_ptr(a.x2, bi);
    float *out = batch_ptr(a.out, bi);
    KernelFn<KT> fn;
    fn.init(batch_ptr(a.params, bi), a.params.s0);

    const int n = (int)a.n;
    const int band_lo = clamp_int(batch_ptr(a.start, bi)[r * a.start.s0], 0, n);
    const int band_hi = max(band_lo, min(batch_ptr(a.end, bi)[r * a.end.s0], n));

    const int tid = threadIdx.x;
    const int rows = (int)min((int64_t)DENSE_TILE_ROWS, a.m - row0);
    if (tid < DENSE_TILE_ROWS) x1s[tid] = tid < rows ? x1[(row0 + tid) * a.x1.s0] : 0.0f;

    const int col0 = (int)(ct * DENSE_TILE_COLS);
    const int colgroup = tid & 127;  // 128 threads cover the 512 columns of the tile
    const int rowgroup = tid >> 7;   // two row groups take alternate rows

    // the columns of a thread: four, VEC from up to three before them on
    constexpr int BEFORE = VEC ? 3 : 0, SPAN = 4 + BEFORE;
    int cols[SPAN];
    float xj[SPAN];
    bool inband[SPAN];
    bool any = false;
#pragma unroll
    for (int q = 0; q < SPAN; q++) {
        cols[q] = VEC ? col0 + colgroup * 4 + q - BEFORE : col0 + colgroup + 128 * q;
        inband[q] = cols[q] >= band_lo && cols[q] < band_hi;
        xj[q] = inband[q] ? x2[(int64_t)cols[q] * a.x2.s0] : 0.0f;
        any = any || inband[q];
    }
    __syncthreads();

    const float scale = fn.scale;
    for (int i = rowgroup; i < rows; i += 2) {
        float *orow = out + (row0 + i) * a.out.s0;
        const float xi = x1s[i];
        const auto row = [&](auto first) {
            constexpr int F = decltype(first)::value;
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (any) {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (inband[F + q]) v[q] = scale * fn.unscaled(xi - xj[F + q]);
            }
            if (VEC && cols[F] >= 0 && cols[F + 3] < n) {
                *reinterpret_cast<float4 *>(orow + cols[F]) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (cols[F + q] >= 0 && cols[F + q] < n) orow[VEC ? (int64_t)cols[F + q] : (int64_t)cols[F + q] * a.out.s1] = v[q];
            }
        };
        if constexpr (VEC) {
            switch ((uintptr_t)orow / sizeof(float) % 4) {
            case 0: row(std::integral_constant<int, 3>()); break;
            case 1: row(std::integral_constant<int, 2>()); break;
            case 2: row(std::integral_constant<int, 1>()); break;
            default: row(std::integral_constant<int, 0>()); break;
            }
        } else {
            row(std::integral_constant<int, 0>());
        }
    }
}

struct DenseBwdArgs {
    Batch batch;
    int64_t m, n;
    int64_t row_blocks;
    View<const float> x1, x2, params, out_grad;
    View<const int> start, end;
    float *partials;
};

// A cluster of BWD_CTAS CTAs shares a row block, 16 rows each; a warp takes pieces of 8 rows x 32 columns of
// them, 8 loads in flight per lane.  The CTAs' sums meet in the first one's shared memory, added in
// their order.
constexpr int BWD_CTAS = 8, BWD_ROWS = KM_BLOCK_SIZE / BWD_CTAS, BWD_PIECE = 8;

template <int KT>
__global__ void __cluster_dims__(BWD_CTAS, 1, 1) __launch_bounds__(256) dense_bwd_kernel(const DenseBwdArgs a) {
    constexpr int NS = KernelFn<KT>::NSUMS;
    __shared__ float x1s[BWD_ROWS];
    __shared__ float warp_sums[8][KM_MAX_PARAMS];
    __shared__ float cta_sums[BWD_CTAS][KM_MAX_PARAMS];  // of the cluster's first CTA

    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int part = (int)(blockIdx.x % BWD_CTAS);
    const int64_t item = blockIdx.x / BWD_CTAS + (int64_t)blockIdx.y * (gridDim.x / BWD_CTAS);
    if (item >= a.batch.count * a.row_blocks) return;  // (a whole cluster)
    cluster.barrier_arrive();
    const int64_t b = item % a.batch.count;
    const int64_t r = item / a.batch.count;
    const BatchIndex bi = decompose(a.batch, b);
    const float *x1 = batch_ptr(a.x1, bi);
    const float *x2 = batch_ptr(a.x2, bi);
    const float *og = batch_ptr(a.out_grad, bi);
    KernelFn<KT> fn;
    fn.init(batch_ptr(a.params, bi), a.params.s0);

    const int n = (int)a.n;
    const int band_lo = clamp_int(batch_ptr(a.start, bi)[r * a.start.s0], 0, n);
    const int band_hi = max(band_lo, min(batch_ptr(a.end, bi)[r * a.end.s0], n));

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t row0 = r * KM_BLOCK_SIZE + part * BWD_ROWS;
    const int rows = (int)max((int64_t)0, min((int64_t)BWD_ROWS, a.m - row0));
    if (tid < BWD_ROWS) x1s[tid] = tid < rows ? x1[(row0 + tid) * a.x1.s0] : 0.0f;
    __syncthreads();

    float sums[NS];
#pragma unroll
    for (int q = 0; q < NS; q++) sums[q] = 0.0f;

    constexpr int STRIPS = BWD_ROWS / BWD_PIECE;
    const int pieces = (band_hi - band_lo + 31) / 32 * STRIPS;
    for (int piece = warp; piece < pieces; piece += 8) {
        const int c = band_lo + piece / STRIPS * 32 + lane, i0 = piece % STRIPS * BWD_PIECE;
        if (c >= band_hi) continue;
        const float xj = x2[(int64_t)c * a.x2.s0];
        const float *ocol = og + (row0 + i0) * a.out_grad.s0 + (int64_t)c * a.out_grad.s1;
        if (i0 + BWD_PIECE <= rows) {
            float g[BWD_PIECE];
#pragma unroll
            for (int u = 0; u < BWD_PIECE; u++) g[u] = ocol[(int64_t)u * a.out_grad.s0];
#pragma unroll
            for (int u = 0; u < BWD_PIECE; u++) fn.accumulate(x1s[i0 + u] - xj, g[u], sums);
        } else {
            for (int i = i0; i < rows; i++) fn.accumulate(x1s[i] - xj, ocol[(int64_t)(i - i0) * a.out_grad.s0], sums);
        }
    }

#pragma unroll
    for (int q = 0; q < NS; q++) {
        float v = sums[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) warp_sums[warp][q] = v;
    }
    __syncthreads();
    cluster.barrier_wait();  // (the first CTA is there to be written to)
    if (tid < NS) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; w++) v += warp_sums[w][tid];
        cluster.map_shared_rank(&cta_sums[0][0], 0)[part * KM_MAX_PARAMS + tid] = v;
    }
    cluster.sync();
    if (part == 0 && tid < KM_MAX_PARAMS) {
        float v = 0.0f;
        if (tid < NS) {
#pragma unroll
            for (int w = 0; w < BWD_CTAS; w++) v += cta_sums[w][tid];
        }
        a.partials[(b * a.row_blocks + r) * KM_MAX_PARAMS + tid] = v;
    }
}

template <int KT>
static int launch_dense(const DenseArgs &a, bool vec, cudaStream_t s) {
    const int64_t items = a.batch.count * a.row_strips * a.col_tiles;
    if (items > 0x7fffffffLL) {
        set_error("km_dense_f32: too many work items (%lld)", (long long)items);
        return KM_ERR_UNSUPPORTED;
    }
    if (vec)
        dense_kernel<KT, true><<<(unsigned)items, 256, 0, s>>>(a);
    else
        dense_kernel<KT, false><<<(unsigned)items, 256, 0, s>>>(a);
    KM_CHECK_LAUNCH("km_dense_f32 launch");
    return KM_OK;
}

}  // namespace km

extern "C" int km_dense_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, const km_view *x1,
                            const km_view *x2, const km_view *params, const km_view *start, const km_view *end,
                            const km_view *out, void *stream) {
    using namespace km;
    KM_REQUIRE(valid_kernel_type(kernel_type), KM_ERR_INVALID_ARGUMENT, "km_dense_f32: unknown kernel type %d", kernel_type);
    KM_REQUIRE(batch && x1 && x2 && params && start && end && out, KM_ERR_INVALID_ARGUMENT, "km_dense_f32: null argument");
    KM_REQUIRE(m >= 0 && n >= 0 && n <= 0x7fffffffLL - 1024, KM_ERR_INVALID_ARGUMENT, "km_dense_f32: bad sizes");
    DenseArgs a;
    int rc = make_batch(batch, &a.batch);
    if (rc != KM_OK) return rc;
    if (a.batch.count == 0 || m == 0 || n == 0) return KM_OK;
    KM_REQUIRE(x1->data && x2->data && params->data && start->data && end->data && out->data,
               KM_ERR_INVALID_ARGUMENT, "km_dense_f32: null data pointer");
    a.m = m;
    a.n = n;
    a.row_strips = ceil_div(m, DENSE_TILE_ROWS);
    a.x1 = make_view<const float>(x1, a.batch);
    a.x2 = make_view<const float>(x2, a.batch);
    a.params = make_view<const float>(params, a.batch);
    a.start = make_view<const int>(start, a.batch);
    a.end = make_view<const int>(end, a.batch);
    a.out = make_view<float>(out, a.batch);
    const bool vec = a.out.s1 == 1;
    bool aligned = a.out.s0 % 4 == 0 && (uintptr_t)a.out.data % 16 == 0;
    for (int d = 0; d < a.batch.ndim; d++) aligned = aligned && a.out.bs[d] % 4 == 0;
    a.col_tiles = ceil_div(n + (vec && !aligned ? 3 : 0), DENSE_TILE_COLS);  // (rows' tiles may begin 3 columns before them)
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (kernel_type) {
    case KM_KERNEL_RBF: return launch_dense<KM_KERNEL_RBF>(a, vec, s);
    case KM_KERNEL_SPECTRAL: return launch_dense<KM_KERNEL_SPECTRAL>(a, vec, s);
    default: return launch_dense<KM_KERNEL_LOCALLY_PERIODIC>(a, vec, s);
    }
}

extern "C" int km_dense_bwd_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, const km_view *x1,
                                const km_view *x2, const km_view *params, const km_view *start,
                                const km_view *end, const km_view *out_grad, const km_view *grad, void *workspace,
                                size_t workspace_bytes, void *stream) {
    using namespace km;
    KM_REQUIRE(valid_kernel_type(kernel_type), KM_ERR_INVALID_ARGUMENT, "km_dense_bwd_f32: unknown kernel type %d", kernel_type);
    KM_REQUIRE(batch && x1 && x2 && params && start && end && out_grad && grad, KM_ERR_INVALID_ARGUMENT,
               "km_dense_bwd_f32: null argument");
    KM_REQUIRE(m >= 0 && n >= 0 && n <= 0x7fffffffLL - 1024, KM_ERR_INVALID_ARGUMENT, "km_dense_bwd_f32: bad sizes");
    DenseBwdArgs a;
    int rc = make_batch(batch, &a.batch);
    if (rc != KM_OK) return rc;
    if (a.batch.count == 0) return KM_OK;
    KM_REQUIRE(params->data && grad->data, KM_ERR_INVALID_ARGUMENT, "km_dense_bwd_f32: null data pointer");
    const size_t need = km_grad_workspace_bytes(kernel_type, batch, m);
    KM_REQUIRE(workspace_bytes >= need && (need == 0 || workspace != nullptr), KM_ERR_WORKSPACE,
               "km_dense_bwd_f32: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
    a.m = m;
    a.n = n;
    a.row_blocks = ceil_div(m, KM_BLOCK_SIZE);
    a.x1 = make_view<const float>(x1, a.batch);
    a.x2 = make_view<const float>(x2, a.batch);
    a.params = make_view<const float>(params, a.batch);
    a.out_grad = make_view<const float>(out_grad, a.batch);
    a.start = make_view<const int>(start, a.batch);
    a.end = make_view<const int>(end, a.batch);
    a.partials = static_cast<float *>(workspace);
    const View<float> g = make_view<float>(grad, a.batch);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int64_t items = a.batch.count * a.row_blocks, per_y = std::min<int64_t>(items, 0x7fffffffLL / BWD_CTAS);
    KM_REQUIRE(items <= 0x7fffffffLL, KM_ERR_UNSUPPORTED, "km_dense_bwd_f32: too many work items");
    if (items > 0) {
        KM_REQUIRE(x1->data && start->data && end->data, KM_ERR_INVALID_ARGUMENT, "km_dense_bwd_f32: null data pointer");
        const dim3 grid((unsigned)(per_y * BWD_CTAS), (unsigned)ceil_div(items, per_y));
        switch (kernel_type) {
        case KM_KERNEL_RBF: dense_bwd_kernel<KM_KERNEL_RBF><<<grid, 256, 0, s>>>(a); break;
        case KM_KERNEL_SPECTRAL: dense_bwd_kernel<KM_KERNEL_SPECTRAL><<<grid, 256, 0, s>>>(a); break;
        default: dense_bwd_kernel<KM_KERNEL_LOCALLY_PERIODIC><<<grid, 256, 0, s>>>(a); break;
        }
        KM_CHECK_LAUNCH("km_dense_bwd_f32 launch");
    }
    return launch_grad_finish(kernel_type, a.batch, a.row_blocks, a.partials, false, a.params, g, s);
}
