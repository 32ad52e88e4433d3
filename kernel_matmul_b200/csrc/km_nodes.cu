// Products and gradients by blockwise interpolation (km_nodes.cuh has the method and its error bound).
//
// The kernels of a call are chained by programmatic dependent launches, each waiting for its predecessor before
// anything but operands is read; those behind the gate wait in Gate::closed.
//
// A call is: extents of the blocks and choice of P (nodes_plan_kernel), Lagrange matrices
// (nodes_lambda_kernel), rhs / left / right at the nodes (nodes_compress_kernel), then the product
// (nodes_product_kernel, which also takes its result back to the 128 rows) or the gradient
// (nodes_grad_kernel).  Whether the call may be done this way is decided on the device: bands aligned
// to blocks and P within bounds.  The kernels of the direct evaluation are launched behind it and
// return at once if it was; the interpolation kernels return at once if not.  So no call waits for
// the host, and inputs without short intervals (unsorted points without a cutoff, frequencies of many
// periods per block) are computed as they always were.
#include <cstddef>
#include <type_traits>

#include "km_nodes.cuh"

namespace km {

constexpr int NODES_CLASSES_PER_LEVEL = 8;
constexpr int NODES_CLASSES = NODES_LEVELS * NODES_CLASSES_PER_LEVEL;

// A class is a number of nodes at one of the half-lengths.  First bytes of the workspace; the first
// three words are zero on entry to the plan kernel.
struct NodesHeader {
    int max_h_bits;  // largest half-length of any block (bits of a non-negative float)
    int bad;         // some band is not aligned to blocks, or an input is not finite
    int done;        // CTAs of the plan kernel that have finished
    int use;         // 1: interpolate, 0: evaluate directly
    float h[NODES_LEVELS];
    int first[NODES_LEVELS + 1];  // classes of level l: first[l] .. first[l + 1] - 1
    int P[NODES_CLASSES];
    int off[NODES_CLASSES];       // nodes of smaller classes of the level: place in the arrays shared by all batches
    float delta[NODES_CLASSES][NODES_MAX];   // node offsets from a block's centre
    float weight[NODES_CLASSES][NODES_MAX];  // barycentric weights
};
constexpr size_t NODES_ZEROED = offsetof(NodesHeader, use);

struct NodesArgs {
    Batch batch;
    int64_t m, n, k;
    int64_t R, C;       // row and column blocks
    int64_t slots1, slots2;  // distinct x1 / x2 rows: batch.count, or 1 if all batches share one
    int same;           // x1 and x2 are the same points
    int block;          // points per block: KM_BLOCK_SIZE, or more where all rows see all columns
    const int *order1, *order2;  // the points in order (not null where block > KM_BLOCK_SIZE)
    int max_p;          // most nodes of a block
    int cap;            // most nodes of a block over all classes of its level, where batches share x
    View<const float> x1, x2, params;
    View<const int> start, end;
    NodesHeader *hdr;
    int *classes;              // [batch][level]
    float *centre1, *centre2;  // [slot][block]
    float *half1, *half2;      // [slot][block] half-lengths
    float *lambda1, *lambda2;  // [slot][block][cap or max_p][points per block]
};

// Row of the caller's arrays that holds point i of the blocks.
__device__ __forceinline__ int64_t point_row(const int *order, int64_t i) { return order == nullptr ? i : (int64_t)order[i]; }

__device__ __forceinline__ int level_of(const NodesHeader *hdr, float half) {
    int l = 0;
#pragma unroll
    for (int i = 1; i < NODES_LEVELS; i++) l += half <= hdr->h[i];
    return l;
}

// Rows (of 128 or kq floats) between blocks, and first row of a class within its block, of an array
// with one copy for all batches (classes side by side) or one per batch.
__device__ __forceinline__ int64_t node_rows(const NodesArgs &a, int64_t slots) { return slots == 1 && a.batch.count > 1 ? a.cap : a.max_p; }
__device__ __forceinline__ int node_first(const NodesArgs &a, int64_t slots, int cls) { return slots == 1 && a.batch.count > 1 ? a.hdr->off[cls] : 0; }

template <int V>
using Int = std::integral_constant<int, V>;

__device__ __forceinline__ int nodes_needed_for(int kt, const float *theta, int64_t stride, float h, int lane) {
    if (kt == KM_KERNEL_RBF) return nodes_needed<KM_KERNEL_RBF>(theta, stride, h, lane);
    if (kt == KM_KERNEL_SPECTRAL) return nodes_needed<KM_KERNEL_SPECTRAL>(theta, stride, h, lane);
    return nodes_needed<KM_KERNEL_LOCALLY_PERIODIC>(theta, stride, h, lane);
}

// Extents of every block (a warp each), alignment of every band, and -- the CTA that finishes last --
// the number of nodes of every kernel of the batch at every half-length.
// (Time is latency, most of it the last CTA's: 16 kernels on 512 blocks took 21 us with 256 threads and the
// classes listed in shared memory.)
constexpr int PLAN_THREADS = 512, PLAN_WARPS = PLAN_THREADS / 32;
__global__ void __launch_bounds__(PLAN_THREADS) nodes_plan_kernel(const NodesArgs a, int kernel_type) {
    grid_release();
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * PLAN_WARPS, first = blockIdx.x * (int64_t)PLAN_WARPS + (threadIdx.x >> 5);
    const int64_t boxes1 = a.slots1 * a.R, boxes = boxes1 + (a.same ? 0 : a.slots2 * a.C);
    float longest = 0.0f;
    int bad = 0;
    for (int64_t w = first; w < boxes; w += warps) {
        const bool one = w < boxes1;
        const int64_t v = one ? w : w - boxes1, blocks = one ? a.R : a.C, rows = one ? a.m : a.n;
        const int64_t slot = v / blocks, block = v % blocks;
        const View<const float> &x = one ? a.x1 : a.x2;
        const float *base = batch_ptr(x, decompose(a.batch, slot));
        float lo = INFINITY, hi = -INFINITY;
        bool nan = false;
        const int *order = one ? a.order1 : a.order2;
        const auto see = [&](int i) {
            const int64_t row = block * a.block + i;
            if (row < rows) {
                const float e = base[point_row(order, row) * x.s0];
                lo = fminf(lo, e);
                hi = fmaxf(hi, e);
                nan = nan || !(fabsf(e) < INFINITY);
            }
        };
        if (order != nullptr) {  // in order: the first and the last point (all are finite, or `bad` is set)
            if (lane < 2) see(lane == 0 ? 0 : (int)min((int64_t)a.block, rows - block * a.block) - 1);
        } else {
#pragma unroll
            for (int i = 0; i < KM_BLOCK_SIZE; i += 32) see(i + lane);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        const float c = 0.5f * lo + 0.5f * hi, h = fmaxf(fmaxf(hi - c, c - lo), NODES_MIN_H);
        bad |= nan || !(h < INFINITY);
        longest = fmaxf(longest, h);
        if (lane == 0) (one ? a.centre1 : a.centre2)[v] = c, (one ? a.half1 : a.half2)[v] = h;
    }
    const int64_t threads = (int64_t)gridDim.x * blockDim.x;
    const int64_t bands = (a.m + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE;  // row blocks of the band
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < a.batch.count * bands; w += threads) {
        const BatchIndex bi = decompose(a.batch, w / bands);
        const int64_t r = w % bands;
        const int s = batch_ptr(a.start, bi)[r * a.start.s0], e = batch_ptr(a.end, bi)[r * a.end.s0];
        if (a.order1 != nullptr) {  // all rows must see all columns
            bad |= s > 0 || e < a.n;
            continue;
        }
        if (s >= e) continue;  // an empty band
        bad |= s < 0 || s % KM_BLOCK_SIZE != 0 || (e < a.n && e % KM_BLOCK_SIZE != 0);
    }
    __shared__ int s_last, s_fits;
    __shared__ int s_class[NODES_LEVELS][NODES_MAX / 2 + 1];  // by P / 2: needed, then its class
    __shared__ int s_nodes, s_P[NODES_CLASSES], s_node_first[NODES_CLASSES];
    __shared__ float s_h[NODES_CLASSES], s_delta[NODES_CLASSES * NODES_MAX];
    __shared__ unsigned char s_node_class[NODES_CLASSES * NODES_MAX];
    if (lane == 0) atomicMax(&a.hdr->max_h_bits, __float_as_int(longest));
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        if (bad) a.hdr->bad = 1;
        __threadfence();
        s_last = atomicAdd(&a.hdr->done, 1) == (int)gridDim.x - 1;
        s_fits = 1;
    }
    for (int i = threadIdx.x; i < NODES_LEVELS * (NODES_MAX / 2 + 1); i += PLAN_THREADS) (&s_class[0][0])[i] = 0;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    float h[NODES_LEVELS];
    h[0] = __int_as_float(*reinterpret_cast<volatile int *>(&a.hdr->max_h_bits));
#pragma unroll
    for (int l = 1; l < NODES_LEVELS; l++) h[l] = h[l - 1] * (1.0f / NODES_RATIO);
    const bool any_bad = *reinterpret_cast<volatile int *>(&a.hdr->bad) != 0;
    for (int64_t w = threadIdx.x >> 5; w < a.batch.count * NODES_LEVELS; w += PLAN_WARPS) {
        const int l = (int)(w % NODES_LEVELS);
        const float *theta = batch_ptr(a.params, decompose(a.batch, w / NODES_LEVELS));
        // (fewer classes where batches share the points: every class has its own Lagrange matrices)
        const int unit = a.batch.count > 1 && (a.slots1 == 1 || a.slots2 == 1) ? 4 : 2;
        const int p = max(4, (min(nodes_needed_for(kernel_type, theta, a.params.s0, h[l], lane), 4096) + unit - 1) & -unit);
        if (lane == 0) {
            if (p > a.max_p) {
                s_fits = 0;
            } else {
                a.classes[w] = p;
                s_class[l][p / 2] = 1;
            }
        }
    }
    __syncthreads();
    const bool use = !any_bad && s_fits;
    // warp l lists the classes of level l: counted from the largest node count down while they fit; smaller
    // ones are served by the smallest that does (the largest always fits)
    static_assert(NODES_LEVELS <= PLAN_WARPS && NODES_MAX / 2 < 64, "a warp per level, a bit per node count");
    __shared__ int s_count[NODES_LEVELS];
    const int l = threadIdx.x >> 5;
    unsigned long long needed = 0, kept = 0;  // bits: P / 2
    if (l < NODES_LEVELS && use) {
        needed = __ballot_sync(0xffffffffu, s_class[l][lane] != 0);
        needed |= (unsigned long long)__ballot_sync(0xffffffffu, lane + 32 <= NODES_MAX / 2 && s_class[l][min(lane + 32, NODES_MAX / 2)] != 0) << 32;
        int total = 0;
        for (unsigned long long left = needed; left != 0;) {
            const int i = 63 - __clzll((long long)left);
            if (__popcll(kept) == NODES_CLASSES_PER_LEVEL || total + 2 * i > a.cap) break;
            kept |= 1ull << i, left &= ~(1ull << i), total += 2 * i;
        }
        if (lane == 0) s_count[l] = __popcll(kept);
    }
    __syncthreads();
    if (l < NODES_LEVELS && lane == 0 && use) {
        int at = 0, off = 0;
        for (int i = 0; i < l; i++) at += s_count[i];
        a.hdr->h[l] = h[l];
        a.hdr->first[l] = at;
        if (l == NODES_LEVELS - 1) a.hdr->first[NODES_LEVELS] = at + s_count[l];
        for (unsigned long long left = needed; left != 0; left &= left - 1) {
            const int i = __ffsll((long long)left) - 1;
            s_class[l][i] = at;
            if (!((kept >> i) & 1)) continue;
            a.hdr->P[at] = s_P[at] = 2 * i;
            a.hdr->off[at] = off;
            s_h[at++] = h[l];
            off += 2 * i;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a.hdr->use = use;
        int at = 0;
        if (use)
            for (int c = 0; c < s_count[0] + s_count[1] + s_count[2] + s_count[3]; c++) s_node_first[c] = at, at += s_P[c];
        s_nodes = at;
    }
    __syncthreads();
    if (!use) return;
    for (int c = threadIdx.x >> 5; c < s_count[0] + s_count[1] + s_count[2] + s_count[3]; c += PLAN_WARPS)
        for (int q = lane; q < s_P[c]; q += 32) s_node_class[s_node_first[c] + q] = (unsigned char)c;
    __syncthreads();
    for (int64_t w = threadIdx.x; w < a.batch.count * NODES_LEVELS; w += PLAN_THREADS) a.classes[w] = s_class[w % NODES_LEVELS][a.classes[w] / 2];
    // offsets, then weights, of all classes: one node per thread and round
    for (int i = threadIdx.x; i < s_nodes; i += PLAN_THREADS) {
        const int c = s_node_class[i], q = i - s_node_first[c];
        s_delta[i] = a.hdr->delta[c][q] = node_offset(s_h[c], q, s_P[c]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < s_nodes; i += PLAN_THREADS) {
        const int c = s_node_class[i], q = i - s_node_first[c];
        a.hdr->weight[c][q] = node_weight(s_delta + s_node_first[c], s_h[c], q, s_P[c]);
    }
}

// Lagrange matrices of 128 rows of one block, one per class in use for it: thread = row,
// lambda[q][row] = (w_q / (x - xi_q)) / sum of the same.
__global__ void __launch_bounds__(128) nodes_lambda_kernel(const NodesArgs a) {
    const NodesHeader *hdr = a.hdr;
    grid_wait();
    if (!hdr->use) return;
    __shared__ float delta[NODES_MAX], weight[NODES_MAX];
    const int64_t boxes1 = a.slots1 * a.R;
    const int parts = a.block / 128, part = blockIdx.x % parts;
    const bool one = blockIdx.x / parts < boxes1;
    const int64_t v = blockIdx.x / parts - (one ? 0 : boxes1), blocks = one ? a.R : a.C, rows = one ? a.m : a.n;
    const int64_t slots = one ? a.slots1 : a.slots2;
    const View<const float> &x = one ? a.x1 : a.x2;
    const int t = threadIdx.x;
    const int level = level_of(hdr, (one ? a.half1 : a.half2)[v]);
    // (differences in units of h: an interval may be as short as NODES_MIN_H)
    const float inv_h = 1.0f / hdr->h[level];
    const int64_t row = (v % blocks) * a.block + part * 128 + t;
    const float d = row < rows ? batch_ptr(x, decompose(a.batch, v / blocks))[point_row(one ? a.order1 : a.order2, row) * x.s0] - (one ? a.centre1 : a.centre2)[v] : 0.0f;
    const bool shared = slots == 1;
    const int c0 = shared ? hdr->first[level] : a.classes[v / blocks * NODES_LEVELS + level], c1 = shared ? hdr->first[level + 1] : c0 + 1;
    for (int cls = c0; cls < c1; cls++) {
        const int P = hdr->P[cls];
        __syncthreads();
        if (t < P) delta[t] = hdr->delta[cls][t], weight[t] = hdr->weight[cls][t];
        __syncthreads();
        float *out = (one ? a.lambda1 : a.lambda2) + (v * node_rows(a, slots) + node_first(a, slots, cls)) * a.block + part * 128 + t;
        if (row >= rows) {
            for (int q = 0; q < P; q++) out[q * a.block] = 0.0f;
            continue;
        }
        float sum = 0.0f;
        int hit = -1;
#pragma unroll 4
        for (int q = 0; q < P; q++) {
            const float e = (d - delta[q]) * inv_h;
            if (e == 0.0f) hit = q;
            sum += __fdividef(weight[q], e);
        }
        const float inv = 1.0f / sum;
#pragma unroll 4
        for (int q = 0; q < P; q++) {
            const float e = (d - delta[q]) * inv_h;
            out[q * a.block] = hit >= 0 ? (q == hit ? 1.0f : 0.0f) : __fdividef(weight[q], e) * inv;
        }
    }
}

// Order of points that no band orders: a counting sort into equal intervals between the smallest and the
// largest point, then every interval (16 points on average) sorted by (value, index) by a warp, so that
// the order, and with it every sum, is the same on every run.  Inputs that fill an interval with more
// than SORT_MOST points are evaluated directly.
constexpr int SORT_BUCKETS = 8192;
constexpr int SORT_MOST = 1024;
struct SortTables {
    unsigned lo, hi;             // smallest and largest point as ordered integers (zero on entry: of ~lo, hi)
    int counts[SORT_BUCKETS];    // zero on entry; later the points placed so far
    int first[SORT_BUCKETS + 1];
};

__device__ __forceinline__ unsigned ordered_bits(float v) {
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float ordered_value(unsigned b) { return __uint_as_float((b & 0x80000000u) ? b & 0x7fffffffu : ~b); }
__device__ __forceinline__ int sort_bucket(float v, float lo, float scale) { return min(max((int)((v - lo) * scale), 0), SORT_BUCKETS - 1); }
__device__ __forceinline__ float sort_scale(float lo, float hi) { return hi > lo ? (float)SORT_BUCKETS / (hi - lo) : 0.0f; }

__global__ void __launch_bounds__(256) sort_bounds_kernel(View<const float> x, int64_t n, SortTables *t) {
    unsigned lo = 0u, hi = 0u;  // of the complement, so that zero is neutral for both
    for (int64_t i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) {
        const unsigned b = ordered_bits(x.data[i * x.s0]);
        lo = max(lo, ~b);
        hi = max(hi, b);
    }
    lo = __reduce_max_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) atomicMax(&t->lo, lo), atomicMax(&t->hi, hi);
}

__global__ void __launch_bounds__(256) sort_count_kernel(View<const float> x, int64_t n, SortTables *t) {
    const float lo = ordered_value(~t->lo), scale = sort_scale(lo, ordered_value(t->hi));
    for (int64_t i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL)
        atomicAdd(&t->counts[sort_bucket(x.data[i * x.s0], lo, scale)], 1);
}

__global__ void __launch_bounds__(1024) sort_scan_kernel(SortTables *t, int *bad) {
    constexpr int PER = SORT_BUCKETS / 1024;
    __shared__ int warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int c[PER], sum = 0;
    bool over = false;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        c[i] = t->counts[threadIdx.x * PER + i];
        over = over || c[i] > SORT_MOST;
        sum += c[i];
    }
    int run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += y;
    }
    if (lane == 31) warp_sum[warp] = run;
    __syncthreads();
    int before = run - sum;
    for (int w = 0; w < warp; w++) before += warp_sum[w];
#pragma unroll
    for (int i = 0; i < PER; i++) {
        t->first[threadIdx.x * PER + i] = before;
        t->counts[threadIdx.x * PER + i] = 0;
        before += c[i];
    }
    if (threadIdx.x == 1023) t->first[SORT_BUCKETS] = before;
    // (the bits of NaNs lie beyond those of the infinities)
    const bool finite = ordered_value(~t->lo) > -INFINITY && ordered_value(t->hi) < INFINITY;
    if (over || !finite) *bad = 1;
}

__global__ void __launch_bounds__(256) sort_place_kernel(View<const float> x, int64_t n, SortTables *t, int *order) {
    const float lo = ordered_value(~t->lo), scale = sort_scale(lo, ordered_value(t->hi));
    for (int64_t i = blockIdx.x * 256LL + threadIdx.x; i < n; i += gridDim.x * 256LL) {
        const int b = sort_bucket(x.data[i * x.s0], lo, scale);
        order[t->first[b] + atomicAdd(&t->counts[b], 1)] = (int)i;
    }
}

// Bitonic sort of each interval's (value, index) pairs in shared memory, a warp per interval.
__global__ void __launch_bounds__(128) sort_intervals_kernel(View<const float> x, const SortTables *t, int *order, const int *bad) {
    if (*bad) return;
    __shared__ unsigned long long keys[4][SORT_MOST];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int b = blockIdx.x * 4 + warp; b < SORT_BUCKETS; b += gridDim.x * 4) {
        const int first = t->first[b], count = t->first[b + 1] - first;
        if (count < 2) continue;
        int size = 2;
        while (size < count) size *= 2;
        for (int i = lane; i < size; i += 32) {
            unsigned long long key = ~0ull;
            if (i < count) {
                const int p = order[first + i];
                key = ((unsigned long long)ordered_bits(x.data[p * x.s0]) << 32) | (unsigned)p;
            }
            keys[warp][i] = key;
        }
        __syncwarp();
        for (int span = 2; span <= size; span *= 2)
            for (int d = span / 2; d > 0; d /= 2) {
                for (int i = lane; i < size / 2; i += 32) {
                    const int u = 2 * d * (i / d) + i % d, v = u + d;
                    const unsigned long long p = keys[warp][u], q = keys[warp][v];
                    if ((p > q) == ((u & span) == 0)) keys[warp][u] = q, keys[warp][v] = p;
                }
                __syncwarp();
            }
        for (int i = lane; i < count; i += 32) order[first + i] = (int)(unsigned)keys[warp][i];
        __syncwarp();
    }
}

static int sort_points(const View<const float> &x, int64_t n, SortTables *t, int *order, int *bad, cudaStream_t s) {
    const cudaError_t err = cudaMemsetAsync(t, 0, offsetof(SortTables, first), s);
    if (err != cudaSuccess) return cuda_fail(err, "interpolation: cudaMemsetAsync");
    const unsigned ctas = (unsigned)std::min<int64_t>((n + 255) / 256, 148 * 4);
    sort_bounds_kernel<<<ctas, 256, 0, s>>>(x, n, t);
    sort_count_kernel<<<ctas, 256, 0, s>>>(x, n, t);
    sort_scan_kernel<<<1, 1024, 0, s>>>(t, bad);
    sort_place_kernel<<<ctas, 256, 0, s>>>(x, n, t, order);
    sort_intervals_kernel<<<148 * 4, 128, 0, s>>>(x, t, order, bad);
    KM_CHECK_LAUNCH("interpolation: sort launch");
    return KM_OK;
}

// Lambda^T of one operand: out[slot][block][q][c] = sum_row lambda[q][row] * v[row][c], columns padded
// to kq = a multiple of 4 with zeros; an operand that all batches share is taken to the nodes of every
// class in use for its block.
struct CompressArgs {
    NodesArgs a;
    int64_t rows, kq, blocks;
    int64_t slots;     // distinct (operand, points) rows
    int64_t x_slots;   // distinct points: one Lagrange matrix per block for all batches if 1
    int vec;           // rows may be read 16 bytes at a time
    View<const float> v;
    const int *order;
    const float *half, *lambda;
    float *out;
};

constexpr int CP_ROWS = 128;             // rows at a time
constexpr int CP_NODES = 40;             // nodes at a time
constexpr int CP_LS = CP_ROWS + 4;       // (lanes of neighbouring nodes read neighbouring 16 bytes)
template <int COLS>
struct CompressShape {
    static constexpr int LAMBDA = CP_ROWS * COLS, PARTS = LAMBDA + CP_NODES * CP_LS;  // floats before them
    static constexpr size_t SMEM = (PARTS + 4 * 32 * 16) * sizeof(float);
};

// A CTA per (slot, block, COLS columns), and per class where an operand is shared by all batches.  What it
// needs of 128 rows -- operand and Lagrange matrix -- is fetched at once; a warp takes 32 of the rows, a
// lane 4 nodes (a quarter of them apart) x 4 columns of them, four rows at a time: 8 shared-memory reads of 16 bytes for
// 32 packed FMAs.  The warps' sums are added in order.  More than 40 nodes, or more units than lanes, go over
// the rows again, which for blocks of 128 are still there.
// (One warp per block and 32 columns, through stages of 32 rows, had 512 - 2000 warps on the GPU and waited: 42 us instead of
// 22 for 65 536 shared rows x 16 columns, 125 instead of 54 for 131 072 x 128 in blocks of 1024, 145 instead of
// 112 for 4 x 262 144 x 32.)
template <int COLS>
__global__ void __launch_bounds__(128) nodes_compress_kernel(const CompressArgs p) {
    const NodesArgs &a = p.a;
    using Shape = CompressShape<COLS>;
    extern __shared__ __align__(16) float smem[];
    float *vs = smem, *ls = smem + Shape::LAMBDA, *parts = smem + Shape::PARTS;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    __shared__ int s_use;
    const int64_t chunks = (p.kq + COLS - 1) / COLS;
    const int64_t chunk = blockIdx.x % chunks, box = blockIdx.x / chunks, slot = box / p.blocks, block = box % p.blocks;
    const int64_t x_slot = p.x_slots == 1 ? 0 : slot;
    const int k0 = (int)chunk * COLS, kc = (int)min((int64_t)COLS, p.kq - k0);  // a multiple of 4
    const float *v = batch_ptr(p.v, decompose(a.batch, slot));
    const int64_t row0 = block * a.block;
    const int groups = kc / 4;
    const int row_count = (int)min((int64_t)a.block, p.rows - row0), steps = (row_count + CP_ROWS - 1) / CP_ROWS;
    const auto fetch_rows = [&](int r) {
        const int count = min(CP_ROWS, row_count - r);
        if (p.vec) {
            for (int e = t; e < CP_ROWS * groups; e += 128) {
                const int i = e / groups, ce = (e - i * groups) * 4;
                if (i < count)
                    cp_async16(vs + i * COLS + ce, v + point_row(p.order, row0 + r + i) * p.v.s0 + k0 + ce);
                else
                    *reinterpret_cast<float4 *>(vs + i * COLS + ce) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        } else {
            for (int e = t; e < CP_ROWS * kc; e += 128) {
                const int i = e / kc, ce = e - i * kc;
                if (i < count && k0 + ce < a.k)
                    cp_async4(vs + i * COLS + ce, v + point_row(p.order, row0 + r + i) * p.v.s0 + (k0 + ce) * p.v.s1);
                else
                    vs[i * COLS + ce] = 0.0f;
            }
        }
    };
    // the operand was there before the plan, whose results come through a chain of loads: it is on the way
    // meanwhile (but not where there is a CTA per class, most of which have nothing to do)
    const bool early = gridDim.y == 1;
    if (early) fetch_rows(0);
    grid_wait();
    if (t == 0) s_use = a.hdr->use;  // (once: another CTA may clear it meanwhile)
    __syncthreads();
    const int level = level_of(a.hdr, p.half[x_slot * p.blocks + block]);
    const int cls = p.slots == 1 ? a.hdr->first[level] + (int)blockIdx.y : a.classes[slot * NODES_LEVELS + level];
    if (!s_use || (p.slots == 1 && cls >= a.hdr->first[level + 1])) {
        cp_async_commit();
        cp_async_wait<0>();
        return;
    }
    const int P = a.hdr->P[cls];
    const float *lambda_cls = p.lambda + ((x_slot * p.blocks + block) * node_rows(a, p.x_slots) + node_first(a, p.x_slots, cls)) * a.block;
    float *out_cls = p.out + (box * node_rows(a, p.slots) + node_first(a, p.slots, cls)) * p.kq + k0;
    bool finite = true;

    for (int p0 = 0; p0 < P; p0 += CP_NODES) {
        const int Pn = min(CP_NODES, P - p0), quads = (Pn + 3) / 4, units = quads * groups;
        for (int u0 = 0; u0 < units; u0 += 32) {
            const int unit = u0 + lane;
            const bool mine = unit < units;
            const int q = mine ? unit % quads : 0, c = mine ? (unit / quads) * 4 : 0;  // nodes q, q + quads, ..
            int at[4];
#pragma unroll
            for (int j = 0; j < 4; j++) at[j] = min(q + j * quads, Pn - 1) * CP_LS;
            f32x2 acc[4][2] = {};
            for (int step = 0; step < steps; step++) {
                const int r = step * CP_ROWS;
                if (steps > 1 || u0 == 0) {
                    __syncthreads();  // (what was there is done with)
                    const bool there = early && p0 == 0 && u0 == 0 && step == 0;
                    if ((steps > 1 || p0 == 0) && !there) fetch_rows(r);
                    const float *lambda = lambda_cls + p0 * a.block + r;
                    for (int n = warp; n < Pn; n += 4) cp_async16(ls + n * CP_LS + lane * 4, lambda + n * a.block + lane * 4);
                    cp_async_commit();
                    cp_async_wait<0>();
                    __syncthreads();
                }
#pragma unroll 2
                for (int i = warp * 32; i < warp * 32 + 32; i += 4) {
                    float l[4][4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float4 f = *reinterpret_cast<const float4 *>(ls + at[j] + i);
                        l[j][0] = f.x, l[j][1] = f.y, l[j][2] = f.z, l[j][3] = f.w;
                    }
#pragma unroll
                    for (int d = 0; d < 4; d++) {
                        const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(vs + (i + d) * COLS + c);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const f32x2 f = splat2(l[j][d]);
                            acc[j][0] = fma2(f, w.x, acc[j][0]), acc[j][1] = fma2(f, w.y, acc[j][1]);
                        }
                    }
                }
            }
            // [warp][j][lane][4]: a warp adds up the sums of one j
#pragma unroll
            for (int j = 0; j < 4; j++) *reinterpret_cast<ulonglong2 *>(parts + ((warp * 4 + j) * 32 + lane) * 4) = make_ulonglong2(acc[j][0], acc[j][1]);
            __syncthreads();
            float4 o = *reinterpret_cast<const float4 *>(parts + (warp * 32 + lane) * 4);
#pragma unroll
            for (int w = 1; w < 4; w++) {
                const float4 x = *reinterpret_cast<const float4 *>(parts + ((w * 4 + warp) * 32 + lane) * 4);
                o.x += x.x, o.y += x.y, o.z += x.z, o.w += x.w;
            }
            const int node = q + warp * quads;
            if (mine && node < Pn) {
                *reinterpret_cast<float4 *>(out_cls + (p0 + node) * p.kq + c) = o;
                finite = finite && fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fmaxf(fabsf(o.z), fabsf(o.w))) <= NODES_MAX_OPERAND &&
                         !isnan(o.x) && !isnan(o.y) && !isnan(o.z) && !isnan(o.w);
            }
            if (steps == 1 && u0 + 32 < units) __syncthreads();  // (parts are written again; elsewhere the next fetch waits)
        }
    }
    if (!finite) a.hdr->use = 0;  // (the kernels after this one see it)
}

// What the product and the gradient at the nodes share.  A CTA of four warps works on one batch and KC
// columns: on four row blocks, a warp each -- then nothing but the tables of phase factors is shared and no
// warp waits for another --, or, in problems with too few row blocks for that, on one, of whose band
// every warp takes every fourth column block.  Lanes own node rows:
// LANES lanes x RPT rows cover the P rows of the block and 32 / LANES column subsets share the warp, so
// that a shared-memory read of an operand row serves LANES * RPT entries per subset and no lane idles
// at the common P.  Per pair of blocks a lane keeps, for its rows, the distance to the column block's
// centre and cosine and sine of its phase; the phase factors of the column nodes are the same for every
// half-length, so an entry costs one SFU exponential and no sine or cosine.  All phase factors are
// evaluated with full precision, the distance of two centres reduced to half turns in fp64.
template <int KC>
struct NodeShape {
    static constexpr int QS = KC + 4;  // floats per staged operand row: column subsets fall into different banks
    // most rows per lane (registers: RPT * KC accumulators or left values)
    static constexpr int CTAS = KC <= 16 ? 4 : 3;  // per SM
    static constexpr int MAX_ROWS = KC <= 16 ? 4 : (KC == 24 ? 3 : 2);
    // shared memory for the warps' operand tiles: two stages while they fit, else one
    static constexpr int TILE_FLOATS = 4 * NODES_MAX * QS;
    // per half-length: offset, cos and sin of W offset of the nodes
    static constexpr int TABLE_FLOATS = NODES_LEVELS * 3 * NODES_MAX;
    static constexpr size_t SMEM = (TILE_FLOATS + TABLE_FLOATS) * sizeof(float);
};

// f(LANES, RPT) for the smallest layout that holds P rows.
template <int MAX_ROWS, typename F>
__device__ __forceinline__ void with_row_layout(int P, F f) {
    if (P <= 16) return f(Int<8>(), Int<2>());
    if constexpr (MAX_ROWS >= 3)
        if (P <= 24) return f(Int<8>(), Int<3>());
    if constexpr (MAX_ROWS >= 4) {
        if (P <= 32) return f(Int<8>(), Int<4>());
        if (P <= 48) return f(Int<16>(), Int<3>());
        if (P <= 64) return f(Int<16>(), Int<4>());
        return f(Int<32>(), Int<3>());
    }
    if (P <= 32) return f(Int<16>(), Int<2>());
    if constexpr (MAX_ROWS >= 3)
        if (P <= 48) return f(Int<16>(), Int<3>());
    if (P <= 64) return f(Int<32>(), Int<2>());
    return f(Int<32>(), Int<3>());
}

// Distance, phase factors and half-length of 32 of a warp's column blocks at a time, one per lane.
template <int KT>
struct NodePairs {
    float D = 0.0f, c = 1.0f, s = 0.0f;
    int level = 0;
    __device__ __forceinline__ void load(const KernelFn<KT> &fn, const NodesHeader *hdr, float row_centre, const float *centre2,
                                         const float *half2, int cb, int c_hi) {
        if (cb >= c_hi) return;
        D = row_centre - centre2[cb];
        level = level_of(hdr, half2[cb]);
        if constexpr (KernelFn<KT>::PHASE) {
            const double t = (double)fn.phase_half_turns() * (double)D;
            sincospif((float)(t - 2.0 * rint(0.5 * t)), &s, &c);
        }
    }
};

// Per node row of a lane: offset from the row block's centre, cos and sin of W times it; and, for the
// current column block, distance to its centre (y) and cos and sin of W times that (rc, rs).
template <int KT, int LANES, int RPT>
struct NodeRows {
    float d[RPT], cw[RPT], sw[RPT];
    f32x2 y[RPT], rc[RPT], rs[RPT];
    __device__ __forceinline__ void init(const float *table, int row, int P) {
#pragma unroll
        for (int i = 0; i < RPT; i++) {
            const int q = row + LANES * i;
            d[i] = q < P ? table[q] : 0.0f;
            cw[i] = q < P ? table[NODES_MAX + q] : 1.0f;
            sw[i] = q < P ? table[2 * NODES_MAX + q] : 0.0f;
        }
    }
    __device__ __forceinline__ void pair(float D, float c, float s) {
#pragma unroll
        for (int i = 0; i < RPT; i++) {
            y[i] = splat2(D + d[i]);
            if constexpr (KernelFn<KT>::PHASE) {
                rc[i] = splat2(c * cw[i] - s * sw[i]);
                rs[i] = splat2(s * cw[i] + c * sw[i]);
            }
        }
    }
};

// Everything about a CTA's work item.
template <int KT, int KC>
struct NodeItem {
    int64_t b, r;
    int chunk, k0, kc, c_lo, c_hi, c_step, P, row_class, stages, stage_floats;
    bool idle;  // a warp of the last CTA without a row block
    int col_P[NODES_LEVELS], col_class[NODES_LEVELS];
    KernelFn<KT> fn;
    float row_centre;
    const NodesHeader *hdr;
    const float *centre2, *half2;
    float *tiles, *tables, *row_table;

    // `wpr`: warps per row block, 1 or 4
    __device__ __forceinline__ void init(const NodesArgs &a, int64_t kq, int wpr, float *smem, BatchIndex *bi_out) {
        hdr = a.hdr;
        const int warp = threadIdx.x >> 5;
        int64_t item = blockIdx.x;
        b = item % a.batch.count;
        item /= a.batch.count;
        const int64_t groups = wpr == 1 ? (a.R + 3) / 4 : a.R;
        r = item % groups;
        chunk = (int)(item / groups);
        if (wpr == 1) r = r * 4 + warp;
        idle = r >= a.R;
        if (idle) r = a.R - 1;
        const BatchIndex bi = decompose(a.batch, b);
        *bi_out = bi;
        k0 = chunk * KC;
        kc = (int)min((int64_t)KC, kq - k0);  // a multiple of 4
        fn.init(batch_ptr(a.params, bi), a.params.s0);
        if (a.order1 != nullptr) {
            c_lo = 0;
            c_hi = idle ? 0 : (int)a.C;
        } else {
            const int s = batch_ptr(a.start, bi)[r * a.start.s0], e = batch_ptr(a.end, bi)[r * a.end.s0];
            c_lo = s < e ? s / KM_BLOCK_SIZE : 0;
            c_hi = s < e && !idle ? (int)((min((int64_t)e, a.n) + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE) : 0;
        }
        c_step = wpr;
        if (wpr > 1) c_lo += warp;
        const int64_t row_box = (a.slots1 == 1 ? 0 : b) * a.R + r;
        row_centre = a.centre1[row_box];
        const int row_level = level_of(hdr, a.half1[row_box]);
        centre2 = a.centre2 + (a.slots2 == 1 ? 0 : b) * a.C;
        half2 = a.half2 + (a.slots2 == 1 ? 0 : b) * a.C;
        tables = smem + NodeShape<KC>::TILE_FLOATS;
        row_table = tables + row_level * 3 * NODES_MAX;
#pragma unroll
        for (int l = 0; l < NODES_LEVELS; l++) {
            col_class[l] = a.classes[b * NODES_LEVELS + l];
            col_P[l] = hdr->P[col_class[l]];
            float *t = tables + l * 3 * NODES_MAX;
            for (int q = threadIdx.x; q < col_P[l]; q += 128) {
                const float d = hdr->delta[col_class[l]][q];
                float c = 1.0f, sn = 0.0f;
                if constexpr (KernelFn<KT>::PHASE) sincospif(fn.phase_half_turns() * d, &sn, &c);
                t[q] = d, t[NODES_MAX + q] = c, t[2 * NODES_MAX + q] = sn;
            }
            if (l == row_level) P = col_P[l], row_class = col_class[l];
        }
        // The most nodes this kernel has at any half-length: NOT always those of the longest, as every level of
        // the plan merges its smaller classes into larger ones by itself.
        stage_floats = max(max(col_P[0], col_P[1]), max(col_P[2], col_P[3])) * NodeShape<KC>::QS;
        static_assert(NODES_LEVELS == 4, "stage_floats");
        stages = 8 * stage_floats <= NodeShape<KC>::TILE_FLOATS ? 2 : 1;
        tiles = smem + (threadIdx.x >> 5) * stages * stage_floats;
        __syncthreads();
    }

    // One column block's operand rows (Pc x KC of an array with rows of kq) into this warp's stage.
    __device__ __forceinline__ void stage(const float *src, int64_t kq, int Pc, int which) const {
        const int lane = threadIdx.x & 31;
        float *to = tiles + which * stage_floats;
        for (int q = lane; q < Pc * (KC / 4); q += 32) {
            const int j = q / (KC / 4), c4 = (q % (KC / 4)) * 4;
            if (c4 < kc)
                cp_async16(to + j * NodeShape<KC>::QS + c4, src + j * kq + c4);
            else
                *reinterpret_cast<float4 *>(to + j * NodeShape<KC>::QS + c4) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        cp_async_commit();
    }

    // Calls body(D, c, s, Pc, table, tile) for each of this warp's column blocks; `operand`: column k0 of
    // an array [column block][block_rows][kq] that has this kernel's nodes of level l at row first[l].
    template <typename Body>
    __device__ __forceinline__ void walk(const NodesArgs &a, const float *operand, int64_t slots, int64_t kq, Body body) const {
        const int lane = threadIdx.x & 31;
        const int64_t block = node_rows(a, slots) * kq;
        int first[NODES_LEVELS];
#pragma unroll
        for (int l = 0; l < NODES_LEVELS; l++) first[l] = node_first(a, slots, col_class[l]);
        const auto pick = [](const int (&v)[NODES_LEVELS], int l) { return l == 0 ? v[0] : (l == 1 ? v[1] : (l == 2 ? v[2] : v[3])); };
        static_assert(NODES_LEVELS == 4, "pick");
        const auto fetch = [&](int cb, int level, int which) { stage(operand + cb * block + pick(first, level) * kq, kq, pick(col_P, level), which); };
        NodePairs<KT> now, next;  // this group of 32 column blocks and the one after it
        next.load(fn, hdr, row_centre, centre2, half2, c_lo + c_step * lane, c_hi);
        int at = 0;
        for (int cb = c_lo; cb < c_hi; cb += c_step, at++) {
            if (at % 32 == 0) {
                now = next;
                next.load(fn, hdr, row_centre, centre2, half2, cb + c_step * (lane + 32), c_hi);
                if (at == 0) fetch(cb, __shfl_sync(0xffffffffu, now.level, 0), 0);
            }
            const bool more = cb + c_step < c_hi;
            const int ahead = at % 32 == 31 ? __shfl_sync(0xffffffffu, next.level, 0) : __shfl_sync(0xffffffffu, now.level, (at + 1) % 32);
            if (stages == 2 && more) {
                fetch(cb + c_step, ahead, (at + 1) & 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncwarp();
            const float D = __shfl_sync(0xffffffffu, now.D, at % 32), c = __shfl_sync(0xffffffffu, now.c, at % 32),
                        s = __shfl_sync(0xffffffffu, now.s, at % 32);
            const int level = __shfl_sync(0xffffffffu, now.level, at % 32);
            body(D, c, s, pick(col_P, level), tables + level * 3 * NODES_MAX, tiles + (stages == 2 ? (at & 1) : 0) * stage_floats);
            __syncwarp();
            if (stages == 1 && more) fetch(cb + c_step, ahead, 0);
        }
    }
};

// One operand row of a tile as packed pairs.
template <int KC>
__device__ __forceinline__ void load_node_row(const float *tile, int j, f32x2 (&rv)[KC / 2]) {
#pragma unroll
    for (int c4 = 0; c4 < KC / 4; c4++) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(tile + j * NodeShape<KC>::QS + c4 * 4);
        rv[2 * c4] = v.x, rv[2 * c4 + 1] = v.y;
    }
}

struct NodesProductArgs {
    NodesArgs a;
    int64_t kq;
    int64_t q_slots;   // 1: one compressed rhs for all batches
    int k_chunks, wpr;
    const float *Q;    // [slot][column block][nodes][kq]
    View<float> out;
    int out_vec;
};

// Product at the nodes and back to the rows.  The lanes accumulate KC sums per row with packed FMAs, the
// four warps' sums meet in shared memory, and thread = row forms lambda_1 times them.
template <int KT, int KC>
__global__ void __launch_bounds__(128, NodeShape<KC>::CTAS) nodes_product_kernel(const NodesProductArgs p) {
    const NodesArgs &a = p.a;
    grid_wait();
    if (!a.hdr->use) return;
    using Fn = KernelFn<KT>;
    constexpr int KC2 = KC / 2, QS = NodeShape<KC>::QS;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, lane = tid & 31;
    NodeItem<KT, KC> it;
    BatchIndex bi;
    it.init(a, p.kq, p.wpr, smem, &bi);
    const Fn fn = it.fn;
    const int P = it.P;
    const float *Q = p.Q + (p.q_slots == 1 ? 0 : it.b) * a.C * node_rows(a, p.q_slots) * p.kq + it.k0;

    with_row_layout<NodeShape<KC>::MAX_ROWS>(P, [&](auto lanes, auto rows_per_lane) {
        constexpr int LANES = decltype(lanes)::value, RPT = decltype(rows_per_lane)::value, SUBSETS = 32 / LANES;
        const int row = lane % LANES, subset = lane / LANES;
        NodeRows<KT, LANES, RPT> rows;
        rows.init(it.row_table, row, P);
        f32x2 acc[RPT][KC2];
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int c = 0; c < KC2; c++) acc[i][c] = 0ull;
        it.walk(a, Q, p.q_slots, p.kq, [&](float D, float c, float s, int Pc, const float *table, const float *tile) {
            rows.pair(D, c, s);
            for (int j = 2 * subset; j < Pc; j += 2 * SUBSETS) {
                const f32x2 dj = *reinterpret_cast<const f32x2 *>(table + j);
                [[maybe_unused]] f32x2 cj = 0ull, sj = 0ull;
                if constexpr (Fn::PHASE) {
                    cj = *reinterpret_cast<const f32x2 *>(table + NODES_MAX + j);
                    sj = *reinterpret_cast<const f32x2 *>(table + 2 * NODES_MAX + j);
                }
                f32x2 kv[RPT];
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    f32x2 cs = 0ull;
                    if constexpr (Fn::PHASE) cs = fma2(rows.rc[i], cj, mul2(rows.rs[i], sj));
                    kv[i] = fn.unscaled2_ph(sub2(rows.y[i], dj), cs, 0ull);
                }
                f32x2 rv[KC2];
                load_node_row<KC>(tile, j, rv);
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    float k_even, k_odd;
                    unpack2(kv[i], k_even, k_odd);
                    const f32x2 kk = splat2(k_even);
#pragma unroll
                    for (int c = 0; c < KC2; c++) acc[i][c] = fma2(kk, rv[c], acc[i][c]);
                }
                load_node_row<KC>(tile, j + 1, rv);
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    float k_even, k_odd;
                    unpack2(kv[i], k_even, k_odd);
                    const f32x2 kk = splat2(k_odd);
#pragma unroll
                    for (int c = 0; c < KC2; c++) acc[i][c] = fma2(kk, rv[c], acc[i][c]);
                }
            }
        });
#pragma unroll
        for (int i = 0; i < RPT; i++) {
#pragma unroll
            for (int c = 0; c < KC2; c++) {
                float v0, v1;
                unpack2(acc[i][c], v0, v1);
#pragma unroll
                for (int o = LANES; o < 32; o <<= 1) {
                    v0 += __shfl_xor_sync(0xffffffffu, v0, o);
                    v1 += __shfl_xor_sync(0xffffffffu, v1, o);
                }
                if (subset == 0 && row + LANES * i < P)
                    *reinterpret_cast<float2 *>(it.tiles + (row + LANES * i) * QS + 2 * c) = make_float2(v0, v1);
            }
        }
    });
    const float *sums = it.tiles;  // [P][QS]
    if (p.wpr == 1) {
        __syncwarp();
    } else {
        __syncthreads();
        const int warp_floats = it.stages * it.stage_floats;
        for (int q = tid; q < P * KC; q += 128) {
            const int e = (q / KC) * QS + q % KC;
            smem[e] = (smem[e] + smem[warp_floats + e]) + (smem[2 * warp_floats + e] + smem[3 * warp_floats + e]);
        }
        sums = smem;
        __syncthreads();
    }
    if (it.idle) return;

    // rows: out[row] = sum_q lambda[q][row] * sums[q].  A lane forms OC columns of its rows at a time: the
    // sums come from shared memory as broadcasts, whose cost is the registers they fill, so that
    // each one read should serve several rows.
    const float *lambda = a.lambda1 + (((a.slots1 == 1 ? 0 : it.b) * a.R + it.r) * node_rows(a, a.slots1) +
                                       node_first(a, a.slots1, it.row_class)) * a.block;
    const auto expand = [&](auto rows_per_lane, int row0) {
        constexpr int OR = decltype(rows_per_lane)::value, OC = KC >= 8 ? 8 : 4;
        for (int g = 0; g < KC / OC; g++) {
            const int k_here = (int)min((int64_t)OC, a.k - it.k0 - g * OC);
            if (k_here <= 0) break;
            f32x2 o2[OR][OC / 2];
#pragma unroll
            for (int i = 0; i < OR; i++)
#pragma unroll
                for (int c = 0; c < OC / 2; c++) o2[i][c] = 0ull;
#pragma unroll 4
            for (int q = 0; q < P; q++) {
                f32x2 rv[OC / 2];
#pragma unroll
                for (int c4 = 0; c4 < OC / 4; c4++) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(sums + q * QS + g * OC + c4 * 4);
                    rv[2 * c4] = v.x, rv[2 * c4 + 1] = v.y;
                }
#pragma unroll
                for (int i = 0; i < OR; i++) {
                    const f32x2 l = splat2(lambda[q * a.block + row0 + lane + 32 * i] * fn.scale);
#pragma unroll
                    for (int c = 0; c < OC / 2; c++) o2[i][c] = fma2(l, rv[c], o2[i][c]);
                }
            }
#pragma unroll
            for (int i = 0; i < OR; i++) {
                const int64_t row = it.r * a.block + row0 + lane + 32 * i;
                if (row >= a.m) break;
                float *out = batch_ptr(p.out, bi) + point_row(a.order1, row) * p.out.s0 + (it.k0 + g * OC) * p.out.s1;
#pragma unroll
                for (int c4 = 0; c4 < OC / 4; c4++) {
                    float4 v;
                    unpack2(o2[i][2 * c4], v.x, v.y);
                    unpack2(o2[i][2 * c4 + 1], v.z, v.w);
                    if (p.out_vec && c4 * 4 + 4 <= k_here) {
                        *reinterpret_cast<float4 *>(out + c4 * 4) = v;
                    } else {
                        const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            if (c4 * 4 + u < k_here) out[(c4 * 4 + u) * p.out.s1] = w[u];
                    }
                }
            }
        }
    };
    if (p.wpr == 1)
        for (int row0 = 0; row0 < a.block; row0 += 128) expand(Int<4>(), row0);
    else if (a.block == 128)
        expand(Int<1>(), 32 * (tid >> 5));
    else
        for (int row0 = 128 * (tid >> 5); row0 < a.block; row0 += 512) expand(Int<4>(), row0);
}

struct NodesGradArgs {
    NodesArgs a;
    int64_t kq;
    int64_t l_slots, r_slots;
    int k_chunks, wpr;
    const float *L, *Rt;  // compressed left [slot][row block][nodes][kq], right [slot][column block][nodes][kq]
    float *partials;      // [batch][row block][chunk][KM_MAX_PARAMS]
};

// The gradient's sums at the nodes: the left values of a lane's node rows stay in registers, the
// coefficient of an entry is KC / 2 packed FMAs, and the factors of d kappa / d p are added up as in the
// direct kernels.
template <int KT, int KC>
__global__ void __launch_bounds__(128, NodeShape<KC>::CTAS) nodes_grad_kernel(const NodesGradArgs p) {
    const NodesArgs &a = p.a;
    grid_wait();
    if (!a.hdr->use) return;
    using Fn = KernelFn<KT>;
    constexpr int KC2 = KC / 2, NS = Fn::NSUMS;
    extern __shared__ __align__(16) float smem[];
    __shared__ float warp_sums[4][KM_MAX_PARAMS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    NodeItem<KT, KC> it;
    BatchIndex bi;
    it.init(a, p.kq, p.wpr, smem, &bi);
    const Fn fn = it.fn;
    const int P = it.P;
    const float *L = p.L + (((p.l_slots == 1 ? 0 : it.b) * a.R + it.r) * node_rows(a, p.l_slots) + node_first(a, p.l_slots, it.row_class)) * p.kq + it.k0;
    const float *Rt = p.Rt + (p.r_slots == 1 ? 0 : it.b) * a.C * node_rows(a, p.r_slots) * p.kq + it.k0;

    f32x2 sums2[NS];
#pragma unroll
    for (int q = 0; q < NS; q++) sums2[q] = 0ull;
    with_row_layout<NodeShape<KC>::MAX_ROWS>(P, [&](auto lanes, auto rows_per_lane) {
        constexpr int LANES = decltype(lanes)::value, RPT = decltype(rows_per_lane)::value, SUBSETS = 32 / LANES;
        const int row = lane % LANES, subset = lane / LANES;
        NodeRows<KT, LANES, RPT> rows;
        rows.init(it.row_table, row, P);
        f32x2 lv[RPT][KC2];  // (zero for rows past P: their coefficients vanish)
#pragma unroll
        for (int i = 0; i < RPT; i++) {
            const bool valid = row + LANES * i < P;
#pragma unroll
            for (int c4 = 0; c4 < KC / 4; c4++) {
                ulonglong2 v = make_ulonglong2(0ull, 0ull);
                if (valid && c4 * 4 < it.kc) v = *reinterpret_cast<const ulonglong2 *>(L + (row + LANES * i) * p.kq + c4 * 4);
                lv[i][2 * c4] = v.x, lv[i][2 * c4 + 1] = v.y;
            }
        }
        it.walk(a, Rt, p.r_slots, p.kq, [&](float D, float c, float s, int Pc, const float *table, const float *tile) {
            rows.pair(D, c, s);
            for (int j = 2 * subset; j < Pc; j += 2 * SUBSETS) {
                const f32x2 dj = *reinterpret_cast<const f32x2 *>(table + j);
                [[maybe_unused]] f32x2 cj = 0ull, sj = 0ull;
                if constexpr (Fn::PHASE) {
                    cj = *reinterpret_cast<const f32x2 *>(table + NODES_MAX + j);
                    sj = *reinterpret_cast<const f32x2 *>(table + 2 * NODES_MAX + j);
                }
                float co[RPT][2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    f32x2 rv[KC2];
                    load_node_row<KC>(tile, j + h, rv);
#pragma unroll
                    for (int i = 0; i < RPT; i++) {
                        f32x2 t = mul2(lv[i][0], rv[0]);
#pragma unroll
                        for (int c = 1; c < KC2; c++) t = fma2(lv[i][c], rv[c], t);
                        float t0, t1;
                        unpack2(t, t0, t1);
                        co[i][h] = t0 + t1;
                    }
                }
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    f32x2 cs = 0ull, sn = 0ull;
                    if constexpr (Fn::PHASE) {
                        cs = fma2(rows.rc[i], cj, mul2(rows.rs[i], sj));
                        sn = sub2(mul2(rows.rs[i], cj), mul2(rows.rc[i], sj));
                    }
                    fn.accumulate2_ph(sub2(rows.y[i], dj), cs, sn, pack2(co[i][0], co[i][1]), sums2);
                }
            }
        });
    });
    fn.rescale_ph(sums2);
#pragma unroll
    for (int q = 0; q < NS; q++) {
        float v, v_hi;
        unpack2(sums2[q], v, v_hi);
        v += v_hi;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) warp_sums[warp][q] = v;
    }
    float *record = p.partials + ((it.b * a.R + it.r) * p.k_chunks + it.chunk) * KM_MAX_PARAMS;
    if (p.wpr == 1) {
        __syncwarp();
        if (!it.idle && lane < KM_MAX_PARAMS) record[lane] = lane < NS ? warp_sums[warp][lane] : 0.0f;
        return;
    }
    __syncthreads();
    if (tid < KM_MAX_PARAMS) {
        float v = 0.0f;
        if (tid < NS) v = (warp_sums[0][tid] + warp_sums[1][tid]) + (warp_sums[2][tid] + warp_sums[3][tid]);
        record[tid] = v;
    }
}

// ------------------------------------------------------------------------------ host side

// All batch strides zero: one row for all batches.
template <typename T>
static bool shared_by_batches(const View<T> &v, const Batch &b) {
    for (int d = 0; d < b.ndim; d++)
        if (b.size[d] > 1 && v.bs[d] != 0) return false;
    return true;
}

// The node counts for which interpolation is the faster way.  Per entry the kernels here take about
// 4.5 + 0.75 k issue slots per 32 entries; the tensor-core kernels 11 - 15, whatever k.  (128 / P)^2 fewer entries make
// up for that up to P = 64 at 32 columns and up to P = 48 beyond.
static int nodes_limit(int64_t k) { return k <= 16 ? NODES_MAX : (k <= 32 ? 64 : 48); }

// Columns per CTA: chunks of at most 32, all of one width.
static int nodes_kc(int64_t k) {
    if (k <= 4) return 4;
    if (k <= 8) return 8;
    if (k <= 16) return 16;
    const int64_t per = ceil_div(k, ceil_div(k, 32));
    return per <= 16 ? 16 : (per <= 24 ? 24 : 32);
}

// A warp per row block once that gives every SM its 12 - 16 warps; four warps below.
static int nodes_warps_per_row_block(int64_t items) { return items >= 148 * 12 ? 1 : 4; }

// Points per block where all rows see all columns: enough blocks for the GPU, few enough nodes.
static int nodes_sorted_block(int64_t points) { return points >= (1 << 16) ? 1024 : (points >= (1 << 14) ? 512 : 256); }

struct NodesLayout {
    int64_t slots1, slots2, R, C, kq;
    bool same;
    int max_p, cap, block;
    bool sorted;
    size_t sort1, sort2, order1, order2;
    size_t classes, centre1, centre2, half1, half2, lambda1, lambda2, ops[2], partials, direct, total;
    int64_t op_slots[2];

    static size_t up(size_t v) { return (v + 255) / 256 * 256; }
    // operands: rhs of a product (right[0] null), or left and right of a gradient
    NodesLayout(const Batch &b, int64_t m, int64_t n, int64_t k, const View<const float> &x1, const View<const float> &x2,
                const View<const float> *left, const View<const float> &right, bool all_columns, size_t direct_bytes) {
        slots1 = shared_by_batches(x1, b) ? 1 : b.count;
        slots2 = shared_by_batches(x2, b) ? 1 : b.count;
        sorted = all_columns && slots1 == 1 && slots2 == 1;
        block = sorted ? nodes_sorted_block(std::max(m, n)) : KM_BLOCK_SIZE;
        R = ceil_div(m, block);
        C = ceil_div(n, block);
        kq = ceil_div(k, 4) * 4;
        max_p = nodes_limit(k);
        // Where batches share their points every class needs its own Lagrange matrices and operands: room
        // for several node counts, as long as it is not much memory.
        cap = std::max<int>(max_p, R + C <= 16384 ? 160 : 96);
        same = m == n && x1.data == x2.data && x1.s0 == x2.s0;
        for (int d = 0; d < b.ndim; d++) same = same && (b.size[d] == 1 || x1.bs[d] == x2.bs[d]);
        op_slots[1] = shared_by_batches(right, b) && slots2 == 1 ? 1 : b.count;
        op_slots[0] = left == nullptr ? 0 : (shared_by_batches(*left, b) && slots1 == 1 ? 1 : b.count);
        size_t at = up(sizeof(NodesHeader));
        const auto take = [&](size_t bytes) {
            const size_t here = at;
            at += up(bytes);
            return here;
        };
        const auto nodes = [&](int64_t slots) { return (size_t)(slots == 1 && b.count > 1 ? cap : max_p) * slots; };
        classes = take((size_t)(b.count * NODES_LEVELS) * sizeof(int));
        centre1 = take((size_t)(slots1 * R) * sizeof(float));
        centre2 = same ? centre1 : take((size_t)(slots2 * C) * sizeof(float));
        half1 = take((size_t)(slots1 * R) * sizeof(float));
        half2 = same ? half1 : take((size_t)(slots2 * C) * sizeof(float));
        lambda1 = take(nodes(slots1) * R * block * sizeof(float));
        lambda2 = same ? lambda1 : take(nodes(slots2) * C * block * sizeof(float));
        sort1 = take(sorted ? sizeof(SortTables) : 0);
        sort2 = same ? sort1 : take(sorted ? sizeof(SortTables) : 0);
        order1 = take(sorted ? (size_t)m * sizeof(int) : 0);
        order2 = same ? order1 : take(sorted ? (size_t)n * sizeof(int) : 0);
        ops[0] = take(op_slots[0] == 0 ? 0 : nodes(op_slots[0]) * R * kq * sizeof(float));
        ops[1] = take(nodes(op_slots[1]) * C * kq * sizeof(float));
        partials = take(left == nullptr ? 0 : (size_t)(b.count * R * ceil_div(k, nodes_kc(k))) * KM_MAX_PARAMS * sizeof(float));
        direct = take(direct_bytes);
        total = at;
    }
};

// `side` 0: left / row blocks, 1: right / column blocks.
static int nodes_compress(const NodesArgs &a, const NodesLayout &l, const View<const float> &v, int side, float *out, cudaStream_t s) {
    CompressArgs c;
    c.a = a;
    c.rows = side == 0 ? a.m : a.n, c.kq = l.kq, c.blocks = side == 0 ? l.R : l.C;
    c.slots = l.op_slots[side], c.x_slots = side == 0 ? l.slots1 : l.slots2;
    c.vec = a.k % 4 == 0 && rows_vectorizable(v, a.batch);
    c.v = v;
    c.order = side == 0 ? a.order1 : a.order2;
    c.half = side == 0 ? a.half1 : a.half2, c.lambda = side == 0 ? a.lambda1 : a.lambda2;
    c.out = out;
    const auto launch = [&](auto cols) {
        constexpr int COLS = decltype(cols)::value;
        const cudaError_t err = cudaFuncSetAttribute(nodes_compress_kernel<COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)CompressShape<COLS>::SMEM);
        if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(interpolation)");
        // (a shared operand: a CTA per class that the plan may have made -- one per kernel at most --, of which many
        // return at once; 12 000 that do take 30 us)
        const dim3 grid((unsigned)(c.slots * c.blocks * ceil_div(l.kq, COLS)),
                        c.slots == 1 ? (unsigned)std::min<int64_t>(a.batch.count, NODES_CLASSES_PER_LEVEL) : 1);
        return launch_chained("interpolation: operand launch", nodes_compress_kernel<COLS>, grid, 128, CompressShape<COLS>::SMEM, s, c);
    };
    return l.kq <= 16 ? launch(Int<16>()) : launch(Int<32>());
}

static int nodes_begin(NodesArgs &a, const NodesLayout &l, int kernel_type, unsigned char *ws, cudaStream_t s) {
    a.R = l.R, a.C = l.C, a.slots1 = l.slots1, a.slots2 = l.slots2, a.same = l.same ? 1 : 0, a.max_p = l.max_p, a.cap = l.cap;
    a.classes = reinterpret_cast<int *>(ws + l.classes);
    a.half1 = reinterpret_cast<float *>(ws + l.half1), a.half2 = reinterpret_cast<float *>(ws + l.half2);
    a.hdr = reinterpret_cast<NodesHeader *>(ws);
    a.centre1 = reinterpret_cast<float *>(ws + l.centre1), a.centre2 = reinterpret_cast<float *>(ws + l.centre2);
    a.lambda1 = reinterpret_cast<float *>(ws + l.lambda1), a.lambda2 = reinterpret_cast<float *>(ws + l.lambda2);
    cudaError_t err = cudaMemsetAsync(ws, 0, NODES_ZEROED, s);
    if (err != cudaSuccess) return cuda_fail(err, "interpolation: cudaMemsetAsync");
    a.block = l.block;
    a.order1 = a.order2 = nullptr;
    if (l.sorted) {
        int rc = sort_points(a.x1, a.m, reinterpret_cast<SortTables *>(ws + l.sort1), reinterpret_cast<int *>(ws + l.order1), &a.hdr->bad, s);
        if (rc == KM_OK && !l.same)
            rc = sort_points(a.x2, a.n, reinterpret_cast<SortTables *>(ws + l.sort2), reinterpret_cast<int *>(ws + l.order2), &a.hdr->bad, s);
        if (rc != KM_OK) return rc;
        a.order1 = reinterpret_cast<const int *>(ws + l.order1), a.order2 = reinterpret_cast<const int *>(ws + l.order2);
    }
    const int64_t boxes = l.slots1 * l.R + (l.same ? 0 : l.slots2 * l.C), work = std::max(ceil_div(boxes, PLAN_WARPS), ceil_div(a.batch.count * ceil_div(a.m, KM_BLOCK_SIZE), PLAN_THREADS));
    nodes_plan_kernel<<<(unsigned)std::min<int64_t>(work, 148 * 2), PLAN_THREADS, 0, s>>>(a, kernel_type);
    KM_CHECK_LAUNCH("interpolation: plan launch");
    return launch_chained("interpolation: Lagrange matrices launch", nodes_lambda_kernel, (unsigned)(boxes * (l.block / 128)), 128, 0, s, a);
}

template <int KT, int KC>
static int launch_nodes_product(const NodesProductArgs &p, cudaStream_t s) {
    auto kernel = nodes_product_kernel<KT, KC>;
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NodeShape<KC>::SMEM);
    if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(interpolation)");
    return launch_chained("interpolation: product launch", kernel, (unsigned)(p.a.batch.count * (p.wpr == 1 ? ceil_div(p.a.R, 4) : p.a.R) * p.k_chunks),
                          128, NodeShape<KC>::SMEM, s, p);
}
template <int KT, int KC>
static int launch_nodes_grad(const NodesGradArgs &p, cudaStream_t s) {
    auto kernel = nodes_grad_kernel<KT, KC>;
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NodeShape<KC>::SMEM);
    if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(interpolation)");
    return launch_chained("interpolation: gradient launch", kernel, (unsigned)(p.a.batch.count * (p.wpr == 1 ? ceil_div(p.a.R, 4) : p.a.R) * p.k_chunks),
                          128, NodeShape<KC>::SMEM, s, p);
}
#define KM_NODES_DISPATCH(launch, args)                                                                \
    [&](int kt, int kc) {                                                                              \
        const auto width = [&](auto t) {                                                               \
            constexpr int KT = decltype(t)::value;                                                     \
            switch (kc) {                                                                              \
            case 4: return launch<KT, 4>(args, s);                                                     \
            case 8: return launch<KT, 8>(args, s);                                                     \
            case 16: return launch<KT, 16>(args, s);                                                   \
            case 24: return launch<KT, 24>(args, s);                                                   \
            default: return launch<KT, 32>(args, s);                                                   \
            }                                                                                          \
        };                                                                                             \
        switch (kt) {                                                                                  \
        case KM_KERNEL_RBF: return width(std::integral_constant<int, KM_KERNEL_RBF>());                \
        case KM_KERNEL_SPECTRAL: return width(std::integral_constant<int, KM_KERNEL_SPECTRAL>());      \
        default: return width(std::integral_constant<int, KM_KERNEL_LOCALLY_PERIODIC>());              \
        }                                                                                              \
    }

// Sizes beyond which the interpolation is not tried (grid dimensions, workspace).
static bool nodes_fit(const Batch &b, int64_t m, int64_t n, int64_t k, const NodesLayout &l) {
    const int64_t most = 0x7fffffffLL;
    return m >= 1 && n >= 1 && k >= 1 && b.count >= 1 && l.slots1 * l.R + l.slots2 * l.C <= most && b.count <= most / l.R / ceil_div(k, 4) &&
           b.count <= most / l.C / ceil_div(k, 4) && l.total < ((size_t)1 << 36);
}

struct NodesCall {
    int64_t m, n, k;
    const km_batch *kb;
    const km_view *x1, *x2, *left, *right, *params, *start, *end;
};

static int nodes_arguments(const char *name, int kernel_type, const NodesCall &c, Batch *b) {
    KM_REQUIRE(valid_kernel_type(kernel_type), KM_ERR_INVALID_ARGUMENT, "%s: unknown kernel type %d", name, kernel_type);
    KM_REQUIRE(c.kb && c.x1 && c.x2 && c.right && c.params && c.start && c.end, KM_ERR_INVALID_ARGUMENT, "%s: null argument", name);
    KM_REQUIRE(c.m >= 1 && c.n >= 1 && c.k >= 1 && c.n <= 0x7fffffffLL - 64 && c.m <= 0x7fffffffLL, KM_ERR_INVALID_ARGUMENT,
               "%s: bad sizes m=%lld n=%lld k=%lld", name, (long long)c.m, (long long)c.n, (long long)c.k);
    const int rc = make_batch(c.kb, b);
    if (rc != KM_OK) return rc;
    KM_REQUIRE(b->count >= 1, KM_ERR_INVALID_ARGUMENT, "%s: empty batch", name);
    KM_REQUIRE(c.x1->data && c.x2->data && c.right->data && c.params->data && c.start->data && c.end->data && (!c.left || c.left->data),
               KM_ERR_INVALID_ARGUMENT, "%s: null data pointer", name);
    return KM_OK;
}

static size_t product_direct_bytes(const NodesCall &c) { return c.k >= 9 ? km_matmul_tc_workspace_bytes(c.kb, c.n, c.k, c.right) : 0; }
static size_t grad_direct_bytes(int kernel_type, const NodesCall &c) {
    return c.k >= 8 ? km_grad_tc_workspace_bytes(c.kb, c.m, c.n, c.k, c.right) : km_grad_workspace_bytes(kernel_type, c.kb, c.m);
}

static NodesLayout nodes_layout(const NodesCall &c, const Batch &b, bool all_columns, size_t direct_bytes) {
    View<const float> left;
    if (c.left) left = make_view<const float>(c.left, b);
    return NodesLayout(b, c.m, c.n, c.k, make_view<const float>(c.x1, b), make_view<const float>(c.x2, b), c.left ? &left : nullptr,
                       make_view<const float>(c.right, b), all_columns, direct_bytes);
}

static NodesArgs nodes_args(const NodesCall &c, const Batch &b) {
    NodesArgs a = {};
    a.batch = b;
    a.m = c.m, a.n = c.n, a.k = c.k;
    a.x1 = make_view<const float>(c.x1, b), a.x2 = make_view<const float>(c.x2, b);
    a.params = make_view<const float>(c.params, b);
    a.start = make_view<const int>(c.start, b), a.end = make_view<const int>(c.end, b);
    return a;
}

}  // namespace km

extern "C" size_t km_matmul_nodes_workspace_bytes(const km_batch *batch, int64_t m, int64_t n, int64_t k, const km_view *x1,
                                                  const km_view *x2, const km_view *rhs, int32_t all_columns) {
    using namespace km;
    Batch b;
    if (!batch || !x1 || !x2 || !rhs || m < 1 || n < 1 || k < 1 || make_batch(batch, &b) != KM_OK || b.count < 1) return 0;
    const NodesCall c = {m, n, k, batch, x1, x2, nullptr, rhs, nullptr, nullptr, nullptr};
    const NodesLayout l = nodes_layout(c, b, all_columns != 0, product_direct_bytes(c));
    return nodes_fit(b, m, n, k, l) ? l.total : 0;
}

extern "C" int km_matmul_nodes_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t k, const km_view *x1,
                                   const km_view *x2, const km_view *rhs, const km_view *params, const km_view *start,
                                   const km_view *end, const km_view *out, int32_t all_columns, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace km;
    Batch b;
    const NodesCall c = {m, n, k, batch, x1, x2, nullptr, rhs, params, start, end};
    int rc = nodes_arguments("km_matmul_nodes_f32", kernel_type, c, &b);
    if (rc != KM_OK) return rc;
    KM_REQUIRE(out && out->data, KM_ERR_INVALID_ARGUMENT, "km_matmul_nodes_f32: null argument");
    const NodesLayout l = nodes_layout(c, b, all_columns != 0, product_direct_bytes(c));
    KM_REQUIRE(nodes_fit(b, m, n, k, l), KM_ERR_UNSUPPORTED, "km_matmul_nodes_f32: too large");
    KM_REQUIRE(workspace != nullptr && workspace_bytes >= l.total && (uintptr_t)workspace % 256 == 0, KM_ERR_WORKSPACE,
               "km_matmul_nodes_f32: workspace of %zu bytes needed (256-byte aligned), %zu given", l.total, workspace_bytes);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (k >= 9) {
        rc = matmul_tc_prepare(b, k, make_view<const float>(rhs, b), ws + l.direct, s);
        if (rc != KM_OK) return rc;
    }
    NodesProductArgs p;
    p.a = nodes_args(c, b);
    rc = nodes_begin(p.a, l, kernel_type, ws, s);
    if (rc != KM_OK) return rc;
    p.kq = l.kq, p.q_slots = l.op_slots[1];
    float *Q = reinterpret_cast<float *>(ws + l.ops[1]);
    p.Q = Q;
    rc = nodes_compress(p.a, l, make_view<const float>(rhs, b), 1, Q, s);
    if (rc != KM_OK) return rc;
    p.out = make_view<float>(out, b);
    p.out_vec = p.out.s1 == 1 && p.out.s0 % 4 == 0 && (uintptr_t)p.out.data % 16 == 0;
    for (int d = 0; d < b.ndim; d++) p.out_vec = p.out_vec && p.out.bs[d] % 4 == 0;
    const int kc = nodes_kc(k);
    p.k_chunks = (int)ceil_div(k, kc);
    p.wpr = nodes_warps_per_row_block(b.count * l.R * p.k_chunks);
    rc = KM_NODES_DISPATCH(launch_nodes_product, p)(kernel_type, kc);
    if (rc != KM_OK) return rc;
    const Gate gate = {&p.a.hdr->use, 0};
    if (k >= 9)
        return matmul_tc_direct(kernel_type, batch, m, n, k, x1, x2, rhs, params, start, end, out, ws + l.direct, l.total - l.direct,
                                gate, stream);
    return matmul_direct(kernel_type, batch, m, n, k, x1, x2, rhs, params, start, end, out, gate, stream);
}

extern "C" size_t km_grad_nodes_workspace_bytes(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t k,
                                                const km_view *x1, const km_view *x2, const km_view *left, const km_view *right,
                                                int32_t all_columns) {
    using namespace km;
    Batch b;
    if (!batch || !x1 || !x2 || !left || !right || m < 1 || n < 1 || k < 1 || make_batch(batch, &b) != KM_OK || b.count < 1) return 0;
    const NodesCall c = {m, n, k, batch, x1, x2, left, right, nullptr, nullptr, nullptr};
    const NodesLayout l = nodes_layout(c, b, all_columns != 0, grad_direct_bytes(kernel_type, c));
    return nodes_fit(b, m, n, k, l) ? l.total : 0;
}

extern "C" int km_bilinear_derivative_nodes_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t k,
                                                const km_view *x1, const km_view *x2, const km_view *left, const km_view *right,
                                                const km_view *params, const km_view *start, const km_view *end,
                                                const km_view *grad, int32_t all_columns, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace km;
    Batch b;
    const NodesCall c = {m, n, k, batch, x1, x2, left, right, params, start, end};
    KM_REQUIRE(left != nullptr && grad && grad->data, KM_ERR_INVALID_ARGUMENT, "km_bilinear_derivative_nodes_f32: null argument");
    int rc = nodes_arguments("km_bilinear_derivative_nodes_f32", kernel_type, c, &b);
    if (rc != KM_OK) return rc;
    const NodesLayout l = nodes_layout(c, b, all_columns != 0, grad_direct_bytes(kernel_type, c));
    KM_REQUIRE(nodes_fit(b, m, n, k, l), KM_ERR_UNSUPPORTED, "km_bilinear_derivative_nodes_f32: too large");
    KM_REQUIRE(workspace != nullptr && workspace_bytes >= l.total && (uintptr_t)workspace % 256 == 0, KM_ERR_WORKSPACE,
               "km_bilinear_derivative_nodes_f32: workspace of %zu bytes needed (256-byte aligned), %zu given", l.total, workspace_bytes);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    NodesGradArgs p;
    p.a = nodes_args(c, b);
    rc = nodes_begin(p.a, l, kernel_type, ws, s);
    if (rc != KM_OK) return rc;
    p.kq = l.kq, p.l_slots = l.op_slots[0], p.r_slots = l.op_slots[1];
    float *L = reinterpret_cast<float *>(ws + l.ops[0]), *Rt = reinterpret_cast<float *>(ws + l.ops[1]);
    p.L = L, p.Rt = Rt;
    rc = nodes_compress(p.a, l, make_view<const float>(left, b), 0, L, s);
    if (rc != KM_OK) return rc;
    rc = nodes_compress(p.a, l, make_view<const float>(right, b), 1, Rt, s);
    if (rc != KM_OK) return rc;
    const int kc = nodes_kc(k);
    p.k_chunks = (int)ceil_div(k, kc);
    p.wpr = nodes_warps_per_row_block(b.count * l.R * p.k_chunks);
    p.partials = reinterpret_cast<float *>(ws + l.partials);
    rc = KM_NODES_DISPATCH(launch_nodes_grad, p)(kernel_type, kc);
    if (rc != KM_OK) return rc;
    rc = launch_grad_finish(kernel_type, b, l.R * p.k_chunks, p.partials, false, p.a.params, make_view<float>(grad, b), s,
                            Gate{&p.a.hdr->use, 1});
    if (rc != KM_OK) return rc;
    const Gate gate = {&p.a.hdr->use, 0};
    return (k >= 8 ? grad_tc_direct : grad_direct)(kernel_type, batch, m, n, k, x1, x2, left, right, params, start, end, grad,
                                                   ws + l.direct, l.total - l.direct, gate, stream);
}
