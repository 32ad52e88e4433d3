// Products and gradients by blockwise interpolation (km_nodes.cuh has the method and its error bound).
//
// A call is: extents of the blocks and choice of P (nodes_plan_kernel), Lagrange matrices
// (nodes_lambda_kernel), rhs / left / right at the nodes (nodes_compress_kernel), then the product
// (nodes_product_kernel, which also takes its result back to the 128 rows) or the gradient
// (nodes_grad_kernel).  Whether the call may be done this way is decided on the device: bands aligned
// to blocks and P within bounds.  The kernels of the direct evaluation are launched behind it and
// return at once if it was; the interpolation kernels return at once if not.  So no call waits for
// the host, and inputs without short intervals (unsorted points without a cutoff, frequencies of many
// periods per block) are computed as they always were.
#include <type_traits>

#include "km_nodes.cuh"

namespace km {

// First bytes of the workspace, zero on entry to the plan kernel.
struct NodesHeader {
    int max_h_bits;  // largest half-length of any block (bits of a non-negative float)
    int bad;         // some band is not aligned to blocks, or an input is not finite
    int done;        // CTAs of the plan kernel that have finished
    int P;
    int use;         // 1: interpolate, 0: evaluate directly
};

struct NodesArgs {
    Batch batch;
    int64_t m, n, k;
    int64_t R, C;       // row and column blocks
    int64_t slots1, slots2;  // distinct x1 / x2 rows: batch.count, or 1 if all batches share one
    int same;           // x1 and x2 are the same points
    int max_p;
    View<const float> x1, x2, params;
    View<const int> start, end;
    NodesHeader *hdr;
    NodeBox *box1, *box2;    // [slot][block]
    float *lambda1, *lambda2;  // [slot][block][P][128]
};

__device__ __forceinline__ int nodes_needed_for(int kt, const float *theta, int64_t stride, float h, int lane) {
    if (kt == KM_KERNEL_RBF) return nodes_needed<KM_KERNEL_RBF>(theta, stride, h, lane);
    if (kt == KM_KERNEL_SPECTRAL) return nodes_needed<KM_KERNEL_SPECTRAL>(theta, stride, h, lane);
    return nodes_needed<KM_KERNEL_LOCALLY_PERIODIC>(theta, stride, h, lane);
}

// Extents of every block (a warp each), alignment of every band, and -- the CTA that finishes last --
// the number of nodes for the longest interval over all kernels of the batch.
__global__ void __launch_bounds__(256) nodes_plan_kernel(const NodesArgs a, int kernel_type) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * 8, first = blockIdx.x * 8LL + (threadIdx.x >> 5);
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
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t row = block * KM_BLOCK_SIZE + lane + 32 * i;
            if (row < rows) {
                const float e = base[row * x.s0];
                lo = fminf(lo, e);
                hi = fmaxf(hi, e);
                nan = nan || !(fabsf(e) < INFINITY);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        const float c = 0.5f * lo + 0.5f * hi, h = fmaxf(fmaxf(hi - c, c - lo), NODES_MIN_H);
        bad |= nan || !(h < INFINITY);
        longest = fmaxf(longest, h);
        if (lane == 0) (one ? a.box1 : a.box2)[v] = NodeBox{c, h};
    }
    const int64_t threads = (int64_t)gridDim.x * blockDim.x;
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < a.batch.count * a.R; w += threads) {
        const BatchIndex bi = decompose(a.batch, w / a.R);
        const int64_t r = w % a.R;
        const int s = batch_ptr(a.start, bi)[r * a.start.s0], e = batch_ptr(a.end, bi)[r * a.end.s0];
        if (s >= e) continue;  // an empty band
        bad |= s < 0 || s % KM_BLOCK_SIZE != 0 || (e < a.n && e % KM_BLOCK_SIZE != 0);
    }
    __shared__ int s_last, s_p;
    if (lane == 0) atomicMax(&a.hdr->max_h_bits, __float_as_int(longest));
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        if (bad) a.hdr->bad = 1;
        __threadfence();
        s_last = atomicAdd(&a.hdr->done, 1) == (int)gridDim.x - 1;
        s_p = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const float h = __int_as_float(*reinterpret_cast<volatile int *>(&a.hdr->max_h_bits));
    const bool any_bad = *reinterpret_cast<volatile int *>(&a.hdr->bad) != 0;
    for (int64_t b = threadIdx.x >> 5; b < a.batch.count; b += 8) {
        const int p = nodes_needed_for(kernel_type, batch_ptr(a.params, decompose(a.batch, b)), a.params.s0, h, lane);
        if (lane == 0) atomicMax(&s_p, p);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int P = max(4, (min(s_p, 4096) + 3) & ~3);
        a.hdr->P = P;
        a.hdr->use = !any_bad && P <= a.max_p;
    }
}

// Lagrange matrix of one block: thread = row, lambda[q][row] = (w_q / (x - xi_q)) / sum of the same.
__global__ void __launch_bounds__(128) nodes_lambda_kernel(const NodesArgs a) {
    if (!a.hdr->use) return;
    const int P = a.hdr->P;
    __shared__ float delta[NODES_MAX], weight[NODES_MAX];
    const int64_t boxes1 = a.slots1 * a.R;
    const bool one = blockIdx.x < boxes1;
    const int64_t v = one ? blockIdx.x : blockIdx.x - boxes1, blocks = one ? a.R : a.C, rows = one ? a.m : a.n;
    const NodeBox box = (one ? a.box1 : a.box2)[v];
    const View<const float> &x = one ? a.x1 : a.x2;
    const int t = threadIdx.x;
    if (t < P) delta[t] = node_offset(box.h, t, P);
    __syncthreads();
    if (t < P) weight[t] = node_weight(delta, box.h, t, P);
    __syncthreads();
    const int64_t row = (v % blocks) * KM_BLOCK_SIZE + t;
    float *out = (one ? a.lambda1 : a.lambda2) + v * P * KM_BLOCK_SIZE + t;
    if (row >= rows) {
        for (int q = 0; q < P; q++) out[q * KM_BLOCK_SIZE] = 0.0f;
        return;
    }
    const float d = batch_ptr(x, decompose(a.batch, v / blocks))[row * x.s0] - box.c;
    // (differences in units of h: an interval may be as short as NODES_MIN_H)
    const float inv_h = 1.0f / box.h;
    float sum = 0.0f;
    int hit = -1;
    for (int q = 0; q < P; q++) {
        const float e = (d - delta[q]) * inv_h;
        if (e == 0.0f) hit = q;
        sum += weight[q] / e;
    }
    const float inv = 1.0f / sum;
    for (int q = 0; q < P; q++) {
        const float e = (d - delta[q]) * inv_h;
        out[q * KM_BLOCK_SIZE] = hit >= 0 ? (q == hit ? 1.0f : 0.0f) : (weight[q] / e) * inv;
    }
}

// Lambda^T of one operand: out[slot][block][q][c] = sum_row lambda[q][row] * v[row][c], columns padded
// to kq = a multiple of 4 with zeros.
struct CompressArgs {
    Batch batch;
    int64_t rows, k, kq, blocks, slots;
    int64_t lambda_slots;  // 1: one Lagrange matrix per block for all batches
    View<const float> v;
    const float *lambda;
    float *out;
    const NodesHeader *hdr;
};

constexpr int CP_ROWS = 64, CP_COLS = 32;

// One CTA per (slot, block, 32 columns).  A thread owns (node, 4 columns) pairs; rows are staged
// 64 at a time.  Bound by the shared-memory reads (two per four FMAs); the whole pass is a few per cent
// of the direct evaluation it replaces.
__global__ void __launch_bounds__(128) nodes_compress_kernel(const CompressArgs a) {
    if (!a.hdr->use) return;
    const int P = a.hdr->P;
    __shared__ float ls[NODES_MAX][CP_ROWS + 1];
    __shared__ __align__(16) float vs[CP_ROWS][CP_COLS];
    const int64_t chunks = ceil_div(a.kq, CP_COLS);
    const int64_t chunk = blockIdx.x % chunks, box = blockIdx.x / chunks, slot = box / a.blocks, block = box % a.blocks;
    const int k0 = (int)chunk * CP_COLS, kc = (int)min((int64_t)CP_COLS, a.kq - k0);  // a multiple of 4
    const float *v = batch_ptr(a.v, decompose(a.batch, slot));
    const float *lambda = a.lambda + ((a.lambda_slots == 1 ? 0 : slot) * a.blocks + block) * P * KM_BLOCK_SIZE;
    float *out = a.out + box * P * a.kq + k0;
    const int t = threadIdx.x;
    constexpr int UNITS = NODES_MAX * (CP_COLS / 4) / 128;
    float acc[UNITS][4] = {};
    const int groups = kc / 4, units = P * groups;
    for (int half = 0; half < KM_BLOCK_SIZE / CP_ROWS; half++) {
        const int64_t row0 = block * KM_BLOCK_SIZE + half * CP_ROWS;
        if (row0 >= a.rows) break;
        __syncthreads();
        for (int e = t; e < P * CP_ROWS; e += 128) ls[e / CP_ROWS][e % CP_ROWS] = lambda[(e / CP_ROWS) * KM_BLOCK_SIZE + half * CP_ROWS + e % CP_ROWS];
        for (int e = t; e < CP_ROWS * kc; e += 128) {
            const int i = e / kc, c = e % kc;
            vs[i][c] = (row0 + i < a.rows && k0 + c < a.k) ? v[(row0 + i) * a.v.s0 + (k0 + c) * a.v.s1] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < UNITS; u++) {
            const int unit = t + 128 * u;
            if (unit >= units) break;
            const int q = unit % P, c = (unit / P) * 4;
#pragma unroll 8
            for (int i = 0; i < CP_ROWS; i++) {
                const float l = ls[q][i];
                const float4 w = *reinterpret_cast<const float4 *>(&vs[i][c]);
                acc[u][0] = fmaf(l, w.x, acc[u][0]);
                acc[u][1] = fmaf(l, w.y, acc[u][1]);
                acc[u][2] = fmaf(l, w.z, acc[u][2]);
                acc[u][3] = fmaf(l, w.w, acc[u][3]);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < UNITS; u++) {
        const int unit = t + 128 * u;
        if (unit >= units) break;
        *reinterpret_cast<float4 *>(out + (unit % P) * a.kq + (unit / P) * 4) = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
    }
}

// The kernel values of node rows against the nodes of one column block.  Per pair of blocks a lane
// keeps, for its node rows, the distance to the column block's centre and the cosine and sine of its
// phase; per node of the column block the offset and the phase factors lie in shared memory, so an
// entry costs one SFU exponential (as in the tensor-core kernels).  The factors are evaluated with
// full precision, the distance of the centres reduced to half turns in fp64: a few values per pair.
template <int KT>
struct NodePair {
    using Fn = KernelFn<KT>;
    static __device__ __forceinline__ void column_factors(const Fn &fn, float delta, float &c, float &s) {
        c = 1.0f, s = 0.0f;
        if constexpr (Fn::PHASE) sincospif(fn.phase_half_turns() * delta, &s, &c);
    }
    // cos, sin of W (D + delta)
    static __device__ __forceinline__ void row_factors(const Fn &fn, float D, float delta, float &c, float &s) {
        c = 1.0f, s = 0.0f;
        if constexpr (Fn::PHASE) {
            const double t = (double)fn.phase_half_turns() * (double)D;
            sincospif((float)(t - 2.0 * rint(0.5 * t)) + fn.phase_half_turns() * delta, &s, &c);
        }
    }
};

struct NodesProductArgs {
    NodesArgs a;
    int64_t kq;
    int64_t q_slots;   // 1: one compressed rhs for all batches
    int k_chunks;
    const float *Q;    // [slot][column block][P][kq]
    View<float> out;
    int out_vec;
};

// Product at the nodes and back to the rows: one CTA of four warps per (batch, row block, KC columns).
// Each warp takes every fourth column block of the band: it stages the block's compressed rhs
// (P x KC) in its own part of shared memory, its lanes hold node rows (two rows each beyond 32 nodes; two
// or four column subsets per warp up to 16 or 8) and accumulate KC sums per row with packed FMAs.  The four
// warps' sums meet in shared memory, and thread = row forms lambda_1 times them.
// Per entry: about 4.5 issue slots of kernel value, KC / 2 of FMA and KC / 4 + 1 shared-memory reads.
template <int KT, int KC>
__global__ void __launch_bounds__(128) nodes_product_kernel(const NodesProductArgs p) {
    const NodesArgs &a = p.a;
    if (!a.hdr->use) return;
    const int P = a.hdr->P;
    using Fn = KernelFn<KT>;
    constexpr int KC2 = KC / 2;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *qs = smem + warp * (NODES_MAX * KC);                     // [P][KC]; later this warp's sums
    float *cf = smem + 4 * NODES_MAX * KC + warp * (3 * NODES_MAX);  // offset, cosine, sine of the column nodes
    float *unit = smem + 4 * NODES_MAX * KC + 4 * 3 * NODES_MAX;     // offsets for h = 1

    int64_t item = blockIdx.x;
    const int64_t b = item % a.batch.count;
    item /= a.batch.count;
    const int64_t r = item % a.R;
    const int k0 = (int)(item / a.R) * KC;
    const BatchIndex bi = decompose(a.batch, b);
    Fn fn;
    fn.init(batch_ptr(a.params, bi), a.params.s0);
    const int s = batch_ptr(a.start, bi)[r * a.start.s0], e = batch_ptr(a.end, bi)[r * a.end.s0];
    const int c_lo = s < e ? s / KM_BLOCK_SIZE : 0;
    const int c_hi = s < e ? (int)((min((int64_t)e, a.n) + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE) : 0;
    const NodeBox rbox = a.box1[(a.slots1 == 1 ? 0 : b) * a.R + r];
    const NodeBox *cbox = a.box2 + (a.slots2 == 1 ? 0 : b) * a.C;
    const float *Q = p.Q + (p.q_slots == 1 ? 0 : b) * a.C * P * p.kq + k0;
    const int kc = (int)min((int64_t)KC, p.kq - k0);  // a multiple of 4

    if (tid < P) unit[tid] = node_offset(1.0f, tid, P);
    __syncthreads();

    auto walk = [&](auto rows_per_lane) {
        constexpr int RPT = decltype(rows_per_lane)::value;
        const int width = P <= 8 ? 8 : (P <= 16 ? 16 : 32);  // lanes per column subset
        const int row = lane & (width - 1), subset = lane / width, subsets = 32 / width;
        float dr[RPT];
#pragma unroll
        for (int i = 0; i < RPT; i++) dr[i] = row + 32 * i < P ? rbox.h * unit[row + 32 * i] : 0.0f;
        f32x2 acc[RPT][KC2];
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int c = 0; c < KC2; c++) acc[i][c] = 0ull;
        for (int cb = c_lo + warp; cb < c_hi; cb += 4) {
            const NodeBox box = cbox[cb];
            const float *src = Q + (int64_t)cb * P * p.kq;
            __syncwarp();
            for (int q = lane; q < P * (KC / 4); q += 32) {
                const int j = q / (KC / 4), c4 = (q % (KC / 4)) * 4;
                if (c4 < kc)
                    cp_async16(qs + j * KC + c4, src + j * p.kq + c4);
                else
                    *reinterpret_cast<float4 *>(qs + j * KC + c4) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            cp_async_commit();
            for (int j = lane; j < P; j += 32) {
                const float dj = box.h * unit[j];
                float c, sn;
                NodePair<KT>::column_factors(fn, dj, c, sn);
                cf[j] = dj;
                if constexpr (Fn::PHASE) cf[NODES_MAX + j] = c, cf[2 * NODES_MAX + j] = sn;
            }
            const float D = rbox.c - box.c;
            f32x2 y[RPT], rc[RPT], rs[RPT];
#pragma unroll
            for (int i = 0; i < RPT; i++) {
                float c, sn;
                NodePair<KT>::row_factors(fn, D, dr[i], c, sn);
                y[i] = splat2(D + dr[i]), rc[i] = splat2(c), rs[i] = splat2(sn);
            }
            cp_async_wait<0>();
            __syncwarp();
#pragma unroll 2
            for (int j = 2 * subset; j < P; j += 2 * subsets) {
                const f32x2 dj = *reinterpret_cast<const f32x2 *>(cf + j);
                [[maybe_unused]] f32x2 cj = 0ull, sj = 0ull;
                if constexpr (Fn::PHASE) {
                    cj = *reinterpret_cast<const f32x2 *>(cf + NODES_MAX + j);
                    sj = *reinterpret_cast<const f32x2 *>(cf + 2 * NODES_MAX + j);
                }
                f32x2 kv[RPT];
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    const f32x2 cs = Fn::PHASE ? fma2(rc[i], cj, mul2(rs[i], sj)) : 0ull;
                    kv[i] = fn.unscaled2_ph(sub2(y[i], dj), cs, 0ull);
                }
                f32x2 rv[KC2];
                load_staged_row2<KC>(qs, j, rv);
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    float k_even, k_odd;
                    unpack2(kv[i], k_even, k_odd);
                    const f32x2 kk = splat2(k_even);
#pragma unroll
                    for (int c = 0; c < KC2; c++) acc[i][c] = fma2(kk, rv[c], acc[i][c]);
                }
                load_staged_row2<KC>(qs, j + 1, rv);
#pragma unroll
                for (int i = 0; i < RPT; i++) {
                    float k_even, k_odd;
                    unpack2(kv[i], k_even, k_odd);
                    const f32x2 kk = splat2(k_odd);
#pragma unroll
                    for (int c = 0; c < KC2; c++) acc[i][c] = fma2(kk, rv[c], acc[i][c]);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < RPT; i++) {
#pragma unroll
            for (int c = 0; c < KC2; c++) {
                float v0, v1;
                unpack2(acc[i][c], v0, v1);
                for (int o = width; o < 32; o <<= 1) {
                    v0 += __shfl_xor_sync(0xffffffffu, v0, o);
                    v1 += __shfl_xor_sync(0xffffffffu, v1, o);
                }
                if (subset == 0 && row + 32 * i < P) {
                    qs[(row + 32 * i) * KC + 2 * c] = v0;
                    qs[(row + 32 * i) * KC + 2 * c + 1] = v1;
                }
            }
        }
    };
    if (P <= 32)
        walk(std::integral_constant<int, 1>());
    else
        walk(std::integral_constant<int, 2>());
    __syncthreads();
    for (int q = tid; q < P * KC; q += 128)
        smem[q] = ((smem[q] + smem[NODES_MAX * KC + q]) + (smem[2 * NODES_MAX * KC + q] + smem[3 * NODES_MAX * KC + q])) * fn.scale;
    __syncthreads();

    // rows: out[row] = sum_q lambda[q][row] * sums[q]
    const int64_t row = r * KM_BLOCK_SIZE + tid;
    if (row >= a.m) return;
    const float *lambda = a.lambda1 + ((a.slots1 == 1 ? 0 : b) * a.R + r) * P * KM_BLOCK_SIZE + tid;
    f32x2 o2[KC2];
#pragma unroll
    for (int c = 0; c < KC2; c++) o2[c] = 0ull;
#pragma unroll 4
    for (int q = 0; q < P; q++) {
        const f32x2 l = splat2(lambda[q * KM_BLOCK_SIZE]);
        f32x2 rv[KC2];
        load_staged_row2<KC>(smem, q, rv);
#pragma unroll
        for (int c = 0; c < KC2; c++) o2[c] = fma2(l, rv[c], o2[c]);
    }
    float *out = batch_ptr(p.out, bi) + row * p.out.s0 + k0 * p.out.s1;
    const int k_here = (int)min((int64_t)KC, a.k - k0);
#pragma unroll
    for (int c4 = 0; c4 < KC / 4; c4++) {
        float4 v;
        unpack2(o2[2 * c4], v.x, v.y);
        unpack2(o2[2 * c4 + 1], v.z, v.w);
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

struct NodesGradArgs {
    NodesArgs a;
    int64_t kq;
    int64_t l_slots, r_slots;
    int k_chunks;
    const float *L, *Rt;  // compressed left [slot][row block][P][kq], right [slot][column block][P][kq]
    float *partials;      // [batch][row block][chunk][KM_MAX_PARAMS]
};

// The gradient's sums at the nodes: the same walk, with the left values of a lane's node rows in
// registers, the coefficient of an entry KC / 2 packed FMAs, and the factors of d kappa / d p added up
// as in the direct kernels.
template <int KT, int KC>
__global__ void __launch_bounds__(128) nodes_grad_kernel(const NodesGradArgs p) {
    const NodesArgs &a = p.a;
    if (!a.hdr->use) return;
    const int P = a.hdr->P;
    using Fn = KernelFn<KT>;
    constexpr int KC2 = KC / 2, NS = Fn::NSUMS;
    extern __shared__ __align__(16) float smem[];
    __shared__ float warp_sums[4][KM_MAX_PARAMS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *qs = smem + warp * (NODES_MAX * KC);
    float *cf = smem + 4 * NODES_MAX * KC + warp * (3 * NODES_MAX);
    float *unit = smem + 4 * NODES_MAX * KC + 4 * 3 * NODES_MAX;

    int64_t item = blockIdx.x;
    const int64_t b = item % a.batch.count;
    item /= a.batch.count;
    const int64_t r = item % a.R;
    const int chunk = (int)(item / a.R), k0 = chunk * KC;
    const BatchIndex bi = decompose(a.batch, b);
    Fn fn;
    fn.init(batch_ptr(a.params, bi), a.params.s0);
    const int s = batch_ptr(a.start, bi)[r * a.start.s0], e = batch_ptr(a.end, bi)[r * a.end.s0];
    const int c_lo = s < e ? s / KM_BLOCK_SIZE : 0;
    const int c_hi = s < e ? (int)((min((int64_t)e, a.n) + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE) : 0;
    const NodeBox rbox = a.box1[(a.slots1 == 1 ? 0 : b) * a.R + r];
    const NodeBox *cbox = a.box2 + (a.slots2 == 1 ? 0 : b) * a.C;
    const float *L = p.L + ((p.l_slots == 1 ? 0 : b) * a.R + r) * P * p.kq + k0;
    const float *Rt = p.Rt + (p.r_slots == 1 ? 0 : b) * a.C * P * p.kq + k0;
    const int kc = (int)min((int64_t)KC, p.kq - k0);

    if (tid < P) unit[tid] = node_offset(1.0f, tid, P);
    __syncthreads();

    f32x2 sums2[NS];
#pragma unroll
    for (int q = 0; q < NS; q++) sums2[q] = 0ull;
    auto walk = [&](auto rows_per_lane) {
        constexpr int RPT = decltype(rows_per_lane)::value;
        const int width = P <= 8 ? 8 : (P <= 16 ? 16 : 32);
        const int row = lane & (width - 1), subset = lane / width, subsets = 32 / width;
        float dr[RPT];
        f32x2 lv[RPT][KC2];
#pragma unroll
        for (int i = 0; i < RPT; i++) {
            const bool valid = row + 32 * i < P;
            dr[i] = valid ? rbox.h * unit[row + 32 * i] : 0.0f;
#pragma unroll
            for (int c4 = 0; c4 < KC / 4; c4++) {
                ulonglong2 v = make_ulonglong2(0ull, 0ull);
                if (valid && c4 * 4 < kc) v = *reinterpret_cast<const ulonglong2 *>(L + (row + 32 * i) * p.kq + c4 * 4);
                lv[i][2 * c4] = v.x, lv[i][2 * c4 + 1] = v.y;
            }
        }
        for (int cb = c_lo + warp; cb < c_hi; cb += 4) {
            const NodeBox box = cbox[cb];
            const float *src = Rt + (int64_t)cb * P * p.kq;
            __syncwarp();
            for (int q = lane; q < P * (KC / 4); q += 32) {
                const int j = q / (KC / 4), c4 = (q % (KC / 4)) * 4;
                if (c4 < kc)
                    cp_async16(qs + j * KC + c4, src + j * p.kq + c4);
                else
                    *reinterpret_cast<float4 *>(qs + j * KC + c4) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            cp_async_commit();
            for (int j = lane; j < P; j += 32) {
                const float dj = box.h * unit[j];
                float c, sn;
                NodePair<KT>::column_factors(fn, dj, c, sn);
                cf[j] = dj;
                if constexpr (Fn::PHASE) cf[NODES_MAX + j] = c, cf[2 * NODES_MAX + j] = sn;
            }
            const float D = rbox.c - box.c;
            f32x2 y[RPT], rc[RPT], rs[RPT];
#pragma unroll
            for (int i = 0; i < RPT; i++) {
                float c, sn;
                NodePair<KT>::row_factors(fn, D, dr[i], c, sn);
                y[i] = splat2(D + dr[i]), rc[i] = splat2(c), rs[i] = splat2(sn);
            }
            cp_async_wait<0>();
            __syncwarp();
            for (int j = 2 * subset; j < P; j += 2 * subsets) {
                const f32x2 dj = *reinterpret_cast<const f32x2 *>(cf + j);
                [[maybe_unused]] f32x2 cj = 0ull, sj = 0ull;
                if constexpr (Fn::PHASE) {
                    cj = *reinterpret_cast<const f32x2 *>(cf + NODES_MAX + j);
                    sj = *reinterpret_cast<const f32x2 *>(cf + 2 * NODES_MAX + j);
                }
                float co[RPT][2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    f32x2 rv[KC2];
                    load_staged_row2<KC>(qs, j + h, rv);
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
                        cs = fma2(rc[i], cj, mul2(rs[i], sj));
                        sn = sub2(mul2(rs[i], cj), mul2(rc[i], sj));
                    }
                    fn.accumulate2_ph(sub2(y[i], dj), cs, sn, pack2(co[i][0], co[i][1]), sums2);
                }
            }
        }
    };
    if (P <= 32)
        walk(std::integral_constant<int, 1>());
    else
        walk(std::integral_constant<int, 2>());
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
    __syncthreads();
    if (tid < KM_MAX_PARAMS) {
        float v = 0.0f;
        if (tid < NS) v = (warp_sums[0][tid] + warp_sums[1][tid]) + (warp_sums[2][tid] + warp_sums[3][tid]);
        p.partials[((b * a.R + r) * p.k_chunks + chunk) * KM_MAX_PARAMS + tid] = v;
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
static int nodes_limit(int64_t k) { return k <= 32 ? 64 : 48; }

// Columns per CTA: chunks of at most 32, all of one width.
static int nodes_kc(int64_t k) {
    if (k <= 4) return 4;
    if (k <= 8) return 8;
    if (k <= 16) return 16;
    const int64_t per = ceil_div(k, ceil_div(k, 32));
    return per <= 16 ? 16 : (per <= 24 ? 24 : 32);
}

struct NodesLayout {
    int64_t slots1, slots2, R, C, kq;
    bool same;
    int max_p;
    size_t box1, box2, lambda1, lambda2, ops[2], partials, direct, total;
    int64_t op_slots[2];

    static size_t up(size_t v) { return (v + 255) / 256 * 256; }
    // operands: rhs of a product (right[0] null), or left and right of a gradient
    NodesLayout(const Batch &b, int64_t m, int64_t n, int64_t k, const View<const float> &x1, const View<const float> &x2,
                const View<const float> *left, const View<const float> &right, size_t direct_bytes) {
        slots1 = shared_by_batches(x1, b) ? 1 : b.count;
        slots2 = shared_by_batches(x2, b) ? 1 : b.count;
        R = ceil_div(m, KM_BLOCK_SIZE);
        C = ceil_div(n, KM_BLOCK_SIZE);
        kq = ceil_div(k, 4) * 4;
        max_p = nodes_limit(k);
        same = m == n && x1.data == x2.data && x1.s0 == x2.s0;
        for (int d = 0; d < b.ndim; d++) same = same && (b.size[d] == 1 || x1.bs[d] == x2.bs[d]);
        op_slots[1] = shared_by_batches(right, b) && slots2 == 1 ? 1 : b.count;
        op_slots[0] = left == nullptr ? 0 : (shared_by_batches(*left, b) && slots1 == 1 ? 1 : b.count);
        size_t at = 256;
        const auto take = [&](size_t bytes) {
            const size_t here = at;
            at += up(bytes);
            return here;
        };
        const size_t per_block = (size_t)max_p * KM_BLOCK_SIZE * sizeof(float);
        box1 = take((size_t)(slots1 * R) * sizeof(NodeBox));
        box2 = same ? box1 : take((size_t)(slots2 * C) * sizeof(NodeBox));
        lambda1 = take((size_t)(slots1 * R) * per_block);
        lambda2 = same ? lambda1 : take((size_t)(slots2 * C) * per_block);
        ops[0] = take((size_t)(op_slots[0] * R * max_p * kq) * sizeof(float));
        ops[1] = take((size_t)(op_slots[1] * C * max_p * kq) * sizeof(float));
        partials = take(left == nullptr ? 0 : (size_t)(b.count * R * ceil_div(k, nodes_kc(k))) * KM_MAX_PARAMS * sizeof(float));
        direct = take(direct_bytes);
        total = at;
    }
};

static int nodes_compress(const NodesArgs &a, const View<const float> &v, int64_t rows, int64_t blocks, int64_t kq, int64_t slots,
                          int64_t lambda_slots, const float *lambda, float *out, cudaStream_t s) {
    const CompressArgs c = {a.batch, rows, a.k, kq, blocks, slots, lambda_slots, v, lambda, out, a.hdr};
    const int64_t ctas = slots * blocks * ceil_div(kq, CP_COLS);
    nodes_compress_kernel<<<(unsigned)ctas, 128, 0, s>>>(c);
    KM_CHECK_LAUNCH("interpolation: operand launch");
    return KM_OK;
}

static int nodes_begin(NodesArgs &a, const NodesLayout &l, int kernel_type, unsigned char *ws, cudaStream_t s) {
    a.R = l.R, a.C = l.C, a.slots1 = l.slots1, a.slots2 = l.slots2, a.same = l.same ? 1 : 0, a.max_p = l.max_p;
    a.hdr = reinterpret_cast<NodesHeader *>(ws);
    a.box1 = reinterpret_cast<NodeBox *>(ws + l.box1), a.box2 = reinterpret_cast<NodeBox *>(ws + l.box2);
    a.lambda1 = reinterpret_cast<float *>(ws + l.lambda1), a.lambda2 = reinterpret_cast<float *>(ws + l.lambda2);
    cudaError_t err = cudaMemsetAsync(ws, 0, sizeof(NodesHeader), s);
    if (err != cudaSuccess) return cuda_fail(err, "interpolation: cudaMemsetAsync");
    const int64_t boxes = l.slots1 * l.R + (l.same ? 0 : l.slots2 * l.C), work = std::max(ceil_div(boxes, 8), ceil_div(a.batch.count * l.R, 256));
    nodes_plan_kernel<<<(unsigned)std::min<int64_t>(work, 148 * 4), 256, 0, s>>>(a, kernel_type);
    KM_CHECK_LAUNCH("interpolation: plan launch");
    nodes_lambda_kernel<<<(unsigned)boxes, 128, 0, s>>>(a);
    KM_CHECK_LAUNCH("interpolation: Lagrange matrices launch");
    return KM_OK;
}

template <int KC>
constexpr size_t nodes_smem() { return (size_t)(4 * NODES_MAX * KC + 4 * 3 * NODES_MAX + NODES_MAX) * sizeof(float); }

template <int KT, int KC>
static int launch_nodes_product(const NodesProductArgs &p, cudaStream_t s) {
    auto kernel = nodes_product_kernel<KT, KC>;
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nodes_smem<KC>());
    if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(interpolation)");
    kernel<<<(unsigned)(p.a.batch.count * p.a.R * p.k_chunks), 128, nodes_smem<KC>(), s>>>(p);
    KM_CHECK_LAUNCH("interpolation: product launch");
    return KM_OK;
}
template <int KT, int KC>
static int launch_nodes_grad(const NodesGradArgs &p, cudaStream_t s) {
    auto kernel = nodes_grad_kernel<KT, KC>;
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nodes_smem<KC>());
    if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(interpolation)");
    kernel<<<(unsigned)(p.a.batch.count * p.a.R * p.k_chunks), 128, nodes_smem<KC>(), s>>>(p);
    KM_CHECK_LAUNCH("interpolation: gradient launch");
    return KM_OK;
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

static NodesLayout nodes_layout(const NodesCall &c, const Batch &b, size_t direct_bytes) {
    View<const float> left;
    if (c.left) left = make_view<const float>(c.left, b);
    return NodesLayout(b, c.m, c.n, c.k, make_view<const float>(c.x1, b), make_view<const float>(c.x2, b), c.left ? &left : nullptr,
                       make_view<const float>(c.right, b), direct_bytes);
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
                                                  const km_view *x2, const km_view *rhs) {
    using namespace km;
    Batch b;
    if (!batch || !x1 || !x2 || !rhs || m < 1 || n < 1 || k < 1 || make_batch(batch, &b) != KM_OK || b.count < 1) return 0;
    const NodesCall c = {m, n, k, batch, x1, x2, nullptr, rhs, nullptr, nullptr, nullptr};
    const NodesLayout l = nodes_layout(c, b, product_direct_bytes(c));
    return nodes_fit(b, m, n, k, l) ? l.total : 0;
}

extern "C" int km_matmul_nodes_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t k, const km_view *x1,
                                   const km_view *x2, const km_view *rhs, const km_view *params, const km_view *start,
                                   const km_view *end, const km_view *out, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace km;
    Batch b;
    const NodesCall c = {m, n, k, batch, x1, x2, nullptr, rhs, params, start, end};
    int rc = nodes_arguments("km_matmul_nodes_f32", kernel_type, c, &b);
    if (rc != KM_OK) return rc;
    KM_REQUIRE(out && out->data, KM_ERR_INVALID_ARGUMENT, "km_matmul_nodes_f32: null argument");
    const NodesLayout l = nodes_layout(c, b, product_direct_bytes(c));
    KM_REQUIRE(nodes_fit(b, m, n, k, l), KM_ERR_UNSUPPORTED, "km_matmul_nodes_f32: too large");
    KM_REQUIRE(workspace != nullptr && workspace_bytes >= l.total && (uintptr_t)workspace % 256 == 0, KM_ERR_WORKSPACE,
               "km_matmul_nodes_f32: workspace of %zu bytes needed (256-byte aligned), %zu given", l.total, workspace_bytes);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    NodesProductArgs p;
    p.a = nodes_args(c, b);
    rc = nodes_begin(p.a, l, kernel_type, ws, s);
    if (rc != KM_OK) return rc;
    p.kq = l.kq, p.q_slots = l.op_slots[1];
    float *Q = reinterpret_cast<float *>(ws + l.ops[1]);
    p.Q = Q;
    rc = nodes_compress(p.a, make_view<const float>(rhs, b), n, l.C, l.kq, l.op_slots[1], l.slots2, p.a.lambda2, Q, s);
    if (rc != KM_OK) return rc;
    p.out = make_view<float>(out, b);
    p.out_vec = p.out.s1 == 1 && p.out.s0 % 4 == 0 && (uintptr_t)p.out.data % 16 == 0;
    for (int d = 0; d < b.ndim; d++) p.out_vec = p.out_vec && p.out.bs[d] % 4 == 0;
    const int kc = nodes_kc(k);
    p.k_chunks = (int)ceil_div(k, kc);
    rc = KM_NODES_DISPATCH(launch_nodes_product, p)(kernel_type, kc);
    if (rc != KM_OK) return rc;
    const Gate gate = {&p.a.hdr->use, 0};
    if (k >= 9)
        return matmul_tc_direct(kernel_type, batch, m, n, k, x1, x2, rhs, params, start, end, out, ws + l.direct, l.total - l.direct,
                                gate, stream);
    return matmul_direct(kernel_type, batch, m, n, k, x1, x2, rhs, params, start, end, out, gate, stream);
}

extern "C" size_t km_grad_nodes_workspace_bytes(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t k,
                                                const km_view *x1, const km_view *x2, const km_view *left, const km_view *right) {
    using namespace km;
    Batch b;
    if (!batch || !x1 || !x2 || !left || !right || m < 1 || n < 1 || k < 1 || make_batch(batch, &b) != KM_OK || b.count < 1) return 0;
    const NodesCall c = {m, n, k, batch, x1, x2, left, right, nullptr, nullptr, nullptr};
    const NodesLayout l = nodes_layout(c, b, grad_direct_bytes(kernel_type, c));
    return nodes_fit(b, m, n, k, l) ? l.total : 0;
}

extern "C" int km_bilinear_derivative_nodes_f32(int kernel_type, const km_batch *batch, int64_t m, int64_t n, int64_t k,
                                                const km_view *x1, const km_view *x2, const km_view *left, const km_view *right,
                                                const km_view *params, const km_view *start, const km_view *end,
                                                const km_view *grad, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace km;
    Batch b;
    const NodesCall c = {m, n, k, batch, x1, x2, left, right, params, start, end};
    KM_REQUIRE(left != nullptr && grad && grad->data, KM_ERR_INVALID_ARGUMENT, "km_bilinear_derivative_nodes_f32: null argument");
    int rc = nodes_arguments("km_bilinear_derivative_nodes_f32", kernel_type, c, &b);
    if (rc != KM_OK) return rc;
    const NodesLayout l = nodes_layout(c, b, grad_direct_bytes(kernel_type, c));
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
    rc = nodes_compress(p.a, make_view<const float>(left, b), m, l.R, l.kq, l.op_slots[0], l.slots1, p.a.lambda1, L, s);
    if (rc != KM_OK) return rc;
    rc = nodes_compress(p.a, make_view<const float>(right, b), n, l.C, l.kq, l.op_slots[1], l.slots2, p.a.lambda2, Rt, s);
    if (rc != KM_OK) return rc;
    const int kc = nodes_kc(k);
    p.k_chunks = (int)ceil_div(k, kc);
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
