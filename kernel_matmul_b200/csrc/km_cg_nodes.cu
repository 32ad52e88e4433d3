// The operator of a CG solve by blockwise interpolation (km_nodes.cuh has the method and its bound).
//
// A solve applies ONE operator many times, so what the products of km_nodes.cu form on every call is
// laid out once here: P nodes per block of 128 points (one interval length for all blocks), the
// Lagrange matrices, and the kernel matrix between the nodes,
//     G[r][c - c_lo(r)][q][p] = exp(-tau^2 / 2 l^2) sum_b s_b cos(2 pi f_b tau),   tau = xi_{r,p} - xi_{c,q},
// summed over all components of the operator: whatever their number, a product then reads
// P^2 values per pair of blocks instead of evaluating 128^2 x components.  An entry's error is a part of the
// kernel's MAXIMUM (km_nodes.cuh), as that of the tensor-core batch sum is, so only operators that run on that
// one otherwise are laid out: sums of 2 and more spectral components with one lengthscale, for up to
// KM_NODE_MAX_COLUMNS columns.  The FMA kernels that evaluate all others hold every entry to 1e-6 of ITSELF, and
// tens of CG steps bring a difference in the entries' last bits back a thousand times larger.  With P = 14 that is 0.56 GB for
// 4 million points and a band of 22 blocks; a product is 85 us of HBM time for it, 135 us for the vectors
// and Lagrange matrices, where the sum of 64 components took 11 ms on the tensor cores.
//
// An iteration is: p = r + beta p and Lambda^T p (node_compress_kernel), G times that, Lambda times the
// result, q = K p + sigma^2 p and p . q (node_product_kernel), then the updates of x and r (km_cg.cu).
#include <type_traits>

#include "km_cg.cuh"
#include "km_nodes.cuh"

namespace km {

constexpr int NODE_OP_MAX = 32;  // most nodes per block of an operator

struct NodePlan {
    long long lo, hi;        // columns read by the row blocks of the window
    long long checksum;      // of the whole band
    long long P;             // nodes per block; 0: not this way (band not aligned, several lengthscales, too many nodes)
    long long max_blocks;    // widest band of any row block, in blocks
    int max_h_bits, done, bad, width;
    int lo_bits, hi_bits;
};

struct NodePlanArgs {
    Batch batch;
    int64_t n, R, rb0, rb1;
    const float *x;
    int64_t xs;
    View<const float> params;
    const int *start, *end;
    float *centre;
    NodePlan *plan;
};

// (x null: lo, hi and checksum only, P 0)
__global__ void __launch_bounds__(256) node_plan_kernel(const NodePlanArgs a) {
    const int lane = threadIdx.x & 31;
    float longest = 0.0f;
    int bad = 0;
    for (int64_t v = blockIdx.x * 8LL + (threadIdx.x >> 5); a.x != nullptr && v < a.R; v += gridDim.x * 8LL) {
        float lo = INFINITY, hi = -INFINITY;
        bool nan = false;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t row = v * KM_BLOCK_SIZE + lane + 32 * i;
            if (row < a.n) {
                const float e = a.x[row * a.xs];
                lo = fminf(lo, e), hi = fmaxf(hi, e);
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
        if (lane == 0) a.centre[v] = c;
    }
    int first = INT_MAX, last = 0, width = 0;
    unsigned long long sum = 0;
    for (int64_t r = blockIdx.x * 256LL + threadIdx.x; r < a.R; r += gridDim.x * 256LL) {
        const int s = a.start[r], e = a.end[r];
        sum += (unsigned long long)(r + 1) * (31ull * (unsigned long long)s + (unsigned long long)e);
        if (r >= a.rb0 && r < a.rb1) first = min(first, s), last = max(last, e);
        if (s >= e) continue;
        bad |= s < 0 || s % KM_BLOCK_SIZE != 0 || (e < a.n && e % KM_BLOCK_SIZE != 0);
        width = max(width, (int)((min((int64_t)e, a.n) - s + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE));
    }
    first = __reduce_min_sync(0xffffffffu, first);
    last = __reduce_max_sync(0xffffffffu, last);
    width = __reduce_max_sync(0xffffffffu, width);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    __shared__ int s_last, s_p, s_lengthscales;
    bad = __syncthreads_or(bad);
    if (lane == 0) {
        atomicMax(&a.plan->max_h_bits, __float_as_int(longest));
        atomicMax(&a.plan->lo_bits, INT_MAX - first);
        atomicMax(&a.plan->hi_bits, last);
        atomicMax(&a.plan->width, width);
        atomicAdd(reinterpret_cast<unsigned long long *>(&a.plan->checksum), sum);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (bad) a.plan->bad = 1;
        __threadfence();
        s_last = atomicAdd(&a.plan->done, 1) == (int)gridDim.x - 1;
        s_p = a.x != nullptr ? 0 : 4096;
        s_lengthscales = 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    volatile NodePlan *plan = a.plan;
    const float h = __int_as_float(plan->max_h_bits);
    for (int64_t b = threadIdx.x >> 5; a.x != nullptr && b < a.batch.count; b += 8) {
        const float *theta = batch_ptr(a.params, decompose(a.batch, b));
        const int p = nodes_needed<KM_KERNEL_SPECTRAL>(theta, a.params.s0, h, lane);
        if (lane == 0) atomicMax(&s_p, p);
        if (lane == 0 && !(theta[0] == a.params.data[0])) s_lengthscales = 2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int P = max(4, (min(s_p, 4096) + 1) & ~1);
        plan->lo = a.rb1 > a.rb0 ? INT_MAX - plan->lo_bits : 0;
        plan->hi = a.rb1 > a.rb0 ? plan->hi_bits : 0;
        plan->checksum = plan->checksum & ((1ll << 61) - 1);
        plan->P = (plan->bad == 0 && s_lengthscales == 1 && P <= NODE_OP_MAX) ? P : 0;
        plan->max_blocks = plan->width;
    }
}

struct NodeOpArgs {
    Batch batch;
    int64_t n, R, rb0, rb1;
    const float *x;
    int64_t xs;
    View<const float> params;
    const int *start, *end;
    const NodePlan *plan;
    const float *centre;
    float *lambda;  // [R][P][128]
    float *G;       // [rb1 - rb0][max_blocks][P (column node)][P (row node)]
    int P, max_blocks;
};

// Whether points, parameters or band differ in any bit from the copies an operator was laid out from.  (4 million
// points and 64 components: 5 us.)
struct NodeChangedArgs {
    Batch batch;
    int64_t n, R;
    const float *x;
    int64_t xs;
    View<const float> params;
    const int *start, *end;
    int64_t ss, es;
    const float *own_x, *own_params;
    const int *own_start, *own_end;
    int *changed;
};
__global__ void __launch_bounds__(256) node_changed_kernel(const NodeChangedArgs a) {
    const int64_t first = blockIdx.x * 256LL + threadIdx.x, step = gridDim.x * 256LL;
    const auto bits = [](float v) { return __float_as_uint(v); };
    bool differs = false;
    for (int64_t i = first; i < a.n; i += step) differs |= bits(a.x[i * a.xs]) != bits(a.own_x[i]);
    for (int64_t r = first; r < a.R; r += step) differs |= a.start[r * a.ss] != a.own_start[r] || a.end[r * a.es] != a.own_end[r];
    constexpr int P = 3;  // parameters of a spectral component
    for (int64_t i = first; i < a.batch.count * P; i += step)
        differs |= bits(batch_ptr(a.params, decompose(a.batch, i / P))[(i % P) * a.params.s0]) != bits(a.own_params[i]);
    if (differs) *a.changed = 1;
}

// Lagrange matrix of every block: thread = row.
__global__ void __launch_bounds__(128) node_lambda_kernel(const NodeOpArgs a) {
    __shared__ float delta[NODE_OP_MAX], weight[NODE_OP_MAX];
    const int t = threadIdx.x, P = a.P;
    const float h = __int_as_float(a.plan->max_h_bits), inv_h = 1.0f / h;
    if (t < P) delta[t] = node_offset(h, t, P);
    __syncthreads();
    if (t < P) weight[t] = node_weight(delta, h, t, P);
    __syncthreads();
    for (int64_t v = blockIdx.x; v < a.R; v += gridDim.x) {
        const int64_t row = v * KM_BLOCK_SIZE + t;
        float *out = a.lambda + v * P * KM_BLOCK_SIZE + t;
        if (row >= a.n) {
            for (int q = 0; q < P; q++) out[q * KM_BLOCK_SIZE] = 0.0f;
            continue;
        }
        const float d = a.x[row * a.xs] - a.centre[v];
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
            out[q * KM_BLOCK_SIZE] = hit >= 0 ? (q == hit ? 1.0f : 0.0f) : __fdividef(weight[q], e) * inv;
        }
    }
}

// G: a warp per (row block, GB_PAIRS column blocks).  A lane owns row node p = lane mod 16 (or 32) and 8
// column nodes at a time of each pair of blocks; the halves of a warp take alternate groups of 8 where 16 lanes
// hold all rows.  Components are the outer loop: the phase factors of the nodes are the same for
// all pairs and lie in shared memory, all that changes from pair to pair is the phase of the centres'
// distance (reduced in fp64), so a component costs 4 FMAs per pair to rotate the row's factors and 2 per
// entry; the envelope, one for all components, multiplies the finished sum.
constexpr int GB_PAIRS = 6;
constexpr int GB_COMPS = 32;  // components per chunk

__global__ void __launch_bounds__(128) node_matrix_kernel(const NodeOpArgs a) {
    using Fn = KernelFn<KM_KERNEL_SPECTRAL>;
    __shared__ float delta[NODE_OP_MAX + 8];
    __shared__ __align__(16) float2 node_phase[GB_COMPS][NODE_OP_MAX + 8];  // cos, sin of W delta
    __shared__ float2 pair_phase[4][GB_PAIRS][GB_COMPS];
    __shared__ float scales[GB_COMPS];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, P = a.P;
    const float h = __int_as_float(a.plan->max_h_bits);
    if (t < NODE_OP_MAX + 8) delta[t] = t < P ? node_offset(h, t, P) : 0.0f;
    const int64_t groups = (a.max_blocks + GB_PAIRS - 1) / GB_PAIRS;
    const int64_t item = blockIdx.x * 4LL + warp;
    const bool live = item < (a.rb1 - a.rb0) * groups;
    const int64_t r = a.rb0 + (live ? item / groups : 0);
    const int s = a.start[r], e = a.end[r];
    const int c_lo = s < e ? s / KM_BLOCK_SIZE : 0;
    const int blocks = s < e ? (int)((min((int64_t)e, a.n) + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE) - c_lo : 0;
    const int first = (int)(item % groups) * GB_PAIRS, pairs = live ? max(0, min(GB_PAIRS, blocks - first)) : 0;
    __syncthreads();
    const int width = P <= 16 ? 16 : 32, p = min(lane % width, P - 1);
    const float dp = delta[p], centre = a.centre[r];
    float D[GB_PAIRS];
#pragma unroll
    for (int i = 0; i < GB_PAIRS; i++) D[i] = i < pairs ? centre - a.centre[c_lo + first + i] : 0.0f;

    const int q_step = 8 * (32 / width);
    for (int round = 0; round * q_step < P; round++) {
        const int q0 = round * q_step + (lane / width) * 8;  // (may lie past P in one half: computed, not stored)
        const int qs = min(q0, NODE_OP_MAX);
        float acc[GB_PAIRS][8];
#pragma unroll
        for (int i = 0; i < GB_PAIRS; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
        for (int64_t b0 = 0; b0 < a.batch.count; b0 += GB_COMPS) {
            const int comps = (int)min((int64_t)GB_COMPS, a.batch.count - b0);
            __syncthreads();
            for (int i = t; i < comps * P; i += 128) {
                const int b = i / P, q = i % P;
                Fn fn;
                fn.init(batch_ptr(a.params, decompose(a.batch, b0 + b)), a.params.s0);
                float c, sn;
                sincospif(fn.phase_half_turns() * delta[q], &sn, &c);
                node_phase[b][q] = make_float2(c, sn);
                if (q == 0) scales[b] = fn.scale;
            }
            if (lane < comps) {
                Fn fn;
                fn.init(batch_ptr(a.params, decompose(a.batch, b0 + lane)), a.params.s0);
#pragma unroll
                for (int i = 0; i < GB_PAIRS; i++) {
                    const double turns = (double)fn.phase_half_turns() * (double)D[i];
                    float c, sn;
                    sincospif((float)(turns - 2.0 * rint(0.5 * turns)), &sn, &c);
                    pair_phase[warp][i][lane] = make_float2(c, sn);
                }
            }
            __syncthreads();
            for (int b = 0; b < comps; b++) {
                const float scale = scales[b];
                const float2 row_phase = node_phase[b][p];
                float2 col[8];
#pragma unroll
                for (int j = 0; j < 8; j++) col[j] = node_phase[b][qs + j];
#pragma unroll
                for (int i = 0; i < GB_PAIRS; i++) {
                    if (i >= pairs) break;
                    const float2 ph = pair_phase[warp][i][b];
                    const float rc = scale * (ph.x * row_phase.x - ph.y * row_phase.y), rs = scale * (ph.y * row_phase.x + ph.x * row_phase.y);
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[i][j] = fmaf(rc, col[j].x, fmaf(rs, col[j].y, acc[i][j]));
                }
            }
        }
        if (lane % width < P) {
            const float ell = a.params.data[0], c0 = -(0.5f / (ell * ell)) * KM_LOG2E_F;
#pragma unroll
            for (int i = 0; i < GB_PAIRS; i++) {
                if (i >= pairs) break;
                float *out = a.G + ((r - a.rb0) * a.max_blocks + first + i) * P * P + p;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (q0 + j >= P) break;
                    const float tau = (D[i] + dp) - delta[q0 + j];
                    out[(q0 + j) * P] = acc[i][j] * exp2f(c0 * tau * tau);
                }
            }
        }
    }
}

struct NodeVectorArgs {
    int64_t n, k, kq;
    int P;
    int64_t blk0, blk1;   // row blocks
    const float *lambda;  // [R][P][128]
    float *v;             // (n, k): the vector; updated first (v = r + beta v) where r is not null
    const float *r;
    float *nodes;         // [R][P][kq]
    // beta and the bookkeeping of an update (as cg_update_p_kernel)
    CgTotals totals;
    const float *rs_in;
    float *rs_out, *history, *coeff_out;
    const float *ynorm;
    float tiny;
    int vec;
};

// [v = r + beta v on whole blocks, and] nodes = Lambda^T v.  One CTA per row block: thread = row for the
// update, whose result stays in shared memory for the second part; there a warp adds up its own 32
// rows -- a lane owns 4 nodes x 4 columns of every 1st, 2nd, .. 32nd of them, however many lanes that takes to
// fill the warp --, and the warps' sums are added in order.
template <int KC>
__global__ void __launch_bounds__(128) node_compress_kernel(const NodeVectorArgs g) {
    constexpr int KC4 = KC < 4 ? 4 : KC, VS = KC4 + 4;
    __shared__ __align__(16) float vs[KM_BLOCK_SIZE * VS];
    __shared__ float ls[NODE_OP_MAX * (KM_BLOCK_SIZE + 1)];
    __shared__ __align__(16) float part[4][4][32][4];
    __shared__ float beta_s[KC];
    __shared__ double total_s[KC];
    constexpr int LS = KM_BLOCK_SIZE + 1;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, P = g.P;
    const int64_t k = g.k, blk = g.blk0 + blockIdx.x, row = blk * KM_BLOCK_SIZE + t;
    const bool any = blk < g.blk1;  // (an update with no blocks keeps the history all the same)
    if (!any) grid_wait();
    for (int c0 = 0; c0 < g.kq; c0 += KC4) {
        float v[KC], rv[KC];
#pragma unroll
        for (int c = 0; c < KC; c++) v[c] = rv[c] = 0.0f;
        if (any) {
            if (c0 == 0) {
                const float *lambda = g.lambda + blk * P * KM_BLOCK_SIZE + t;
                for (int q = 0; q < P; q++) cp_async4(ls + q * LS + t, lambda + q * KM_BLOCK_SIZE);
                cp_async_commit();
                grid_wait();  // (the Lagrange matrices were there before)
            }
            if (row < g.n) {
                cg_load_row<KC>(g.v + row * k, c0, (int)k, g.vec, v);
                if (g.r != nullptr) cg_load_row<KC>(g.r + row * k, c0, (int)k, g.vec, rv);
            }
        }
        if (g.r != nullptr) {
            cg_totals<KC>(g.totals, k, c0, total_s);
            if (t < KC && c0 + t < k) {
                const int c = c0 + t;
                const float rs_new = (float)total_s[t];
                beta_s[t] = rs_new / fmaxf(g.rs_in[c], g.tiny);
                if (blockIdx.x == 0) {
                    if (g.coeff_out != nullptr) g.coeff_out[c] = beta_s[t];
                    g.rs_out[c] = rs_new;
                    if (g.history != nullptr) g.history[c] = sqrtf(rs_new) / g.ynorm[c];
                }
            }
            __syncthreads();
            if (row < g.n && any) {
#pragma unroll
                for (int c = 0; c < KC; c++) v[c] = fmaf(c0 + c < k ? beta_s[c] : 0.0f, v[c], rv[c]);
                cg_store_row<KC>(g.v + row * k, c0, (int)k, g.vec, v);
            }
        }
        if (!any) continue;
        if constexpr (KC >= 4) {
#pragma unroll
            for (int c = 0; c < KC; c += 4) *reinterpret_cast<float4 *>(vs + t * VS + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        } else {
            *reinterpret_cast<float4 *>(vs + t * VS) = make_float4(v[0], KC > 1 ? v[KC - 1] : 0.0f, 0.0f, 0.0f);
        }
        cp_async_wait<0>();
        __syncthreads();
        const int groups = (int)min((int64_t)KC4, g.kq - c0) / 4, quads = (P + 3) / 4, units = quads * groups;  // <= 32
        const int span = units <= 4 ? 4 : (units <= 8 ? 8 : (units <= 16 ? 16 : 32)), unit = lane & (span - 1), step = 32 / span;
        const bool mine = unit < units;
        const int q = mine ? (unit % quads) * 4 : 0, c = mine ? (unit / quads) * 4 : 0;
        f32x2 acc[4][2] = {};
        const float *l[4];
#pragma unroll
        for (int j = 0; j < 4; j++) l[j] = ls + min(q + j, P - 1) * LS + warp * 32;
#pragma unroll 4
        for (int i = lane / span; i < 32; i += step) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(vs + (warp * 32 + i) * VS + c);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const f32x2 f = splat2(l[j][i]);
                acc[j][0] = fma2(f, w.x, acc[j][0]), acc[j][1] = fma2(f, w.y, acc[j][1]);
            }
        }
        for (int o = span; o < 32; o <<= 1) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                acc[j][0] = add2(acc[j][0], __shfl_xor_sync(0xffffffffu, acc[j][0], o));
                acc[j][1] = add2(acc[j][1], __shfl_xor_sync(0xffffffffu, acc[j][1], o));
            }
        }
        if (lane < span) {
#pragma unroll
            for (int j = 0; j < 4; j++) *reinterpret_cast<ulonglong2 *>(part[warp][j][lane]) = make_ulonglong2(acc[j][0], acc[j][1]);
        }
        __syncthreads();
        if (lane < span && mine && q + warp < P) {
            float4 o = *reinterpret_cast<const float4 *>(part[0][warp][lane]);
#pragma unroll
            for (int w = 1; w < 4; w++) {
                const float4 x = *reinterpret_cast<const float4 *>(part[w][warp][lane]);
                o.x += x.x, o.y += x.y, o.z += x.z, o.w += x.w;
            }
            *reinterpret_cast<float4 *>(g.nodes + (blk * P + q + warp) * g.kq + c0 + c) = o;
        }
    }
}

struct NodeProductArgs {
    int64_t n, k, kq, rb0, rb1;
    int P, max_blocks;
    int chunk;           // column nodes staged at a time, a multiple of 16
    const int *start, *end;
    const float *lambda, *G, *nodes;
    float *out;          // row rb0 * 128 of the window first
    const float *p;      // not null: out = K v + sigma2 p, and partials of p . out
    float sigma2;
    float *block_partials;
    int vec;
};

// K v of one row block per CTA.  Everything a block needs is contiguous -- its part of G, the nodes of
// its band, its Lagrange matrix -- and is fetched at once into shared memory, several CTAs per SM
// overlapping each other's fetches.  Lanes own two row nodes, 8 (16 beyond 16 nodes) lanes a column node; the sums
// over column nodes end in shared memory, and a thread forms two rows x half of the columns of
// Lambda times them.  Inner products are those of cg_q_dots to the bit (rows of a warp in a shuffle
// tree, then the four warps).
template <int KC4>
__global__ void __launch_bounds__(128) node_product_kernel(const NodeProductArgs g) {
    constexpr int KC2 = KC4 / 2, HC = KC4 / 2;  // pairs of columns; columns of a thread in the second part
    extern __shared__ __align__(16) float smem[];
    __shared__ float warp_part[4][32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, P = g.P;
    const int64_t k = g.k, r = g.rb0 + blockIdx.x;
    float *ls = smem;                       // [P][128]
    float *gs = ls + P * KM_BLOCK_SIZE;     // [chunk][P]; later the warps' sums [4][P][KC4]
    float *qs = gs + max(g.chunk * P, 4 * P * KC4);  // [chunk][KC4]
    const int s = g.start[r], e = g.end[r];
    const int64_t c_lo = s < e ? s / KM_BLOCK_SIZE : 0;
    const int count = s < e ? max(0, (int)((min((int64_t)e, g.n) + KM_BLOCK_SIZE - 1) / KM_BLOCK_SIZE - c_lo)) * P : 0;
    const float *G = g.G + (int64_t)blockIdx.x * g.max_blocks * P * P;
    const float *lambda = g.lambda + r * P * KM_BLOCK_SIZE;
    for (int i = t; i < P * (KM_BLOCK_SIZE / 4); i += 128) cp_async16(ls + i * 4, lambda + i * 4);
    // second part: rows (t & 63) and that + 64, columns of half t >> 6
    const int row_in = t & 63, half = t >> 6;
    const int64_t row0 = r * KM_BLOCK_SIZE + row_in;

    const int width = P <= 16 ? 8 : 16, pair = min(lane & (width - 1), P / 2 - 1), slices = 128 / width, slice = t / width;
    for (int c0 = 0; c0 < g.kq; c0 += KC4) {
        const int valid = (int)min((int64_t)KC4, g.kq - c0);  // a multiple of 4
        const float *nodes = g.nodes + c_lo * P * g.kq + c0;
        f32x2 acc[2][KC2];
#pragma unroll
        for (int c = 0; c < KC2; c++) acc[0][c] = acc[1][c] = 0ull;
        float w[2][HC];
        for (int j0 = 0; j0 < count; j0 += g.chunk) {
            const int here = min(g.chunk, count - j0);
            if (j0 > 0 || c0 > 0) __syncthreads();
            for (int i = t; i < here * P / 4; i += 128) cp_async16(gs + i * 4, G + (int64_t)j0 * P + i * 4);
            if (j0 == 0 && c0 == 0) grid_wait();  // (the matrix was there before)
            if (valid == KC4 && g.kq == KC4) {
                for (int i = t; i < here * (KC4 / 4); i += 128) cp_async16(qs + i * 4, nodes + (int64_t)j0 * KC4 + i * 4);
            } else {
                for (int i = t; i < here * (KC4 / 4); i += 128) {
                    const int j = i / (KC4 / 4), c = (i % (KC4 / 4)) * 4;
                    if (c < valid)
                        cp_async16(qs + j * KC4 + c, nodes + (int64_t)(j0 + j) * g.kq + c);
                    else
                        *reinterpret_cast<float4 *>(qs + j * KC4 + c) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
            }
            cp_async_commit();
            if (j0 == 0 && g.p != nullptr) {  // on the way with the rest
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if (row0 + 64 * i < g.n) cg_load_row<HC>(g.p + (row0 + 64 * i) * k, c0 + half * HC, (int)k, g.vec && HC >= 4, w[i]);
            }
            cp_async_wait<0>();
            __syncthreads();
#pragma unroll 2
            for (int j = slice; j < here; j += slices) {
                const float2 m = *reinterpret_cast<const float2 *>(gs + j * P + 2 * pair);
                const f32x2 m0 = splat2(m.x), m1 = splat2(m.y);
#pragma unroll
                for (int c4 = 0; c4 < KC4 / 4; c4++) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(qs + j * KC4 + c4 * 4);
                    acc[0][2 * c4] = fma2(m0, v.x, acc[0][2 * c4]), acc[0][2 * c4 + 1] = fma2(m0, v.y, acc[0][2 * c4 + 1]);
                    acc[1][2 * c4] = fma2(m1, v.x, acc[1][2 * c4]), acc[1][2 * c4 + 1] = fma2(m1, v.y, acc[1][2 * c4 + 1]);
                }
            }
        }
        if (count == 0) {
            if (c0 == 0) grid_wait();
            cp_async_commit();
            cp_async_wait<0>();
            if (g.p != nullptr)
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if (row0 + 64 * i < g.n) cg_load_row<HC>(g.p + (row0 + 64 * i) * k, c0 + half * HC, (int)k, g.vec && HC >= 4, w[i]);
        }
        for (int o = width; o < 32; o <<= 1) {
#pragma unroll
            for (int c = 0; c < KC2; c++) {
                acc[0][c] = add2(acc[0][c], __shfl_xor_sync(0xffffffffu, acc[0][c], o));
                acc[1][c] = add2(acc[1][c], __shfl_xor_sync(0xffffffffu, acc[1][c], o));
            }
        }
        __syncthreads();  // every warp is done with gs
        if (lane < P / 2) {
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int c4 = 0; c4 < KC4 / 4; c4++)
                    *reinterpret_cast<ulonglong2 *>(gs + (warp * P + 2 * lane + i) * KC4 + c4 * 4) = make_ulonglong2(acc[i][2 * c4], acc[i][2 * c4 + 1]);
        }
        __syncthreads();
        for (int i = t; i < P * KC4; i += 128) gs[i] = (gs[i] + gs[P * KC4 + i]) + (gs[2 * P * KC4 + i] + gs[3 * P * KC4 + i]);
        __syncthreads();
        float u[2][HC];
#pragma unroll
        for (int c = 0; c < HC; c++) u[0][c] = u[1][c] = 0.0f;
#pragma unroll 2
        for (int q = 0; q < P; q++) {
            const float l0 = ls[q * KM_BLOCK_SIZE + row_in], l1 = ls[q * KM_BLOCK_SIZE + row_in + 64];
            const float *sums = gs + q * KC4 + half * HC;
#pragma unroll
            for (int c = 0; c < HC; c += 2) {
                const float2 v = *reinterpret_cast<const float2 *>(sums + c);
                u[0][c] = fmaf(l0, v.x, u[0][c]), u[0][c + 1] = fmaf(l0, v.y, u[0][c + 1]);
                u[1][c] = fmaf(l1, v.x, u[1][c]), u[1][c + 1] = fmaf(l1, v.y, u[1][c + 1]);
            }
        }
        float dot[2][HC];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int64_t row = row0 + 64 * i;
#pragma unroll
            for (int c = 0; c < HC; c++) dot[i][c] = 0.0f;
            if (row < g.n) {
                if (g.p != nullptr) {
#pragma unroll
                    for (int c = 0; c < HC; c++) {
                        u[i][c] = fmaf(g.sigma2, w[i][c], u[i][c]);
                        dot[i][c] = w[i][c] * u[i][c];
                    }
                }
                cg_store_row<HC>(g.out + (row - g.rb0 * KM_BLOCK_SIZE) * k, c0 + half * HC, (int)k, g.vec && HC >= 4, u[i]);
            }
        }
        if (g.p != nullptr) {
            // rows 32 w .. 32 w + 31 of the block are those of one warp and one i: w = (warp & 1) + 2 i
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int c = 0; c < HC; c++) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) dot[i][c] += __shfl_xor_sync(0xffffffffu, dot[i][c], o);
                    if (lane == 0) warp_part[(warp & 1) + 2 * i][half * HC + c] = dot[i][c];
                }
            __syncthreads();
            if (t < KC4 && c0 + t < k)
                g.block_partials[(int64_t)blockIdx.x * k + c0 + t] = (warp_part[0][t] + warp_part[1][t]) + (warp_part[2][t] + warp_part[3][t]);
        }
    }
}

template <typename F>
static int node_dispatch_kc(int64_t k, F f) {
    if (k <= 1) return f(std::integral_constant<int, 1>());
    if (k <= 2) return f(std::integral_constant<int, 2>());
    if (k <= 4) return f(std::integral_constant<int, 4>());
    if (k <= 8) return f(std::integral_constant<int, 8>());
    return f(std::integral_constant<int, 16>());
}

static int node_compress(NodeVectorArgs g, cudaStream_t s) {
    g.kq = ceil_div(g.k, 4) * 4;
    g.tiny = 1.17549435e-38f;
    g.vec = g.k % 4 == 0 && (uintptr_t)g.v % 16 == 0 && (uintptr_t)g.r % 16 == 0;
    if (g.blk1 <= g.blk0 && g.r == nullptr) return KM_OK;
    // (an update always runs one CTA: it keeps the residual history)
    const unsigned ctas = (unsigned)std::max<int64_t>(1, g.blk1 - g.blk0);
    return node_dispatch_kc(g.k, [&](auto kc) {
        return launch_chained("node compression launch", node_compress_kernel<decltype(kc)::value>, ctas, 128, 0, s, g);
    });
}

}  // namespace km

extern "C" int km_node_operator_plan_f32(const km_batch *batch, int64_t n, const float *x, int64_t x_stride,
                                         const km_view *params, const int32_t *start, const int32_t *end, int64_t row_block_begin,
                                         int64_t row_block_count, float *centre, void *plan, void *stream) {
    using namespace km;
    KM_REQUIRE((x == nullptr) == (params == nullptr) && (x == nullptr || batch), KM_ERR_INVALID_ARGUMENT,
               "km_node_operator_plan_f32: bad arguments");
    NodePlanArgs a = {};
    if (x != nullptr) {
        const int rc = make_batch(batch, &a.batch);
        if (rc != KM_OK) return rc;
        KM_REQUIRE(a.batch.count >= 1 && params->data && centre, KM_ERR_INVALID_ARGUMENT, "km_node_operator_plan_f32: bad arguments");
        a.params = make_view<const float>(params, a.batch);
    }
    const int64_t R = ceil_div(n, KM_BLOCK_SIZE);
    KM_REQUIRE(n >= 1 && n <= 0x7fffffffLL - 256 && row_block_begin >= 0 && row_block_count >= 0 &&
                   row_block_begin + row_block_count <= R,
               KM_ERR_INVALID_ARGUMENT, "km_node_operator_plan_f32: bad sizes");
    KM_REQUIRE(start && end && plan && (uintptr_t)plan % 8 == 0, KM_ERR_INVALID_ARGUMENT, "km_node_operator_plan_f32: null pointer");
    a.n = n, a.R = R, a.rb0 = row_block_begin, a.rb1 = row_block_begin + row_block_count;
    a.x = x, a.xs = x_stride, a.start = start, a.end = end;
    a.centre = centre, a.plan = static_cast<NodePlan *>(plan);
    static_assert(sizeof(NodePlan) <= KM_NODE_PLAN_BYTES, "plan size");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const cudaError_t err = cudaMemsetAsync(plan, 0, sizeof(NodePlan), s);
    if (err != cudaSuccess) return cuda_fail(err, "km_node_operator_plan_f32");
    const unsigned ctas = (unsigned)std::min<int64_t>(ceil_div(R, 8), 148 * 4);
    node_plan_kernel<<<ctas, 256, 0, s>>>(a);
    KM_CHECK_LAUNCH("km_node_operator_plan_f32 launch");
    return KM_OK;
}

extern "C" int km_node_operator_build_f32(const km_batch *batch, int64_t n, const float *x, int64_t x_stride,
                                          const km_view *params, const int32_t *start, const int32_t *end, int64_t row_block_begin,
                                          int64_t row_block_count, const float *centre, const void *plan, int64_t nodes,
                                          int64_t max_blocks, float *lambda, float *matrix, void *stream) {
    using namespace km;
    KM_REQUIRE(batch && params, KM_ERR_INVALID_ARGUMENT, "km_node_operator_build_f32: bad arguments");
    NodeOpArgs a;
    const int rc = make_batch(batch, &a.batch);
    if (rc != KM_OK) return rc;
    const int64_t R = ceil_div(n, KM_BLOCK_SIZE);
    KM_REQUIRE(n >= 1 && n <= 0x7fffffffLL - 256 && a.batch.count >= 1 && row_block_begin >= 0 && row_block_count >= 0 &&
                   row_block_begin + row_block_count <= R && nodes >= 4 && nodes <= NODE_OP_MAX && nodes % 2 == 0 && max_blocks >= 0 &&
                   max_blocks <= R,
               KM_ERR_INVALID_ARGUMENT, "km_node_operator_build_f32: bad sizes");
    KM_REQUIRE(x && params->data && start && end && centre && plan && lambda && (matrix || row_block_count * max_blocks == 0),
               KM_ERR_INVALID_ARGUMENT, "km_node_operator_build_f32: null pointer");
    a.n = n, a.R = R, a.rb0 = row_block_begin, a.rb1 = row_block_begin + row_block_count;
    a.x = x, a.xs = x_stride, a.params = make_view<const float>(params, a.batch), a.start = start, a.end = end;
    a.plan = static_cast<const NodePlan *>(plan), a.centre = centre, a.lambda = lambda, a.G = matrix;
    a.P = (int)nodes, a.max_blocks = (int)max_blocks;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    node_lambda_kernel<<<(unsigned)std::min<int64_t>(R, 148 * 16), 128, 0, s>>>(a);
    KM_CHECK_LAUNCH("km_node_operator_build_f32 launch");
    const int64_t items = row_block_count * ceil_div(max_blocks, GB_PAIRS);
    if (items == 0) return KM_OK;
    KM_REQUIRE(items <= 0x7fffffffLL, KM_ERR_UNSUPPORTED, "km_node_operator_build_f32: too many blocks");
    node_matrix_kernel<<<(unsigned)ceil_div(items, 4), 128, 0, s>>>(a);
    KM_CHECK_LAUNCH("km_node_operator_build_f32 launch");
    return KM_OK;
}

extern "C" int km_node_operator_changed(const km_batch *batch, int64_t n, const float *x, int64_t x_stride, const km_view *params,
                                        const km_view *start, const km_view *end, const float *own_x, const float *own_params,
                                        const int32_t *own_start, const int32_t *own_end, int32_t *changed, void *stream) {
    using namespace km;
    KM_REQUIRE(batch && params && start && end, KM_ERR_INVALID_ARGUMENT, "km_node_operator_changed: bad arguments");
    NodeChangedArgs a = {};
    const int rc = make_batch(batch, &a.batch);
    if (rc != KM_OK) return rc;
    KM_REQUIRE(n >= 1 && n <= 0x7fffffffLL - 256 && x && params->data && start->data && end->data && own_x && own_params && own_start &&
                   own_end && changed,
               KM_ERR_INVALID_ARGUMENT, "km_node_operator_changed: bad arguments");
    a.n = n, a.R = ceil_div(n, KM_BLOCK_SIZE), a.x = x, a.xs = x_stride, a.params = make_view<const float>(params, a.batch);
    a.start = static_cast<const int *>(start->data), a.ss = start->stride[0];
    a.end = static_cast<const int *>(end->data), a.es = end->stride[0];
    a.own_x = own_x, a.own_params = own_params, a.own_start = own_start, a.own_end = own_end, a.changed = changed;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const cudaError_t err = cudaMemsetAsync(changed, 0, sizeof(int32_t), s);
    if (err != cudaSuccess) return cuda_fail(err, "km_node_operator_changed");
    node_changed_kernel<<<(unsigned)std::min<int64_t>(ceil_div(n, 256), 148 * 8), 256, 0, s>>>(a);
    KM_CHECK_LAUNCH("km_node_operator_changed launch");
    return KM_OK;
}

extern "C" int km_node_compress_f32(int64_t k, int64_t n, int64_t nodes_per_block, const float *lambda, const float *v, float *nodes,
                                    int64_t block_begin, int64_t block_end, void *stream) {
    using namespace km;
    KM_REQUIRE(k >= 1 && k <= KM_NODE_MAX_COLUMNS && n >= 1 && nodes_per_block >= 4 && nodes_per_block <= NODE_OP_MAX && block_begin >= 0 && block_end >= block_begin &&
                   block_end <= ceil_div(n, KM_BLOCK_SIZE) && lambda && v && nodes,
               KM_ERR_INVALID_ARGUMENT, "km_node_compress_f32: bad arguments");
    NodeVectorArgs g{};
    g.n = n, g.k = k, g.P = (int)nodes_per_block, g.blk0 = block_begin, g.blk1 = block_end, g.lambda = lambda;
    g.v = const_cast<float *>(v), g.nodes = nodes;
    return node_compress(g, static_cast<cudaStream_t>(stream));
}

extern "C" int km_node_update_p_f32(int64_t k, int64_t n, int64_t nodes_per_block, const float *lambda, float *p, const float *r,
                                    float *nodes, int64_t block_begin, int64_t block_end, const void *rr_seg_sums,
                                    int64_t seg_rank_stride_bytes, int32_t seg_ranks, int32_t seg_slots, const float *rs_old,
                                    float *rs_new, const float *ynorm, float *history_row, float *beta_row, void *stream) {
    using namespace km;
    KM_REQUIRE(k >= 1 && k <= KM_NODE_MAX_COLUMNS && n >= 1 && nodes_per_block >= 4 && nodes_per_block <= NODE_OP_MAX && block_begin >= 0 && block_end >= block_begin &&
                   block_end <= ceil_div(n, KM_BLOCK_SIZE) && lambda && p && r && nodes && rr_seg_sums && rs_old && rs_new &&
                   rs_old != rs_new && (history_row == nullptr || ynorm) && seg_ranks >= 1 && seg_slots >= 0 && seg_rank_stride_bytes % 8 == 0,
               KM_ERR_INVALID_ARGUMENT, "km_node_update_p_f32: bad arguments");
    NodeVectorArgs g{};
    g.n = n, g.k = k, g.P = (int)nodes_per_block, g.blk0 = block_begin, g.blk1 = block_end, g.lambda = lambda;
    g.v = p, g.r = r, g.nodes = nodes;
    g.totals = {static_cast<const unsigned char *>(rr_seg_sums), seg_rank_stride_bytes, seg_ranks, seg_slots};
    g.rs_in = rs_old, g.rs_out = rs_new, g.ynorm = ynorm, g.history = history_row, g.coeff_out = beta_row;
    return node_compress(g, static_cast<cudaStream_t>(stream));
}

extern "C" int km_node_product_f32(int64_t k, int64_t n, int64_t nodes_per_block, int64_t max_blocks, const int32_t *start,
                                   const int32_t *end, const float *lambda, const float *matrix, const float *nodes,
                                   int64_t row_block_begin, int64_t row_block_count, float *out, const float *p, float sigma2,
                                   float *block_partials, void *stream) {
    using namespace km;
    KM_REQUIRE(k >= 1 && k <= KM_NODE_MAX_COLUMNS && n >= 1 && nodes_per_block >= 4 && nodes_per_block <= NODE_OP_MAX && row_block_begin >= 0 && row_block_count >= 0 &&
                   row_block_begin + row_block_count <= ceil_div(n, KM_BLOCK_SIZE) && row_block_count <= 0x7fffffffLL && start && end &&
                   lambda && nodes && out && (matrix || max_blocks == 0) && (p == nullptr || block_partials),
               KM_ERR_INVALID_ARGUMENT, "km_node_product_f32: bad arguments");
    if (row_block_count == 0) return KM_OK;
    NodeProductArgs g{};
    g.n = n, g.k = k, g.kq = ceil_div(k, 4) * 4, g.rb0 = row_block_begin, g.rb1 = row_block_begin + row_block_count;
    g.P = (int)nodes_per_block, g.max_blocks = (int)max_blocks, g.start = start, g.end = end, g.lambda = lambda, g.G = matrix;
    g.nodes = nodes, g.out = out, g.p = p, g.sigma2 = sigma2, g.block_partials = block_partials;
    g.vec = k % 4 == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)p % 16 == 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const auto launch = [&](auto cols) {
        constexpr int KC4 = decltype(cols)::value;
        // 32 KB of matrix and operand at a time: four CTAs per SM with the Lagrange matrices
        const int P = g.P;
        g.chunk = std::max(16, (int)std::min<int64_t>(8192 / (P + KC4), max_blocks * P) / 16 * 16);
        const size_t smem = (size_t)(P * KM_BLOCK_SIZE + std::max(g.chunk * P, 4 * P * KC4) + g.chunk * KC4) * sizeof(float);
        auto kernel = node_product_kernel<KC4>;
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
        if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(node product)");
        return launch_chained("km_node_product_f32 launch", kernel, (unsigned)row_block_count, 128, smem, s, g);
    };
    if (k <= 4) return launch(std::integral_constant<int, 4>());
    if (k <= 8) return launch(std::integral_constant<int, 8>());
    return launch(std::integral_constant<int, 16>());
}
