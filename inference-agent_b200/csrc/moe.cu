// Mixture of experts: routing, and the plain form of the experts' products (the tensor-core form is the grouped product of
// backend/linear_sm100.cu). No counterpart in the reference, whose feed-forwards are dense.
//
// A token's pairs are its `top` experts; pair p = token * top + k. The experts work on ROWS: the pairs sorted by expert, in token
// order within one, so that an expert's rows are a run [group_start[e], group_start[e + 1]) and the order is the same in every run.
#include "ingot_internal.cuh"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One warp per token: its `top` largest logits, larger first, the lower expert of equal ones; the weight is the logit's sigmoid.
// The k-th choice is the largest (logit, -expert) below the one before, so nothing has to be marked as taken.
__global__ void __launch_bounds__(128) moe_select_kernel(const float* logits, int ld, int n_tok, int n_expert, int top, int32_t* expert_of, float* weight_of) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= n_tok) return;
    const float* z = logits + (size_t)t * ld;
    float last = INFINITY;
    int last_e = -1;
    for (int k = 0; k < top; k++) {
        float best = -INFINITY;
        int best_e = n_expert;
        for (int e = lane; e < n_expert; e += 32) {
            float v = z[e];
            if (!(v == v)) v = -INFINITY;
            if ((v < last || (v == last && e > last_e)) && (v > best || best_e == n_expert)) { best = v; best_e = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float v = __shfl_xor_sync(0xffffffffu, best, o);
            const int e = __shfl_xor_sync(0xffffffffu, best_e, o);
            if (e < n_expert && (best_e == n_expert || v > best || (v == best && e < best_e))) { best = v; best_e = e; }
        }
        if (lane == 0) {
            expert_of[(size_t)t * top + k] = best_e;
            weight_of[(size_t)t * top + k] = 1.0f / (1.0f + expf(-best));
        }
        last = best;
        last_e = best_e;
    }
}

// Routers that choose by softmax score plus a correction, within the best groups of neighbouring outputs, and weigh by the score alone.
// One warp per token; the outputs behind the experts' are identity experts (the input itself) and, if asked for, one gate.
struct GroupedRouter {
    ingot_moe_router r;
    const float* logits;
    int ld, n_tok;
    int32_t* expert_of;
    float* weight_of;
    int32_t* row_of;
    float *self_gain, *shared_gain;
};
// The largest of get(0..n-1) below (last, -last_i) in the order of (value, lower index first); -1 if there is none.
template <class F>
__device__ __forceinline__ int warp_next_largest(int n, float last, int last_i, float* value, F&& get) {
    const int lane = threadIdx.x & 31;
    float best = -INFINITY;
    int best_i = n;
    for (int i = lane; i < n; i += 32) {
        const float v = get(i);
        if ((v < last || (v == last && i > last_i)) && (v > best || best_i == n)) { best = v; best_i = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v = __shfl_xor_sync(0xffffffffu, best, o);
        const int i = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (i < n && (best_i == n || v > best || (v == best && i < best_i))) { best = v; best_i = i; }
    }
    *value = best;
    return best_i < n ? best_i : -1;
}
constexpr int kRouterOutputs = 1024, kRouterWarps = 4;  // most outputs of a router (experts and identity experts)
__global__ void __launch_bounds__(kRouterWarps * 32) moe_select_grouped_kernel(const GroupedRouter p) {
    extern __shared__ float s_choice_all[];  // per warp: choice scores [n], group scores [count], weights [top]
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int t = blockIdx.x * kRouterWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= p.n_tok) return;
    const int n = p.r.n_expert + p.r.n_identity, top = p.r.top, count = p.r.groups, per = n / count;
    float* choice = s_choice_all + (threadIdx.x >> 5) * (n + count + top);
    float *group = choice + n, *weight = group + count;
    const float* z = p.logits + (size_t)t * p.ld;
    float most = -INFINITY;
    for (int e = lane; e < n; e += 32) most = fmaxf(most, z[e]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
    float sum = 0.f;
    for (int e = lane; e < n; e += 32) sum += expf(z[e] - most);
    const float inv = 1.0f / warp_sum(sum);
    for (int e = lane; e < n; e += 32) {
        const float c = expf(z[e] - most) * inv + (p.r.correction ? p.r.correction[e] : 0.f);
        choice[e] = c == c ? c : -INFINITY;
    }
    __syncwarp();
    if (p.r.keep < count) {
        for (int g = lane; g < count; g += 32) {
            float best = -INFINITY;
            for (int i = 0; i < per; i++) best = fmaxf(best, choice[g * per + i]);
            group[g] = best;
        }
        __syncwarp();
        // groups at and above the keep-th best are open
        float last = INFINITY;
        int last_g = -1;
        for (int k = 0; k < p.r.keep; k++) last_g = warp_next_largest(count, last, last_g, &last, [&](int g) { return group[g]; });
        __syncwarp();
        for (int e = lane; e < n; e += 32) {
            const int g = e / per;
            if (group[g] < last || (group[g] == last && g > last_g)) choice[e] = -INFINITY;
        }
        __syncwarp();
    }
    float last = INFINITY, total = 0.f;
    int last_e = -1;
    for (int k = 0; k < top; k++) {
        last_e = warp_next_largest(n, last, last_e, &last, [&](int e) { return choice[e]; });
        const float s = expf(z[last_e] - most) * inv;
        total += s;
        if (lane == 0) {
            weight[k] = s;
            p.expert_of[(size_t)t * top + k] = last_e;
        }
    }
    if (lane == 0) {
        const float f = p.r.scale / (total + 1e-20f);
        float self = 0.f;
        for (int k = 0; k < top; k++) {
            const float w = weight[k] * f;
            const size_t pair = (size_t)t * top + k;
            p.weight_of[pair] = w;
            if (p.expert_of[pair] >= p.r.n_expert) { self += w; p.row_of[pair] = -1; }
        }
        if (p.self_gain) p.self_gain[t] = self;
        if (p.shared_gain) p.shared_gain[t] = 1.0f / (1.0f + expf(-z[n]));
    }
}

// One CTA per expert: where its rows start (pairs of lower experts), then its pairs in order. A thread owns a run of pairs, so one scan
// over the threads' counts places them all.
// kTable: a pair's expert is looked up, expert_of being the table [token id][top], and all weights are the same.
constexpr int kSortThreads = 1024;
struct TableChoice {
    const int32_t* tokens;
    int top;
    float weight;
};
template <bool kTable>
__global__ void __launch_bounds__(kSortThreads) moe_sort_kernel(const int32_t* expert_of, const float* weight_of, int n_pairs, int n_expert, int32_t* group_start,
                                                                int32_t* row_of, int32_t* pair_of, float* row_weight, const TableChoice tc) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    auto expert = [&](int i) { return kTable ? expert_of[(size_t)tc.tokens[i / tc.top] * tc.top + i % tc.top] : expert_of[i]; };
    __shared__ int s_lower[kSortThreads / 32], s_mine[kSortThreads / 32];
    const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int run = ((n_pairs + kSortThreads - 1) / kSortThreads + 3) / 4 * 4, first = min((int)threadIdx.x * run, n_pairs), last = min(first + run, n_pairs);
    int lower = 0, mine = 0;
    for (int i = first; i < last; i += 4) {
        int v[4];
        if (!kTable && i + 4 <= last) {
            *reinterpret_cast<int4*>(v) = *reinterpret_cast<const int4*>(expert_of + i);
        } else {
            for (int k = 0; k < 4; k++) v[k] = i + k < last ? expert(i + k) : 0x7fffffff;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            lower += v[k] < e;
            mine += v[k] == e;
        }
    }
    int upto = mine;  // within the warp, then over the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lower += __shfl_xor_sync(0xffffffffu, lower, o);
    if (lane == 31) s_mine[warp] = upto;
    if (lane == 0) s_lower[warp] = lower;
    __syncthreads();
    int row = upto - mine;
    for (int w = 0; w < kSortThreads / 32; w++) {
        row += s_lower[w];
        if (w < warp) row += s_mine[w];
    }
    if (threadIdx.x == 0) {
        group_start[e] = row;
        if (e == n_expert - 1) {  // pairs of what lies behind the experts have no rows
            int all = row;
            for (int w = 0; w < kSortThreads / 32; w++) all += s_mine[w];
            group_start[n_expert] = all;
        }
    }
    if (mine == 0) return;
    for (int i = first; i < last; i++)
        if (expert(i) == e) {
            row_of[i] = row;
            pair_of[row] = i;
            row_weight[row] = kTable ? tc.weight : weight_of[i];
            row++;
        }
}

// Experts by table: every token id has its `top` experts.
__global__ void __launch_bounds__(256) moe_table_kernel(const int32_t* table, const int32_t* tokens, int n_pairs, int top, float weight, int32_t* expert_of, float* weight_of) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n_pairs) return;
    expert_of[i] = table[(size_t)tokens[i / top] * top + i % top];
    weight_of[i] = weight;
}

// bf16 planes of the rows: row r is its token's row, a CTA per row. n_rows_dev (may be null): how many of the launch's rows there are.
__global__ void __launch_bounds__(128) moe_gather_few_kernel(uint4* hi, uint4* lo, const uint4* src_hi, const uint4* src_lo, const int32_t* pair_of, int top, int n8,
                                                             const int32_t* n_rows_dev) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    if (n_rows_dev && (int)blockIdx.x >= *n_rows_dev) return;
    const size_t r = blockIdx.x, t = size_t(pair_of[r] / top);
    for (int i = threadIdx.x; i < n8; i += 128) {
        hi[r * n8 + i] = src_hi[t * n8 + i];
        if (lo) lo[r * n8 + i] = src_lo[t * n8 + i];
    }
}

// The same for many rows. n_rows_dev (may be null): how many of the n_rows there are. A warp per row, eight 16-byte pieces
// per lane in flight: 8000 rows of 2048 9.4 -> 7.4 us against a CTA per row (B200, inside a step).
__global__ void __launch_bounds__(256) moe_gather_kernel(uint4* hi, uint4* lo, const uint4* src_hi, const uint4* src_lo, const int32_t* pair_of, int top, int n8, int n_rows,
                                                         const int32_t* n_rows_dev) {
    constexpr int kPieces = 8;
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= n_rows || (n_rows_dev && r >= *n_rows_dev)) return;
    const size_t to = (size_t)r * n8, from = size_t(pair_of[r] / top) * n8;
    auto copy = [&](uint4* dst, const uint4* src) {
        for (int i = lane; i < n8; i += 32 * kPieces) {
            uint4 v[kPieces];
#pragma unroll
            for (int k = 0; k < kPieces; k++)
                if (i + 32 * k < n8) v[k] = src[from + i + 32 * k];
#pragma unroll
            for (int k = 0; k < kPieces; k++)
                if (i + 32 * k < n8) dst[to + i + 32 * k] = v[k];
        }
    };
    copy(hi, src_hi);
    if (lo) copy(lo, src_lo);
}

// Plain products: out[row][o] = act(row_weight * W_e[o] . x[source(row)]), f32 arithmetic on bf16 weights. A warp owns one output of
// up to kRowTile rows of one expert; grid.y counts row tiles, expert after expert.
// kGated: the matrices hold gate and up rows interleaved (gate_row), an output is row_weight * silu(gate) * up.
constexpr int kRowTile = 8;
__device__ __forceinline__ int gate_row(int o) { return o / 32 * 64 + o % 32; }  // the up row is 32 further on
__device__ __forceinline__ float silu(float v) { return v / (1.0f + expf(-v)); }
template <bool kGated>
__global__ void __launch_bounds__(256) moe_linear_kernel(float* out, const __nv_bfloat16* w, const float* x, int x_ld, int n_in, int n_out, int n_expert,
                                                         const int32_t* group_start, const int32_t* pair_of, int top, const float* row_weight, int act) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // which expert's which tile: 32 experts at a time
    int tile = blockIdx.y, e = -1, r0 = 0, r1 = 0;
    for (int e0 = 0; e0 < n_expert && e < 0; e0 += 32) {
        const int mine = e0 + lane;
        const int a = mine < n_expert ? group_start[mine] : 0, b = mine < n_expert ? group_start[mine + 1] : 0;
        const int n = (b - a + kRowTile - 1) / kRowTile;
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, tile < upto);
        if (hit) {
            const int src = __ffs(hit) - 1;
            const int local = tile - (__shfl_sync(0xffffffffu, upto, src) - __shfl_sync(0xffffffffu, n, src));
            e = e0 + src;
            r0 = __shfl_sync(0xffffffffu, a, src) + local * kRowTile;
            r1 = min(__shfl_sync(0xffffffffu, b, src), r0 + kRowTile);
        } else {
            tile -= __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    if (e < 0) return;
    const int o = blockIdx.x * 8 + warp;
    if (o >= n_out) return;
    const __nv_bfloat16* wr = w + (kGated ? (size_t)e * 2 * n_out + gate_row(o) : (size_t)e * n_out + o) * n_in;
    const float* xr[kRowTile];
#pragma unroll
    for (int i = 0; i < kRowTile; i++) {
        const int r = min(r0 + i, r1 - 1);
        xr[i] = x + (size_t)(pair_of ? pair_of[r] / top : r) * x_ld;
    }
    float acc[kRowTile], up[kRowTile];
#pragma unroll
    for (int i = 0; i < kRowTile; i++) acc[i] = up[i] = 0.f;
    auto widen = [](const uint4& raw, float (&wv)[8]) {
        const uint32_t u[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            wv[2 * i] = __uint_as_float(u[i] << 16);
            wv[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
        }
    };
    auto dot = [](const float (&wv)[8], const float4& a, const float4& b, float v) {
        v = fmaf(wv[0], a.x, v); v = fmaf(wv[1], a.y, v);
        v = fmaf(wv[2], a.z, v); v = fmaf(wv[3], a.w, v);
        v = fmaf(wv[4], b.x, v); v = fmaf(wv[5], b.y, v);
        v = fmaf(wv[6], b.z, v); return fmaf(wv[7], b.w, v);
    };
    for (int c = lane * 8; c < n_in; c += 256) {
        float wv[8], uv[8];
        widen(*reinterpret_cast<const uint4*>(wr + c), wv);
        if (kGated) widen(*reinterpret_cast<const uint4*>(wr + (size_t)32 * n_in + c), uv);
#pragma unroll
        for (int i = 0; i < kRowTile; i++) {
            if (r0 + i >= r1) break;
            const float4 a = *reinterpret_cast<const float4*>(xr[i] + c), b = *reinterpret_cast<const float4*>(xr[i] + c + 4);
            acc[i] = dot(wv, a, b, acc[i]);
            if (kGated) up[i] = dot(uv, a, b, up[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < kRowTile; i++) {
        if (r0 + i >= r1) break;
        float v = warp_sum(acc[i]);
        if (kGated) v = silu(v) * warp_sum(up[i]);
        if (lane == 0) {
            if (row_weight) v *= row_weight[r0 + i];
            if (act == INGOT_ACT_RELU2) v = v > 0.f ? v * v : 0.f;
            out[(size_t)(r0 + i) * n_out + o] = v;
        }
    }
}

// The same for the few rows of one token, bound by streaming the weights: a warp owns two outputs of one row and keeps eight 16-byte
// weight loads in flight while it multiplies the eight before; the row's x is read once for both. kGated: the two are the gate and the
// up row of one output.
constexpr int kGemvLoads = 4;
template <bool kGated>
__global__ void __launch_bounds__(256) moe_gemv_kernel(float* out, const __nv_bfloat16* w, const float* x, int x_ld, int n_in, int n_out, const int32_t* group_start,
                                                       int n_expert, const int32_t* pair_of, int top, const float* row_weight, int act) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.y;
    int e = 0;  // the expert whose run holds this row: runs start in ascending order
    for (int e0 = 0; e0 < n_expert; e0 += 32) {
        const bool past = e0 + lane < n_expert && group_start[e0 + lane + 1] <= row;
        e += __popc(__ballot_sync(0xffffffffu, past));
    }
    const int o = (blockIdx.x * 8 + warp) * (kGated ? 1 : 2);
    if (o >= n_out || e >= n_expert) return;
    const bool two = !kGated && o + 1 < n_out;
    const uint4* wa = reinterpret_cast<const uint4*>(w + (kGated ? (size_t)e * 2 * n_out + gate_row(o) : (size_t)e * n_out + o) * n_in);
    const uint4* wb = kGated ? wa + (size_t)32 * (n_in / 8) : two ? wa + n_in / 8 : wa;
    const float* xr = x + (size_t)(pair_of ? pair_of[row] / top : row) * x_ld;
    const int n8 = n_in / 8;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 a[2][kGemvLoads], b[2][kGemvLoads];
    auto request = [&](uint4 (&u)[kGemvLoads], uint4 (&v)[kGemvLoads], int c0) {
#pragma unroll
        for (int k = 0; k < kGemvLoads; k++) {
            const int c = c0 + k * 32 + lane;
            u[k] = c < n8 ? __ldcs(wa + c) : zero;
            v[k] = c < n8 ? __ldcs(wb + c) : zero;
        }
    };
    float acc_a = 0.f, acc_b = 0.f;
    auto dot = [](const uint4& raw, const float4& p, const float4& q, float acc) {
        acc = fmaf(__uint_as_float(raw.x << 16), p.x, acc); acc = fmaf(__uint_as_float(raw.x & 0xffff0000u), p.y, acc);
        acc = fmaf(__uint_as_float(raw.y << 16), p.z, acc); acc = fmaf(__uint_as_float(raw.y & 0xffff0000u), p.w, acc);
        acc = fmaf(__uint_as_float(raw.z << 16), q.x, acc); acc = fmaf(__uint_as_float(raw.z & 0xffff0000u), q.y, acc);
        acc = fmaf(__uint_as_float(raw.w << 16), q.z, acc); return fmaf(__uint_as_float(raw.w & 0xffff0000u), q.w, acc);
    };
    auto consume = [&](const uint4 (&u)[kGemvLoads], const uint4 (&v)[kGemvLoads], int c0) {
#pragma unroll
        for (int k = 0; k < kGemvLoads; k++) {
            const int c = c0 + k * 32 + lane;
            if (c >= n8) break;
            const float4 p = *reinterpret_cast<const float4*>(xr + c * 8), q = *reinterpret_cast<const float4*>(xr + c * 8 + 4);
            acc_a = dot(u[k], p, q, acc_a);
            acc_b = dot(v[k], p, q, acc_b);
        }
    };
    constexpr int kStep = kGemvLoads * 32;
    request(a[0], b[0], 0);
    for (int c = 0; c < n8; c += 2 * kStep) {
        request(a[1], b[1], c + kStep);
        consume(a[0], b[0], c);
        request(a[0], b[0], c + 2 * kStep);
        consume(a[1], b[1], c + kStep);
    }
    acc_a = warp_sum(acc_a);
    acc_b = warp_sum(acc_b);
    if (lane == 0) {
        const float f = row_weight ? row_weight[row] : 1.0f;
        if (kGated) acc_a = silu(acc_a) * acc_b;
        acc_a *= f;
        acc_b *= f;
        if (act == INGOT_ACT_RELU2) {
            acc_a = acc_a > 0.f ? acc_a * acc_a : 0.f;
            acc_b = acc_b > 0.f ? acc_b * acc_b : 0.f;
        }
        out[(size_t)row * n_out + o] = acc_a;
        if (two) out[(size_t)row * n_out + o + 1] = acc_b;
    }
}

// x[t] += sum over the token's pairs of rows[row_of[pair]]; row_of null: rows[t]
__global__ void moe_add_kernel(float* x, const float* rows, const int32_t* row_of, int top, int n4) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    const size_t t = blockIdx.y;
    float4 v = reinterpret_cast<const float4*>(x)[t * n4 + i];
    for (int k = 0; k < top; k++) {
        const float4 a = reinterpret_cast<const float4*>(rows)[(row_of ? (size_t)row_of[t * top + k] : t) * n4 + i];
        v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
    }
    reinterpret_cast<float4*>(x)[t * n4 + i] = v;
}

}  // namespace

extern "C" {

int ingot_moe_route(const float* logits_dev, int ld, int n_tok, int n_expert, int top, int32_t* expert_of_dev, float* weight_of_dev, int32_t* group_start_dev,
                    int32_t* row_of_dev, int32_t* pair_of_dev, float* row_weight_dev, void* stream) {
    INGOT_REQUIRE(logits_dev && expert_of_dev && weight_of_dev && group_start_dev && row_of_dev && pair_of_dev && row_weight_dev, "ingot_moe_route: null argument");
    INGOT_REQUIRE(n_tok >= 1 && n_expert >= 1 && top >= 1 && top <= n_expert && ld >= n_expert && (long long)n_tok * top < (1ll << 30), "ingot_moe_route: bad sizes");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    INGOT_CUDA_TRY(ingot_launch_pdl(moe_select_kernel, dim3((n_tok + 3) / 4), dim3(128), 0, s, logits_dev, ld, n_tok, n_expert, top, expert_of_dev, weight_of_dev));
    INGOT_CUDA_TRY(ingot_launch_pdl(moe_sort_kernel<false>, dim3(n_expert), dim3(kSortThreads), 0, s, (const int32_t*)expert_of_dev, (const float*)weight_of_dev, n_tok * top, n_expert,
                                    group_start_dev, row_of_dev, pair_of_dev, row_weight_dev, TableChoice{}));
    return INGOT_OK;
}

int ingot_moe_route_table(const int32_t* table_dev, const int32_t* tokens_dev, int n_tok, int n_expert, int top, float weight, int32_t* expert_of_dev, float* weight_of_dev,
                          int32_t* group_start_dev, int32_t* row_of_dev, int32_t* pair_of_dev, float* row_weight_dev, void* stream) {
    INGOT_REQUIRE(table_dev && tokens_dev && expert_of_dev && weight_of_dev && group_start_dev && row_of_dev && pair_of_dev && row_weight_dev, "ingot_moe_route_table: null argument");
    INGOT_REQUIRE(n_tok >= 1 && n_expert >= 1 && top >= 1 && (long long)n_tok * top < (1ll << 30), "ingot_moe_route_table: bad sizes");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int pairs = n_tok * top;
    if (pairs <= 4096) {  // every expert's CTA looks all of them up
        INGOT_CUDA_TRY(ingot_launch_pdl(moe_sort_kernel<true>, dim3(n_expert), dim3(kSortThreads), 0, s, table_dev, (const float*)nullptr, pairs, n_expert, group_start_dev, row_of_dev,
                                        pair_of_dev, row_weight_dev, TableChoice{tokens_dev, top, weight}));
        return INGOT_OK;
    }
    INGOT_CUDA_TRY(ingot_launch_pdl(moe_table_kernel, dim3((pairs + 255) / 256), dim3(256), 0, s, table_dev, tokens_dev, pairs, top, weight, expert_of_dev, weight_of_dev));
    INGOT_CUDA_TRY(ingot_launch_pdl(moe_sort_kernel<false>, dim3(n_expert), dim3(kSortThreads), 0, s, (const int32_t*)expert_of_dev, (const float*)weight_of_dev, pairs, n_expert,
                                    group_start_dev, row_of_dev, pair_of_dev, row_weight_dev, TableChoice{}));
    return INGOT_OK;
}

int ingot_moe_route_grouped(const ingot_moe_router* router, const float* logits_dev, int ld, int n_tok, int32_t* expert_of_dev, float* weight_of_dev,
                            int32_t* group_start_dev, int32_t* row_of_dev, int32_t* pair_of_dev, float* row_weight_dev, float* self_gain_dev, float* shared_gain_dev,
                            void* stream) {
    INGOT_REQUIRE(router && logits_dev && expert_of_dev && weight_of_dev && group_start_dev && row_of_dev && pair_of_dev && row_weight_dev,
                  "ingot_moe_route_grouped: null argument");
    const ingot_moe_router& r = *router;
    const int n = r.n_expert + r.n_identity;
    INGOT_REQUIRE(n_tok >= 1 && r.n_expert >= 1 && r.n_identity >= 0 && r.groups >= 1 && n % r.groups == 0 && r.keep >= 1 && r.keep <= r.groups && r.top >= 1 &&
                      r.top <= n / r.groups * r.keep && ld >= n + (shared_gain_dev ? 1 : 0) && (long long)n_tok * r.top < (1ll << 30) &&
                      (r.n_identity == 0 || self_gain_dev), "ingot_moe_route_grouped: bad sizes");
    if (n > kRouterOutputs) {
        ingot_set_error("ingot_moe_route_grouped: at most " + std::to_string(kRouterOutputs) + " experts");
        return INGOT_ERR_UNSUPPORTED;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const GroupedRouter p = {r, logits_dev, ld, n_tok, expert_of_dev, weight_of_dev, row_of_dev, self_gain_dev, shared_gain_dev};
    const size_t smem = size_t(kRouterWarps) * (n + r.groups + r.top) * sizeof(float);
    INGOT_CUDA_TRY(ingot_launch_pdl(moe_select_grouped_kernel, dim3((n_tok + kRouterWarps - 1) / kRouterWarps), dim3(kRouterWarps * 32), smem, s, p));
    INGOT_CUDA_TRY(ingot_launch_pdl(moe_sort_kernel<false>, dim3(r.n_expert), dim3(kSortThreads), 0, s, (const int32_t*)expert_of_dev, (const float*)weight_of_dev, n_tok * r.top,
                                    r.n_expert, group_start_dev, row_of_dev, pair_of_dev, row_weight_dev, TableChoice{}));
    return INGOT_OK;
}

int ingot_moe_gather(void* hi_dev, void* lo_dev, const void* src_hi_dev, const void* src_lo_dev, const int32_t* pair_of_dev, int n_rows, const int32_t* n_rows_dev, int top,
                     int n, void* stream) {
    INGOT_REQUIRE(hi_dev && src_hi_dev && pair_of_dev && (!lo_dev || src_lo_dev), "ingot_moe_gather: null argument");
    INGOT_REQUIRE(n_rows >= 1 && top >= 1 && n >= 8 && n % 8 == 0, "ingot_moe_gather: bad sizes");
    // A row per CTA while that is at most four CTAs an SM: a row's pieces are then all requested together, by 128 threads. 32 rows of 4096 in two planes 3.1 us,
    // by a warp each 4.3; 512: 4.1 and 4.7; 1000 of one plane 4.0 and 3.7; 8000 of 2048 in two 22.3 and 19.1 (B200, calls replayed as a graph).
    if (n_rows <= 592) {
        INGOT_CUDA_TRY(ingot_launch_pdl(moe_gather_few_kernel, dim3(n_rows), dim3(128), 0, static_cast<cudaStream_t>(stream), static_cast<uint4*>(hi_dev), static_cast<uint4*>(lo_dev),
                                        static_cast<const uint4*>(src_hi_dev), static_cast<const uint4*>(src_lo_dev), pair_of_dev, top, n / 8, n_rows_dev));
        return INGOT_OK;
    }
    INGOT_CUDA_TRY(ingot_launch_pdl(moe_gather_kernel, dim3((n_rows + 7) / 8), dim3(256), 0, static_cast<cudaStream_t>(stream), static_cast<uint4*>(hi_dev), static_cast<uint4*>(lo_dev),
                                    static_cast<const uint4*>(src_hi_dev), static_cast<const uint4*>(src_lo_dev), pair_of_dev, top, n / 8, n_rows, n_rows_dev));
    return INGOT_OK;
}

int ingot_moe_linear(float* out_dev, const void* w_dev, const float* x_dev, int x_ld, int n_in, int n_out, int n_expert, int n_rows, const int32_t* group_start_dev,
                     const int32_t* pair_of_dev, int top, const float* row_weight_dev, int act, void* stream) {
    INGOT_REQUIRE(out_dev && w_dev && x_dev && group_start_dev, "ingot_moe_linear: null argument");
    INGOT_REQUIRE(n_in >= 8 && n_in % 8 == 0 && x_ld % 4 == 0 && n_out >= 1 && n_expert >= 1 && n_rows >= 1 && top >= 1, "ingot_moe_linear: bad sizes");
    const bool gated = act == INGOT_ACT_SILU_GATED;
    INGOT_REQUIRE(!gated || n_out % 32 == 0, "ingot_moe_linear: gated outputs come in runs of 32");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(w_dev);
    if (n_rows <= 2 * top) {  // one token (or two): a row per expert, as good as always
        auto kernel = gated ? moe_gemv_kernel<true> : moe_gemv_kernel<false>;
        const int per = gated ? 8 : 16;
        INGOT_CUDA_TRY(ingot_launch_pdl(kernel, dim3((n_out + per - 1) / per, n_rows), dim3(256), 0, s, out_dev, w, x_dev, x_ld, n_in, n_out, group_start_dev, n_expert, pair_of_dev,
                                        top, row_weight_dev, act));
        return INGOT_OK;
    }
    const int tiles = n_rows / kRowTile + (n_rows < n_expert ? n_rows : n_expert);  // at least as many as there can be
    INGOT_REQUIRE(tiles <= 65535, "ingot_moe_linear: too many rows");
    auto kernel = gated ? moe_linear_kernel<true> : moe_linear_kernel<false>;
    INGOT_CUDA_TRY(ingot_launch_pdl(kernel, dim3((n_out + 7) / 8, tiles), dim3(256), 0, s, out_dev, w, x_dev, x_ld, n_in, n_out, n_expert, group_start_dev, pair_of_dev, top,
                                    row_weight_dev, act));
    return INGOT_OK;
}

int ingot_moe_add(float* x_dev, const float* rows_dev, const int32_t* row_of_dev, int n_tok, int top, int n, void* stream) {
    INGOT_REQUIRE(x_dev && rows_dev, "ingot_moe_add: null argument");
    INGOT_REQUIRE(n_tok >= 1 && top >= 1 && (row_of_dev || top == 1) && n >= 4 && n % 4 == 0, "ingot_moe_add: bad sizes");
    INGOT_CUDA_TRY(ingot_launch_pdl(moe_add_kernel, dim3((n / 4 + 127) / 128, n_tok), dim3(128), 0, static_cast<cudaStream_t>(stream), x_dev, rows_dev, row_of_dev, top, n / 4));
    return INGOT_OK;
}

}  // extern "C"
