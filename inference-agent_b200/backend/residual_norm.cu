// Residual sum with norms before and after it: the sum of a product's slices, of routed rows and of the part's own input, the norm of that
// result, the residual add, and the norm the next part reads x through, as f32 rows or as the bf16 operand of its products. One CTA per
// row, which stays in registers throughout.
#include "residual_norm.h"

#include <cuda_bf16.h>

#include "../csrc/ingot_internal.cuh"

namespace {

template <int kKeep>
struct Row {
    float4 v[kKeep];
};

// Sum over the block, the warps' parts in order. red: a float per warp (of kMaxWarps, 16-byte aligned) that no other exchange of the kernel
// uses. Four parts per load: one at a time in a loop over blockDim, 16 warps took about 500 cycles at every sum.
template <int kMaxWarps>
__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.f;
    const int warps = blockDim.x >> 5;
#pragma unroll
    for (int w = 0; w < kMaxWarps; w += 4) {
        if (w >= warps) break;
        const float4 r = *reinterpret_cast<const float4*>(red + w);
        t += r.x;
        if (w + 1 < warps) t += r.y;
        if (w + 2 < warps) t += r.z;
        if (w + 3 < warps) t += r.w;
    }
    return t;
}

// (mean, 1 / deviation) of the first n_mean values of the row the block holds, the deviation around the mean in a second pass over the
// registers; the mean is 0 for norms that do not centre.
template <int kKeep, int kMaxWarps>
__device__ __forceinline__ float2 moments(const Row<kKeep>& r, int n_mean, bool centred, float inv_n, float eps, float* red) {
    float mean = 0.f, sq = 0.f;
    if (centred) {
        float sum = 0.f;  // the padding holds zeros
#pragma unroll
        for (int k = 0; k < kKeep; k++) sum += (r.v[k].x + r.v[k].y) + (r.v[k].z + r.v[k].w);
        mean = block_sum<kMaxWarps>(sum, red) * inv_n;
    }
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        const int left = n_mean - int(threadIdx.x + k * blockDim.x) * 4;
        const float d[4] = {r.v[k].x - mean, r.v[k].y - mean, r.v[k].z - mean, r.v[k].w - mean};
        if (left >= 4) {
            sq = fmaf(d[0], d[0], sq); sq = fmaf(d[1], d[1], sq); sq = fmaf(d[2], d[2], sq); sq = fmaf(d[3], d[3], sq);
        } else {
#pragma unroll
            for (int e = 0; e < 3; e++)
                if (e < left) sq = fmaf(d[e], d[e], sq);
        }
    }
    return make_float2(mean, rsqrtf(fmaf(block_sum<kMaxWarps>(sq, red + kMaxWarps), inv_n, eps)));
}

// 1 / rms of the group each value the block holds belongs to, as `groups` equal runs of the first n_mean values. seg: a float per 128 values
// of the row that no other exchange of the kernel uses.
template <int kKeep, int kMaxWarps>
__device__ __forceinline__ void group_moments(const Row<kKeep>& r, Row<kKeep>& inv, int groups, int n_mean, float eps, float* red, float* seg) {
    const int size = n_mean / groups, step = blockDim.x * 4;
    const float inv_n = 1.0f / float(size);
    if (size % 128 == 0) {  // a warp's quads lie in one group
        float ss[kKeep];
#pragma unroll
        for (int k = 0; k < kKeep; k++) {
            const float4 v = r.v[k];
            ss[k] = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w)));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < kKeep; k++) ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], o);
        if ((threadIdx.x & 31) == 0) {
#pragma unroll
            for (int k = 0; k < kKeep; k++) seg[(threadIdx.x + k * blockDim.x) >> 5] = ss[k];
        }
        __syncthreads();
        const int per = size / 128;
        int have = -1;
        float f = 0.f;
#pragma unroll
        for (int k = 0; k < kKeep; k++) {
            const int g = min((int(threadIdx.x) * 4 + k * step) / size, groups - 1);
            if (g != have) {
                float t = 0.f;
#pragma unroll 8
                for (int i = 0; i < per; i++) t += seg[g * per + i];
                f = rsqrtf(fmaf(t, inv_n, eps));
                have = g;
            }
            inv.v[k] = make_float4(f, f, f, f);
        }
        return;
    }
    for (int g = 0; g < groups; g++) {
        const int first = g * size, last = first + size;
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < kKeep; k++) {
            const int i = threadIdx.x * 4 + k * step;
            const float d[4] = {r.v[k].x, r.v[k].y, r.v[k].z, r.v[k].w};
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (i + e >= first && i + e < last) ss = fmaf(d[e], d[e], ss);
        }
        const float f = rsqrtf(fmaf(block_sum<kMaxWarps>(ss, red + (g & 1) * kMaxWarps), inv_n, eps));
#pragma unroll
        for (int k = 0; k < kKeep; k++) {
            const int i = threadIdx.x * 4 + k * step;
            if (i >= first && i < last) inv.v[k].x = f;
            if (i + 1 >= first && i + 1 < last) inv.v[k].y = f;
            if (i + 2 >= first && i + 2 < last) inv.v[k].z = f;
            if (i + 3 >= first && i + 3 < last) inv.v[k].w = f;
        }
    }
}

// The part of a norm's weights that belongs to this thread's values, requested ahead of the moments.
template <int kKeep>
struct Weights {
    Row<kKeep> w, b;
    __device__ __forceinline__ void load(const ingot_norm& n, int len, int step) {
#pragma unroll
        for (int k = 0; k < kKeep; k++) {
            const int i = threadIdx.x * 4 + k * step;
            w.v[k] = n.w && i < len ? *reinterpret_cast<const float4*>(n.w + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            b.v[k] = n.b && i < len ? *reinterpret_cast<const float4*>(n.b + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ float4 apply(float4 v, float2 m, int k) const {
        return make_float4(fmaf((v.x - m.x) * m.y, w.v[k].x, b.v[k].x), fmaf((v.y - m.x) * m.y, w.v[k].y, b.v[k].y),
                           fmaf((v.z - m.x) * m.y, w.v[k].z, b.v[k].z), fmaf((v.w - m.x) * m.y, w.v[k].w, b.v[k].w));
    }
    __device__ __forceinline__ float4 scale(float4 v, float4 f, int k) const { return make_float4(v.x * f.x * w.v[k].x, v.y * f.y * w.v[k].y, v.z * f.z * w.v[k].z, v.w * f.w * w.v[k].w); }
};
__device__ __forceinline__ void add(float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }

template <int kKeep, int kThreads, int kBlocks, bool kGrouped, bool kConv = false>
__global__ void __launch_bounds__(kThreads, kBlocks) residual_norm_kernel(const ingot_residual_norm p, float inv_n) {
    constexpr int kWarps = (kThreads / 32 + 3) / 4 * 4;
    __shared__ __align__(16) float red[3][2 * kWarps];  // of the three norms
    __shared__ float seg[kGrouped ? 2 : 1][kGrouped ? kThreads * kKeep / 32 : 1];
    INGOT_PDL_TRIGGER();
    const int row = blockIdx.x, step = blockDim.x * 4;
    const bool sum = p.n_slices > 0 || p.top > 0 || p.self_gain;
    Weights<kKeep> w;  // weights do not depend on the kernel before
    w.load(sum && p.post.w ? p.post : p.next, p.n, step);
    // taps of the convolution and the inputs it looks back on: not the work of the kernel before either
    float4 cw[kConv ? kKeep : 1][4], back[kConv ? kKeep : 1][3];
    int slot = 0, pos0 = 0;
    if (kConv) {
        INGOT_PDL_WAIT();
        slot = p.slot[row];
        pos0 = p.pos0[row];
#pragma unroll
        for (int k = 0; k < (kConv ? kKeep : 1); k++) {
            const int i = threadIdx.x * 4 + k * step;
            float4 four[4];  // of one channel each
            if (p.taps == 4 && i < p.n) {
#pragma unroll
                for (int e = 0; e < 4; e++) four[e] = reinterpret_cast<const float4*>(p.conv)[i + e];
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool on = i < p.n && j < p.taps;
                if (on && p.taps == 4) {
                    const float* t = &four[0].x + j;
                    cw[k][j] = make_float4(t[0], t[4], t[8], t[12]);
                } else cw[k][j] = on ? make_float4(p.conv[i * p.taps + j], p.conv[(i + 1) * p.taps + j], p.conv[(i + 2) * p.taps + j], p.conv[(i + 3) * p.taps + j]) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (j < 3)
                    back[k][j] = on && j < p.taps - 1 && pos0 - (p.taps - 1) + j >= 0 ? *reinterpret_cast<const float4*>(p.conv_state + ((size_t)slot * (p.taps - 1) + j) * p.n + i)
                                                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    INGOT_PDL_WAIT();
    float* xr = p.x + (size_t)(p.rows ? p.rows[row] : row) * p.n;
    Row<kKeep> x;
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        const int i = threadIdx.x * 4 + k * step;
        x.v[k] = i < p.n ? *reinterpret_cast<const float4*>(xr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (sum) {
        Row<kKeep> y;
#pragma unroll
        for (int k = 0; k < kKeep; k++) y.v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        const size_t slice = (size_t)p.n_rows * p.n;
        auto take = [&](const float* from) {  // all of the thread's pieces of a row in flight together
#pragma unroll
            for (int k = 0; k < kKeep; k++) {
                const int i = threadIdx.x * 4 + k * step;
                if (i < p.n) add(y.v[k], *reinterpret_cast<const float4*>(from + i));
            }
        };
        for (int s = 0; s < p.n_slices; s++) take(p.product + s * slice + (size_t)row * p.n);
        if (p.gain) {
            const float gain = p.gain[row];
#pragma unroll
            for (int k = 0; k < kKeep; k++) { y.v[k].x *= gain; y.v[k].y *= gain; y.v[k].z *= gain; y.v[k].w *= gain; }
        }
        for (int t0 = 0; t0 < p.top; t0 += 4) {
            int r[4];
#pragma unroll
            for (int t = 0; t < 4; t++) r[t] = t0 + t < p.top ? p.row_of[(size_t)row * p.top + t0 + t] : -1;
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (r[t] >= 0) take(p.branch + (size_t)r[t] * p.n);
        }
        const float self = p.self_gain ? p.self_gain[row] : 0.f;
        if (self != 0.f) {  // block-uniform
            const float2 m = moments<kKeep, kWarps>(x, p.n_mean, p.self.b != nullptr, inv_n, p.eps, red[0]);
#pragma unroll
            for (int k = 0; k < kKeep; k++) {
                const int i = threadIdx.x * 4 + k * step;
                if (i >= p.n) continue;
                const float4 g = *reinterpret_cast<const float4*>(p.self.w + i);
                const float4 b = p.self.b ? *reinterpret_cast<const float4*>(p.self.b + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                y.v[k].x = fmaf(self, fmaf((x.v[k].x - m.x) * m.y, g.x, b.x), y.v[k].x);
                y.v[k].y = fmaf(self, fmaf((x.v[k].y - m.x) * m.y, g.y, b.y), y.v[k].y);
                y.v[k].z = fmaf(self, fmaf((x.v[k].z - m.x) * m.y, g.z, b.z), y.v[k].z);
                y.v[k].w = fmaf(self, fmaf((x.v[k].w - m.x) * m.y, g.w, b.w), y.v[k].w);
            }
        }
        if (kGrouped && p.post.w) {
            Row<kKeep> f = {};
            group_moments<kKeep, kWarps>(y, f, p.post.groups, p.n_mean, p.eps, red[1], seg[0]);
#pragma unroll
            for (int k = 0; k < kKeep; k++) y.v[k] = w.scale(y.v[k], f.v[k], k);
            if (p.next.w) w.load(p.next, p.n, step);
        } else if (p.post.w) {
            const float2 m = moments<kKeep, kWarps>(y, p.n_mean, p.post.b != nullptr, inv_n, p.eps, red[1]);
#pragma unroll
            for (int k = 0; k < kKeep; k++) y.v[k] = w.apply(y.v[k], m, k);
            if (p.next.w) w.load(p.next, p.n, step);
        }
#pragma unroll
        for (int k = 0; k < kKeep; k++) {
            const int i = threadIdx.x * 4 + k * step;
            add(x.v[k], y.v[k]);
            if (i < p.n && !p.shift) *reinterpret_cast<float4*>(xr + i) = x.v[k];
        }
    }
    if (p.shift) {
#pragma unroll
        for (int k = 0; k < kKeep; k++) {
            const int i = threadIdx.x * 4 + k * step;
            if (i >= p.n) continue;
            add(x.v[k], *reinterpret_cast<const float4*>(p.shift + i));
            *reinterpret_cast<float4*>(xr + i) = x.v[k];
        }
    }
    if (!p.next.w) return;
    float2 m = make_float2(0.f, 0.f);
    Row<kKeep> f = {};
    if (kGrouped) group_moments<kKeep, kWarps>(x, f, p.next.groups, p.n_mean, p.eps, red[2], seg[kGrouped ? 1 : 0]);
    else m = moments<kKeep, kWarps>(x, p.n_mean, p.next.b != nullptr, inv_n, p.eps, red[2]);
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        const int i = threadIdx.x * 4 + k * step;
        if (i >= p.n) continue;
        float4 v = kGrouped ? w.scale(x.v[k], f.v[k], k) : w.apply(x.v[k], m, k);
        if (kConv) {
            const int kk = kConv ? k : 0;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 u = j < p.taps - 1 ? back[kk][j < 3 ? j : 0] : j == p.taps - 1 ? v : make_float4(0.f, 0.f, 0.f, 0.f);
                a.x = fmaf(cw[kk][j].x, u.x, a.x);
                a.y = fmaf(cw[kk][j].y, u.y, a.y);
                a.z = fmaf(cw[kk][j].z, u.z, a.z);
                a.w = fmaf(cw[kk][j].w, u.w, a.w);
            }
#pragma unroll
            for (int j = 0; j < 3; j++)
                if (j < p.taps - 1)
                    *reinterpret_cast<float4*>(p.conv_state + ((size_t)slot * (p.taps - 1) + j) * p.n + i) = j + 1 < p.taps - 1 ? back[kk][j + 1 < 3 ? j + 1 : 0] : v;
            v = a;
        }
        const size_t at = (size_t)row * p.n + i;
        if (p.out) *reinterpret_cast<float4*>(p.out + at) = v;
        if (p.hi) {
            const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
            *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.hi) + at) = *reinterpret_cast<const uint2*>(h);
            if (p.lo) {
                const __nv_bfloat162 l[2] = {__floats2bfloat162_rn(v.x - __low2float(h[0]), v.y - __high2float(h[0])),
                                             __floats2bfloat162_rn(v.z - __low2float(h[1]), v.w - __high2float(h[1]))};
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.lo) + at) = *reinterpret_cast<const uint2*>(l);
            }
        }
    }
}

// The same for many whole rows (no padding, no convolution, no chosen rows): CTAs that stay, each with every gridDim-th row. Row by row, what
// bounded a prompt's residual was neither memory nor the number of rows in flight but what every row repeats and waits for: its 16 KB of
// each weight vector from L2, the loads of x and the product, exchanges that add up warp after warp in a loop of unknown length, a condition
// per access. Here the weights are in shared memory once per CTA (each thread keeps and reads its own quads, no barrier), the next row's x and
// product are requested before the current row's norms, and sizes are constants. Sums are taken in the same order as above.
// Inside a prompt's step (B200): 4096 rows of 4096, layer norms before and after, 72-76 -> 50-53 us (36 at the copy rate), before the last one only
// 53 -> 39; 1000 rows of 2048, norms in two groups, 12 -> 10 us.
enum { kRms = 0, kCentred = 1, kGroups = 2 };
template <int kThreads>
struct RowsSmem {
    static constexpr int kN = kThreads * 16;                                  // values of a row: four quads per thread
    static constexpr int kVectors = 4;                                        // post w, b, next w, b
    static constexpr int kBytes = kVectors * kN * 4;
};

template <int kThreads>
__device__ __forceinline__ float rows_sum(float v, float* red) {
    constexpr int kWarps = kThreads / 32;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; w += 4) {
        const float4 r = *reinterpret_cast<const float4*>(red + w);
        t += r.x; t += r.y; t += r.z; t += r.w;
    }
    return t;
}

// v <- norm of v as the block holds it. w: this thread's weights, kN floats before its biases. red: two exchanges that take turns.
template <int kThreads, int kMode>
__device__ __forceinline__ void rows_norm(Row<4>& v, const float* w, int groups, float inv_n, float eps, float (*red)[kThreads / 8], int& turn) {
    constexpr int kN = kThreads * 16;
    auto next_red = [&] { return red[turn ^= 1]; };
    if (kMode == kGroups) {
        float* const seg = next_red();  // a float per 128 values
        float ss[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float4 a = v.v[k];
            ss[k] = fmaf(a.x, a.x, fmaf(a.y, a.y, fmaf(a.z, a.z, a.w * a.w)));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 4; k++) ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], o);
        if ((threadIdx.x & 31) == 0) {
#pragma unroll
            for (int k = 0; k < 4; k++) seg[(threadIdx.x + k * kThreads) >> 5] = ss[k];
        }
        __syncthreads();
        const int per = kN / 128 / groups;  // runs of 128 values in a group
        const float inv = 1.0f / float(kN / groups);
        int have = -1;
        float f = 0.f;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int g = int((threadIdx.x + k * kThreads) >> 5) / per;
            if (g != have) {
                float t = 0.f;
#pragma unroll 8
                for (int i = 0; i < per; i++) t += seg[g * per + i];
                f = rsqrtf(fmaf(t, inv, eps));
                have = g;
            }
            const float4 a = *reinterpret_cast<const float4*>(w + k * kThreads * 4);
            v.v[k] = make_float4(v.v[k].x * f * a.x, v.v[k].y * f * a.y, v.v[k].z * f * a.z, v.v[k].w * f * a.w);
        }
        return;
    }
    float mean = 0.f, sq = 0.f;
    if (kMode == kCentred) {
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < 4; k++) sum += (v.v[k].x + v.v[k].y) + (v.v[k].z + v.v[k].w);
        mean = rows_sum<kThreads>(sum, next_red()) * inv_n;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float d[4] = {v.v[k].x - mean, v.v[k].y - mean, v.v[k].z - mean, v.v[k].w - mean};
        sq = fmaf(d[0], d[0], sq); sq = fmaf(d[1], d[1], sq); sq = fmaf(d[2], d[2], sq); sq = fmaf(d[3], d[3], sq);
    }
    const float f = rsqrtf(fmaf(rows_sum<kThreads>(sq, next_red()), inv_n, eps));
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float4 a = *reinterpret_cast<const float4*>(w + k * kThreads * 4);
        const float4 b = kMode == kCentred ? *reinterpret_cast<const float4*>(w + kN + k * kThreads * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        v.v[k] = make_float4(fmaf((v.v[k].x - mean) * f, a.x, b.x), fmaf((v.v[k].y - mean) * f, a.y, b.y), fmaf((v.v[k].z - mean) * f, a.z, b.z), fmaf((v.v[k].w - mean) * f, a.w, b.w));
    }
}

template <int kThreads, int kMode>
__global__ void __launch_bounds__(kThreads, 512 / kThreads) residual_rows_kernel(const ingot_residual_norm p, float inv_n) {
    constexpr int kN = kThreads * 16;
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(16) float red[2][kThreads / 8];
    INGOT_PDL_TRIGGER();
    const int at = threadIdx.x * 4;
    {  // weights do not depend on the kernel before
        const float* from[4] = {p.post.w, p.post.b, p.next.w, p.next.b};
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (from[i]) {
#pragma unroll
                for (int k = 0; k < 4; k++) *reinterpret_cast<float4*>(smem + i * kN + at + k * kThreads * 4) = *reinterpret_cast<const float4*>(from[i] + at + k * kThreads * 4);
            }
    }
    INGOT_PDL_WAIT();
    const size_t slice = (size_t)p.n_rows * kN;
    const bool sum = p.n_slices > 0 || p.top > 0;
    Row<4> nx, ny;  // of the row after the current one
    auto fetch = [&](int row) {
        const size_t base = (size_t)row * kN + at;
#pragma unroll
        for (int k = 0; k < 4; k++) nx.v[k] = *reinterpret_cast<const float4*>(p.x + base + k * kThreads * 4);
        if (p.n_slices > 0) {
#pragma unroll
            for (int k = 0; k < 4; k++) ny.v[k] = *reinterpret_cast<const float4*>(p.product + base + k * kThreads * 4);
        }
    };
    int row = blockIdx.x, turn = 0;
    if (row < p.n_rows) fetch(row);
    for (; row < p.n_rows; row += gridDim.x) {
        Row<4> x = nx, y = ny;
        const size_t base = (size_t)row * kN + at;
        if (row + (int)gridDim.x < p.n_rows) fetch(row + gridDim.x);
        if (sum) {
            auto take = [&](const float* from) {
#pragma unroll
                for (int k = 0; k < 4; k++) add(y.v[k], *reinterpret_cast<const float4*>(from + at + k * kThreads * 4));
            };
            if (p.n_slices == 0) y = Row<4>{};
            for (int s = 1; s < p.n_slices; s++) take(p.product + s * slice + (size_t)row * kN);
            if (p.gain) {
                const float gain = p.gain[row];
#pragma unroll
                for (int k = 0; k < 4; k++) { y.v[k].x *= gain; y.v[k].y *= gain; y.v[k].z *= gain; y.v[k].w *= gain; }
            }
            for (int t0 = 0; t0 < p.top; t0 += 4) {
                int r[4];
#pragma unroll
                for (int t = 0; t < 4; t++) r[t] = t0 + t < p.top ? p.row_of[(size_t)row * p.top + t0 + t] : -1;
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (r[t] >= 0) take(p.branch + (size_t)r[t] * kN);
            }
            if (p.post.w) rows_norm<kThreads, kMode>(y, smem + at, p.post.groups, inv_n, p.eps, red, turn);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                add(x.v[k], y.v[k]);
                *reinterpret_cast<float4*>(p.x + base + k * kThreads * 4) = x.v[k];
            }
        }
        if (!p.next.w) continue;
        rows_norm<kThreads, kMode>(x, smem + 2 * kN + at, p.next.groups, inv_n, p.eps, red, turn);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const size_t i = base + k * kThreads * 4;
            const float4 v = x.v[k];
            if (p.out) *reinterpret_cast<float4*>(p.out + i) = v;
            if (p.hi) {
                const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.hi) + i) = *reinterpret_cast<const uint2*>(h);
                if (p.lo) {
                    const __nv_bfloat162 l[2] = {__floats2bfloat162_rn(v.x - __low2float(h[0]), v.y - __high2float(h[0])),
                                                 __floats2bfloat162_rn(v.z - __low2float(h[1]), v.w - __high2float(h[1]))};
                    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.lo) + i) = *reinterpret_cast<const uint2*>(l);
                }
            }
        }
    }
}

// Which launches that is: more rows than a decoding step has, rows of 2048 or 4096 values without padding, norms of one kind.
template <int kThreads>
cudaError_t launch_rows(const ingot_residual_norm& r, int groups, cudaStream_t s) {
    int dev = 0, num_sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const bool centred = (r.post.w && r.post.b) || (r.next.w && r.next.b);  // a bias without a weight is no norm's
    auto kernel = groups > 1 ? residual_rows_kernel<kThreads, kGroups> : centred ? residual_rows_kernel<kThreads, kCentred> : residual_rows_kernel<kThreads, kRms>;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RowsSmem<kThreads>::kBytes)) != cudaSuccess) return e;
    const int slots = num_sms * (512 / kThreads), rounds = (r.n_rows + slots - 1) / slots;
    return ingot_launch_pdl(kernel, dim3((r.n_rows + rounds - 1) / rounds), dim3(kThreads), RowsSmem<kThreads>::kBytes, s, r, 1.0f / float(r.n_mean));
}
bool rows_take(const ingot_residual_norm& r, int groups) {
    const bool whole = r.n == r.n_mean && (r.n == 2048 || r.n == 4096) && r.n_rows > 64 && !r.rows && !r.conv && !r.shift && !r.self_gain;
    const bool alike = !r.post.w || !r.next.w || !r.post.b == !r.next.b;
    return whole && alike && (groups <= 1 || r.n / groups % 128 == 0);
}

}  // namespace

extern "C" cudaError_t ingot_residual_norm_run(const ingot_residual_norm* r, cudaStream_t s) {
    if (!r->x || r->n < 4 || r->n % 4 != 0 || r->n_mean < 1 || r->n_mean > r->n || r->n_rows < 1 || (r->n_slices > 0 && !r->product) ||
        (r->top > 0 && (!r->branch || !r->row_of)) || (r->self_gain && !r->self.w) || (r->next.w && !r->out && !r->hi))
        return cudaErrorInvalidValue;
    const int groups = r->post.w ? r->post.groups : r->next.w ? r->next.groups : 1;
    if (groups > 1 && (r->n_mean % groups != 0 || (r->post.w && r->next.w && r->post.groups != r->next.groups) || r->self_gain || r->post.b || r->next.b)) return cudaErrorInvalidValue;
    if (r->conv && (r->taps < 1 || r->taps > 4 || !r->slot || !r->pos0 || (r->taps > 1 && !r->conv_state) || !r->next.w || r->rows)) return cudaErrorInvalidValue;
    if (rows_take(*r, groups)) return r->n == 2048 ? launch_rows<128>(*r, groups, s) : launch_rows<256>(*r, groups, s);
    const int quads = r->n / 4;
    auto launch = [&](auto kernel, int threads) { return ingot_launch_pdl(kernel, dim3(r->n_rows), dim3(threads), 0, s, *r, 1.0f / float(r->n_mean)); };
    auto run = [&](auto plain, auto grouped, int threads) { return groups > 1 ? launch(grouped, threads) : launch(plain, threads); };
    auto warps = [&](int keep) { return (quads + 32 * keep - 1) / (32 * keep) * 32; };  // threads that hold a row of `keep` quads each
    if (r->conv) {
        if (quads <= 256) return run(residual_norm_kernel<1, 256, 2, false, true>, residual_norm_kernel<1, 256, 2, true, true>, warps(1));
        if (quads <= 1024) return run(residual_norm_kernel<1, 1024, 1, false, true>, residual_norm_kernel<1, 1024, 1, true, true>, warps(1));
        if (quads <= 2048) return run(residual_norm_kernel<4, 512, 1, false, true>, residual_norm_kernel<4, 512, 1, true, true>, warps(4));
        return run(residual_norm_kernel<8, 1024, 1, false, true>, residual_norm_kernel<8, 1024, 1, true, true>, 1024);
    }
    if (quads <= 256) return run(residual_norm_kernel<1, 256, 2, false>, residual_norm_kernel<1, 256, 2, true>, warps(1));
    if (quads <= 1024 && r->n_rows <= 64) return run(residual_norm_kernel<1, 1024, 1, false>, residual_norm_kernel<1, 1024, 1, true>, warps(1));  // a CTA per SM anyway
    if (quads <= 1024) return run(residual_norm_kernel<4, 256, 2, false>, residual_norm_kernel<4, 256, 2, true>, warps(4));
    if (quads <= 2048) return run(residual_norm_kernel<4, 512, 1, false>, residual_norm_kernel<4, 512, 1, true>, warps(4));
    if (quads <= 8192) return run(residual_norm_kernel<8, 1024, 1, false>, residual_norm_kernel<8, 1024, 1, true>, 1024);
    return cudaErrorInvalidValue;
}
