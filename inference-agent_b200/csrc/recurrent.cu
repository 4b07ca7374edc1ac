// Recurrent sequence mixers over a ragged batch: per-channel causal convolution, the selective scan (state-space models
// with input-dependent step size) and the real-gated linear recurrent unit. No counterpart in the reference, which only
// has attention layers.
//
// A step carries tokens of several sequences (ingot_step). Each sequence owns one slot of every layer's state; a sequence
// whose first token of the step is at position 0 starts from the zero state whatever its slot holds, so a slot needs no
// clearing when it is handed to the next sequence. All recurrences run in f32.
//
// Time parallelism. A recurrence S_t = a_t S_(t-1) + b_t is cut into time chunks (ingot_scan_plan, made on the host):
//   pass 1  every chunk runs from the zero state (a sequence's first chunk from its slot) and leaves its end state and the
//           total decay of the chunk - for the selective scan exp(A * sum dt), for the gated unit exp(sum log a), so only
//           one sum per channel is kept;
//   pass 2  one thread per state element walks a sequence's chunks in order and turns end states into start states;
//   pass 3  every chunk runs again from its start state and writes the outputs; the last chunk writes the slot.
// A sequence that is a single chunk (every decoded token) takes pass 3 alone, straight from and to its slot.
// One launch may do all three (the stream kernels), to the same bits: which launches a call takes is a matter of time alone (scan_routes.h).
//
// Decays. A slow channel multiplies its state by a = exp(x), x near 0, at every token, so an error of a that is always of
// the same sign adds up over the memory of the channel (the 2^x unit is good to about 2^-22). Where that matters - the gated
// unit, and the selective scan in its exact form - the state moves by S + S expm1(x), whose error is relative to 1 - a.
#include "recurrent_common.cuh"
#include "scan_routes.h"

namespace {

// ---- causal convolution -------------------------------------------------------------------------------------------
// out[t][c] = act(bias[c] + sum_j w[c][j] * in[t - (taps-1) + j][c]), in = raw + in_bias, zeros before position 0.
// state [slot][taps-1][channels]: the sequence's last taps-1 inputs, oldest first. A CTA owns 128 channels and one run
// of kConvRun tokens of one sequence; the run that starts at the sequence's first token reads the slot, computes, and
// afterwards writes it, so no other CTA touches the slot and a run is never shorter than the history it replaces.
constexpr int kConvRun = 16;
constexpr int kMaxTaps = 16, kMaxConvTaps4 = 4;  // taps of the four-channel form
struct ConvParams {
    ingot_step st;
    const float* raw;
    int raw_ld;
    const float *in_bias, *w, *bias;
    int taps, channels, silu;
    float* state;
    ActOut out;
};
template <int kTaps>  // 0: run-time tap count
__global__ void __launch_bounds__(128) causal_conv_kernel(const ConvParams p) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int taps = kTaps ? kTaps : p.taps;
    const int seq = blockIdx.z, c = blockIdx.x * 128 + threadIdx.x;
    const int len = p.st.len[seq], t0 = blockIdx.y * kConvRun;
    if (c >= p.channels || t0 >= len) return;
    const int pos0 = p.st.pos0[seq];
    const float* in = p.raw + (size_t)p.st.row_start[seq] * p.raw_ld + c;
    const size_t row0 = p.st.row_start[seq];
    float* slot = p.state + (size_t)p.st.slot[seq] * (taps - 1) * p.channels + c;
    const float ib = p.in_bias ? p.in_bias[c] : 0.f, b = p.bias ? p.bias[c] : 0.f;
    constexpr int kH = kTaps ? kTaps : kMaxTaps;
    float w[kH], h[kH];  // h: the last taps inputs, newest at taps-1
#pragma unroll
    for (int j = 0; j < kH; j++) w[j] = j < taps ? p.w[(size_t)c * taps + j] : 0.f;
    // input at position t of this step (t < 0: from the slot, or zero before the sequence's start)
    auto input = [&](int t) -> float {
        if (t >= 0) return in[(size_t)t * p.raw_ld] + ib;
        return pos0 + t >= 0 ? slot[(size_t)(taps - 1 + t) * p.channels] : 0.f;
    };
#pragma unroll
    for (int j = 0; j < kH; j++) h[j] = j < taps - 1 ? input(t0 - (taps - 1) + j) : 0.f;
    const int t_end = min(len, t0 + kConvRun);
    for (int t = t0; t < t_end; t++) {
        const float x = in[(size_t)t * p.raw_ld] + ib;
        float acc = b;
#pragma unroll
        for (int j = 0; j < kH; j++)
            if (j < taps - 1) acc = fmaf(w[j], h[j], acc);
#pragma unroll
        for (int j = 0; j < kH; j++)
            if (j == taps - 1) acc = fmaf(w[j], x, acc);
        p.out.store(row0 + t, c, p.silu == 0 ? acc : p.silu == 1 ? siluf(acc) : fast_silu(acc));
#pragma unroll
        for (int j = 0; j + 1 < kH; j++) h[j] = j < taps - 2 ? h[j + 1] : x;
    }
    if (t0 == 0) {
        // the slot's new contents: inputs len-(taps-1) .. len-1; the ones that are older than this step move down
        float n[kH];
#pragma unroll
        for (int j = 0; j < kH; j++) n[j] = j < taps - 1 ? input(len - (taps - 1) + j) : 0.f;
#pragma unroll
        for (int j = 0; j < kH; j++)
            if (j < taps - 1) slot[(size_t)j * p.channels] = n[j];
    }
}

// The same for 2 to 4 taps and four channels per thread (channels and row lengths multiples of 4), a run of kRun tokens whose inputs are all
// requested together. Bound by DRAM (large steps) or by the latency of one round trip (small ones). Against runs of 16 in four dependent rounds
// of loads (B200, inside a prompt's step): 1000 tokens x 2048 channels 12.8 -> 5.0 us, 2048 x 4096 25 -> 19.4, 2048 x 8192
// 43 -> 39.5. Runs of 4 read 1.75 times what they write from L2, but give a short step four times the CTAs; which run a launch takes is
// decided in ingot_causal_conv.
// kPacked: grid.y holds the runs of all sequences one after the other, instead of those of the longest one for every sequence (grid.z).
template <int kTaps, int kRun, bool kPacked>
__global__ void __launch_bounds__(128) causal_conv4_kernel(const ConvParams p) {
    static_assert(kRun >= kMaxConvTaps4 - 1, "a run replaces its history");
    INGOT_PDL_TRIGGER();
    const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
    const bool on = c < p.channels;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 ib = zero, b = zero;
    float w[4][kTaps];
    if (on) {  // weights do not depend on the kernel before
        if (p.in_bias) ib = *reinterpret_cast<const float4*>(p.in_bias + c);
        if (p.bias) b = *reinterpret_cast<const float4*>(p.bias + c);
        if (kTaps == 4 && reinterpret_cast<uintptr_t>(p.w) % 16 == 0) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float4 v = reinterpret_cast<const float4*>(p.w)[c + e];
                const float t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < kTaps; j++) w[e][j] = t[j];
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int j = 0; j < kTaps; j++) w[e][j] = p.w[(size_t)(c + e) * kTaps + j];
        }
    }
    INGOT_PDL_WAIT();
    int seq = blockIdx.z, run = blockIdx.y;
    if (kPacked) {  // every warp finds the sequence by the runs before it
        const int lane = threadIdx.x & 31;
        seq = -1;
        for (int s0 = 0; s0 < p.st.n_seq; s0 += 32) {
            const int own = s0 + lane < p.st.n_seq ? (p.st.len[s0 + lane] + kRun - 1) / kRun : 0;
            int upto = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const unsigned past = __ballot_sync(0xffffffffu, upto > run);
            if (past) {
                const int at = __ffs(past) - 1;
                seq = s0 + at;
                run -= __shfl_sync(0xffffffffu, upto - own, at);
                break;
            }
            run -= __shfl_sync(0xffffffffu, upto, 31);
        }
        if (seq < 0) return;
    }
    const int len = p.st.len[seq], t0 = run * kRun;
    if (!on || t0 >= len) return;
    const int pos0 = p.st.pos0[seq];
    const size_t row0 = p.st.row_start[seq];
    const float* in = p.raw + row0 * p.raw_ld + c;
    float* slot = p.state + (size_t)p.st.slot[seq] * (kTaps - 1) * p.channels + c;
    auto add = [](float4 a, float4 v) { return make_float4(a.x + v.x, a.y + v.y, a.z + v.z, a.w + v.w); };
    auto input = [&](int t) -> float4 {
        if (t >= 0) return add(*reinterpret_cast<const float4*>(in + (size_t)t * p.raw_ld), ib);
        return pos0 + t >= 0 ? *reinterpret_cast<const float4*>(slot + (size_t)(kTaps - 1 + t) * p.channels) : zero;
    };
    float4 h[kTaps - 1 + kRun];  // inputs t0 - (taps-1) .. t0 + run - 1
    if (t0 > 0 && t0 + kRun <= len) {  // no conditions between the loads
#pragma unroll
        for (int j = 0; j < kTaps - 1 + kRun; j++) h[j] = *reinterpret_cast<const float4*>(in + (size_t)(t0 - (kTaps - 1) + j) * p.raw_ld);
#pragma unroll
        for (int j = 0; j < kTaps - 1 + kRun; j++) h[j] = add(h[j], ib);
    } else {
#pragma unroll
        for (int j = 0; j < kTaps - 1 + kRun; j++) h[j] = t0 - (kTaps - 1) + j < len ? input(t0 - (kTaps - 1) + j) : zero;
    }
#pragma unroll
    for (int i = 0; i < kRun; i++) {
        if (t0 + i >= len) break;
        float4 a = b;
#pragma unroll
        for (int j = 0; j < kTaps; j++) {
            a.x = fmaf(w[0][j], h[i + j].x, a.x);
            a.y = fmaf(w[1][j], h[i + j].y, a.y);
            a.z = fmaf(w[2][j], h[i + j].z, a.z);
            a.w = fmaf(w[3][j], h[i + j].w, a.w);
        }
        if (p.silu == 1) a = make_float4(siluf(a.x), siluf(a.y), siluf(a.z), siluf(a.w));
        else if (p.silu == 2) a = make_float4(fast_silu(a.x), fast_silu(a.y), fast_silu(a.z), fast_silu(a.w));
        p.out.store4(row0 + t0 + i, c, a);
    }
    if (t0 == 0) {
        float4 n[kTaps - 1];
#pragma unroll
        for (int j = 0; j < kTaps - 1; j++) n[j] = input(len - (kTaps - 1) + j);
#pragma unroll
        for (int j = 0; j < kTaps - 1; j++) *reinterpret_cast<float4*>(slot + (size_t)j * p.channels) = n[j];
    }
}

// ---- selective scan -------------------------------------------------------------------------------------------------
// Per channel c and state n: S <- exp(dt A) S + dt x B, y = sum_n S C + D x, out = y * silu(z); dt = softplus(raw + bias).
// 4 or more lanes share two channels, each holding kS of their states in registers. A CTA of 128 threads owns 256 / lanes channels
// over one time chunk; inputs are staged 16 tokens at a time in shared memory, the next 16 requested (cp.async) while the
// current ones are computed.
constexpr int kScanTile = 16;
struct ScanParams {
    ingot_step st;
    const int32_t *chunk_seq, *chunk_t0, *chunk_len, *seq_chunk0;
    int n_chunks;
    const float* x; int x_ld;
    const float* dt; int dt_ld;
    const float* dt_bias;
    const float* bc; int bc_ld, b_off, c_off;
    const float* z; int z_ld;
    const float* a2;     // [inner][n_pad]: -exp(A_log) * log2(e), 0 in the padding
    const float* d;
    float* state;        // [slot][inner][n_pad]
    float* part;         // [chunk][inner][n_pad] end states, then start states
    float* part_sum;     // [chunk][inner] sum of dt
    int inner, n_pad, lanes_log2;
    ActOut out;
    bool whole;          // grid.y: sequences
};
// Pairs of f32 in one 64-bit register: two multiply-adds per instruction.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpair(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// kS consecutive floats of shared memory as pairs
template <int kS>
__device__ __forceinline__ void load_pairs(const float* p, f32x2 (&v)[kS / 2]) {
    if (kS % 4 == 0) {
#pragma unroll
        for (int i = 0; i < kS / 4; i++) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(p + 4 * i);
            v[2 * i] = q.x;
            v[2 * i + 1] = q.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kS / 2; i++) v[i] = *reinterpret_cast<const f32x2*>(p + 2 * i);
    }
}

// kLg: log2 of the lanes per pair of channels, or -1 for p.lanes_log2. A thread holds the same kS states of two neighbouring
// channels, so that every B and C value it fetches from shared memory is used twice.
template <int kS, bool kOutput, int kLg, bool kExact>
__global__ void __launch_bounds__(128) selective_scan_kernel(const ScanParams p) {
    extern __shared__ __align__(16) float smem[];
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int chunk = blockIdx.y;
    const bool whole = kOutput && p.whole;  // sequences as they are instead of chunks
    const int seq = whole ? chunk : p.chunk_seq[chunk], t0 = whole ? 0 : p.chunk_t0[chunk], len = whole ? p.st.len[seq] : p.chunk_len[chunk];
    const bool first = t0 == 0, last = t0 + len == p.st.len[seq];
    if ((!kOutput && last) || (whole && len < 1)) return;  // nothing follows a sequence's last chunk
    const int lg = kLg >= 0 ? kLg : p.lanes_log2;
    const int lanes = 1 << lg, n_ch = 256 >> lg;
    const int ch = threadIdx.x >> lg, part = threadIdx.x & (lanes - 1);
    const int c_base = blockIdx.x * n_ch, c = c_base + 2 * ch;
    const bool live = c < p.inner;  // the channel count is even
    const size_t row0 = (size_t)p.st.row_start[seq] + t0;
    const int np = p.n_pad;

    // [2 buffers][16 tokens]: x, dt, z [n_ch], B, C [np]; then dt * x of the current tile and y
    const int tile_floats = kScanTile * (3 * n_ch + 2 * np);
    float* const s_dtx = smem + 2 * tile_floats;
    float* const s_y = s_dtx + kScanTile * n_ch;
    const int ch4 = n_ch >> 2, np4 = np >> 2;

    auto stage = [&](int tile) {
        float* sx = smem + (tile & 1) * tile_floats;
        float* sdt = sx + kScanTile * n_ch;
        float* sz = sdt + kScanTile * n_ch;
        float* sb = sz + kScanTile * n_ch;
        float* sc = sb + kScanTile * np;
        const int t_base = tile * kScanTile;
        for (int i = threadIdx.x; i < kScanTile * ch4; i += 128) {
            const int t = i / ch4, q = (i - t * ch4) * 4;
            const bool on = t_base + t < len && c_base + q < p.inner;
            const size_t row = row0 + min(t_base + t, len - 1);
            const int cc = min(c_base + q, p.inner - 4);
            cp_async16(sx + t * n_ch + q, p.x + row * p.x_ld + cc, on);
            cp_async16(sdt + t * n_ch + q, p.dt + row * p.dt_ld + cc, on);
            if (kOutput) cp_async16(sz + t * n_ch + q, p.z + row * p.z_ld + cc, on);
        }
        for (int i = threadIdx.x; i < kScanTile * np4; i += 128) {
            const int t = i / np4, q = (i - t * np4) * 4;
            const bool on = t_base + t < len;
            const size_t row = row0 + min(t_base + t, len - 1);
            cp_async16(sb + t * np + q, p.bc + row * p.bc_ld + p.b_off + q, on);
            if (kOutput) cp_async16(sc + t * np + q, p.bc + row * p.bc_ld + p.c_off + q, on);
        }
        cp_async_commit();
    };

    const int n_tiles = (len + kScanTile - 1) / kScanTile;
    stage(0);

    f32x2 a[2][kS / 2], s[2][kS / 2];
    const size_t sidx = (size_t)(live ? c : 0) * np + part * kS;
    const size_t slot_base = (size_t)p.st.slot[seq] * p.inner * np;
    {
        // Start state: the slot for a sequence's first chunk (zero before position 0), else what pass 2 left. Pass 3 of a
        // multi-chunk sequence takes the first chunk's from there too: the last chunk's CTA may write the slot before this
        // CTA gets to read it.
        const float* from = nullptr;
        if (kOutput && !(first && last)) from = p.part + (size_t)chunk * p.inner * np + sidx;
        else if (first && p.st.pos0[seq] > 0) from = p.state + slot_base + sidx;
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
            for (int i = 0; i < kS / 2; i++) {
                a[e][i] = live ? *reinterpret_cast<const f32x2*>(p.a2 + sidx + e * np + 2 * i) : 0;
                s[e][i] = live && from ? *reinterpret_cast<const f32x2*>(from + e * np + 2 * i) : 0;
            }
    }
    const int my_q = (threadIdx.x % ch4) * 4;  // the four channels this thread prepares and writes (ch4 divides 128)
    const bool my_live = c_base + my_q < p.inner;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 my_bias = my_live ? *reinterpret_cast<const float4*>(p.dt_bias + c_base + my_q) : zero4;
    const float4 my_d = kOutput && my_live ? *reinterpret_cast<const float4*>(p.d + c_base + my_q) : zero4;
    float sum_dt[2] = {0.f, 0.f};

    for (int tile = 0; tile < n_tiles; tile++) {
        if (tile + 1 < n_tiles) { stage(tile + 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
        __syncthreads();
        float* sx = smem + (tile & 1) * tile_floats;
        float* sdt = sx + kScanTile * n_ch;
        const float* sz = sdt + kScanTile * n_ch;
        const float* sb = sz + kScanTile * n_ch;
        const float* sc = sb + kScanTile * np;
        const int n_t = min(kScanTile, len - tile * kScanTile);
        for (int i = threadIdx.x; i < n_t * ch4; i += 128) {
            const float4 raw = reinterpret_cast<const float4*>(sdt)[i], xv = reinterpret_cast<const float4*>(sx)[i];
            auto sp = [](float v) { return kExact ? softplusf(v) : fast_softplus(v); };
            const float4 dt = make_float4(sp(raw.x + my_bias.x), sp(raw.y + my_bias.y), sp(raw.z + my_bias.z), sp(raw.w + my_bias.w));
            reinterpret_cast<float4*>(sdt)[i] = dt;
            reinterpret_cast<float4*>(s_dtx)[i] = make_float4(dt.x * xv.x, dt.y * xv.y, dt.z * xv.z, dt.w * xv.w);
        }
        __syncthreads();
        auto token = [&](int t) {
            const float2 dt = *reinterpret_cast<const float2*>(sdt + t * n_ch + 2 * ch), dtx = *reinterpret_cast<const float2*>(s_dtx + t * n_ch + 2 * ch);
            f32x2 b[kS / 2], cc[kS / 2];
            load_pairs<kS>(sb + t * np + part * kS, b);
            if (kOutput) load_pairs<kS>(sc + t * np + part * kS, cc);
            float y[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float d = kExact ? (e ? dt.y : dt.x) * 0.69314718f : (e ? dt.y : dt.x);
                const f32x2 dt2 = pair(d, d), dtx2 = e ? pair(dtx.y, dtx.y) : pair(dtx.x, dtx.x);
                f32x2 y2 = 0;
#pragma unroll
                for (int i = 0; i < kS / 2; i++) {
                    const float2 x = unpair(mul2(dt2, a[e][i]));
                    const f32x2 in = mul2(dtx2, b[i]);
                    if (kExact) {
                        const float2 sv = unpair(s[e][i]), iv = unpair(in);
                        s[e][i] = pair(sv.x + fmaf(expm1f(x.x), sv.x, iv.x), sv.y + fmaf(expm1f(x.y), sv.y, iv.y));
                    } else {
                        s[e][i] = fma2(pair(ex2f(x.x), ex2f(x.y)), s[e][i], in);
                    }
                    if (kOutput) y2 = fma2(s[e][i], cc[i], y2);
                }
                const float2 yv = unpair(y2);
                y[e] = yv.x + yv.y;
            }
            if (kOutput) {
                // the first exchange halves the work: the upper lanes of a group go on with the second channel only
                const bool upper = part & (lanes >> 1);
                float v = upper ? y[1] : y[0];
                v += __shfl_xor_sync(0xffffffffu, upper ? y[0] : y[1], lanes >> 1);
                if (kLg == 2) v += __shfl_xor_sync(0xffffffffu, v, 1);
                else for (int o = lanes >> 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if ((part & ((lanes >> 1) - 1)) == 0) s_y[t * n_ch + 2 * ch + (upper ? 1 : 0)] = v;
            } else {
                sum_dt[0] += dt.x;
                sum_dt[1] += dt.y;
            }
        };
        if (n_t == kScanTile) {
#pragma unroll 4
            for (int t = 0; t < kScanTile; t++) token(t);
        } else {
            for (int t = 0; t < n_t; t++) token(t);
        }
        if (kOutput) {
            __syncthreads();
            if (my_live) {
                for (int i = threadIdx.x; i < n_t * ch4; i += 128) {
                    const size_t row = row0 + tile * kScanTile + i / ch4;
                    const float4 xv = reinterpret_cast<const float4*>(sx)[i], yv = reinterpret_cast<const float4*>(s_y)[i],
                                 zv = reinterpret_cast<const float4*>(sz)[i];
                    auto act = [](float v) { return kExact ? siluf(v) : fast_silu(v); };
                    p.out.store4(row, c_base + my_q, make_float4(fmaf(my_d.x, xv.x, yv.x) * act(zv.x), fmaf(my_d.y, xv.y, yv.y) * act(zv.y),
                                                                 fmaf(my_d.z, xv.z, yv.z) * act(zv.z), fmaf(my_d.w, xv.w, yv.w) * act(zv.w)));
                }
            }
        }
        __syncthreads();  // the tile's buffers are staged over two tiles from now, s_dtx / s_y in the next one
    }
    if (!live) return;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        if (!kOutput) {
#pragma unroll
            for (int i = 0; i < kS / 2; i++) *reinterpret_cast<f32x2*>(p.part + (size_t)chunk * p.inner * np + sidx + e * np + 2 * i) = s[e][i];
            if (part == 0) p.part_sum[(size_t)chunk * p.inner + c + e] = sum_dt[e];
        } else if (last) {
#pragma unroll
            for (int i = 0; i < kS / 2; i++) *reinterpret_cast<f32x2*>(p.state + slot_base + sidx + e * np + 2 * i) = s[e][i];
        }
    }
}

// ---- selective scan as a stream --------------------------------------------------------------------------------------
// The three passes in one, to the same bits: a CTA walks a sequence's chunks one after the other. The tile kernel above does its phases one after the other
// (stage, step sizes, tokens, gates) and waits between them, so a single chunk per sequence would leave the GPU idle (2048 tokens, 8192 channels: 433 us). Here one
// half of a CTA does nothing but the recurrence and the other everything around it. Four lanes share a channel, each with kS of its states; kNch channels per CTA.
//   helpers   request tiles of 16 tokens of a chunk three ahead (cp.async, a ring of kStreamSlots), turn dt into softplus(dt + bias) and dt x, and
//             write (y + D x) silu(z) of the tile before last
//   scanners  walk the tokens of the tile that is ready and leave y. Beside the state they keep what the chunk adds up to from zero, and its sum of dt:
//             the next chunk begins with what pass 2 makes of those
// Hand-over by named barriers: kBarReady + parity (helpers arrive, scanners wait), kBarDone + parity (the reverse).
// What bounds it: instruction issue and shared memory next to the 2^x. 64 channels of 16 states take 165 cycles a token; 80 are the 2^x of scan,
// softplus and gates at 16 per clock, about 85 the instructions, 110 the shared-memory cycles. Eight lanes a channel with half the states each fetch B and C
// twice as often (64 channels: 195 us below; 32: 59 us per 1000 tokens of 4096 channels, 55 with four), and sum y in another order than the tile kernel.
// Against the passes over chunks (B200, calls replayed as a graph): 2048 tokens x 8192 channels 228 -> 178 us, 300 x 8192 44 -> 29, 1000 x 4096 63 -> 56,
// 300 x 4096 32 -> 19.
constexpr int kStreamSlots = 6, kStreamHelpers = 256;
enum : int { kBarHelpers = 1, kBarReady = 2, kBarDone = 4 };  // + parity
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_wait(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
// floats of a ring slot: x, dt, z, dt x, y of n_ch channels, B and C of np states
__host__ __device__ constexpr int stream_slot_floats(int n_ch, int np) { return kScanTile * (5 * n_ch + 2 * np); }

// A channel's states lie in four lanes as in the tile kernel, so that its y is summed in the same order.
template <int kS, int kNch>
__global__ void __launch_bounds__(kNch * 4 + kStreamHelpers) selective_scan_stream_kernel(const ScanParams p) {
    extern __shared__ __align__(16) float smem[];
    struct Tile { int t, n; bool links; };  // first token and number of tokens (0: past the end); another chunk begins behind it
    __shared__ Tile s_tile[kStreamSlots];
    constexpr int kLanes = 4, kScanners = kNch * kLanes, kAll = kScanners + kStreamHelpers, kNp = kS * kLanes, kCh4 = kNch / 4, kNp4 = kNp / 4;
    constexpr int kSlot = stream_slot_floats(kNch, kNp), kDt = kScanTile * kNch, kZ = 2 * kDt, kDtx = 3 * kDt, kY = 4 * kDt, kB = 5 * kDt, kC = kB + kScanTile * kNp;
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int seq = gridDim.y - 1 - blockIdx.y, k0 = p.seq_chunk0[seq], k1 = p.seq_chunk0[seq + 1];  // the last first: steps hold their sequences in ascending order of tokens
    if (k0 == k1) return;
    const int c_base = blockIdx.x * kNch, seq_len = p.st.len[seq];
    const size_t row0 = (size_t)p.st.row_start[seq];

    if (threadIdx.x >= kScanners) {
        // ---------------- helpers ----------------
        const int tid = threadIdx.x - kScanners;
        // of the tile that is staged next; the length of the chunk after its own is requested a chunk ahead
        int chunk = k0, at = 0, left = min(p.chunk_len[k0], seq_len), next_len = k0 + 1 < k1 ? p.chunk_len[k0 + 1] : 0;
        auto next_chunk = [&] {
            while (left == 0 && chunk + 1 < k1) {
                left = min(next_len, seq_len - at);
                next_len = ++chunk + 1 < k1 ? p.chunk_len[chunk + 1] : 0;
            }
        };
        next_chunk();
        auto stage = [&](int tile) {
            const int n = min(kScanTile, left);
            if (tid == 0) s_tile[tile % kStreamSlots] = Tile{at, n, n == left && chunk + 1 < k1};
            if (n > 0) {
                float* s = smem + tile % kStreamSlots * kSlot;
#pragma unroll
                for (int i = tid; i < kScanTile * kCh4; i += kStreamHelpers) {
                    const int t = i / kCh4, q = (i - t * kCh4) * 4;
                    const bool on = t < n && c_base + q < p.inner;
                    const size_t row = row0 + at + min(t, n - 1);
                    const int cc = min(c_base + q, p.inner - 4);
                    cp_async16(s + t * kNch + q, p.x + row * p.x_ld + cc, on);
                    cp_async16(s + kDt + t * kNch + q, p.dt + row * p.dt_ld + cc, on);
                    cp_async16(s + kZ + t * kNch + q, p.z + row * p.z_ld + cc, on);
                }
#pragma unroll
                for (int i = kStreamHelpers - 1 - tid; i < kScanTile * kNp4; i += kStreamHelpers) {
                    const int t = i / kNp4, q = (i - t * kNp4) * 4;
                    const bool on = t < n;
                    const size_t row = row0 + at + min(t, n - 1);
                    cp_async16(s + kB + t * kNp + q, p.bc + row * p.bc_ld + p.b_off + q, on);
                    cp_async16(s + kC + t * kNp + q, p.bc + row * p.bc_ld + p.c_off + q, on);
                }
                at += n;
                left -= n;
                next_chunk();
            }
            cp_async_commit();  // a group per tile, also past the end, so that the count of those in flight stays the same
        };
        const int my_q = tid % kCh4 * 4;  // the four channels this thread prepares and writes
        const bool my_live = c_base + my_q < p.inner;
        const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 my_bias = my_live ? *reinterpret_cast<const float4*>(p.dt_bias + c_base + my_q) : zero4;
        const float4 my_d = my_live ? *reinterpret_cast<const float4*>(p.d + c_base + my_q) : zero4;
        auto finish = [&](int tile) {  // y of a tile is there
            const float* s = smem + tile % kStreamSlots * kSlot;
            const Tile of = s_tile[tile % kStreamSlots];
            if (!my_live) return;
#pragma unroll
            for (int i = tid; i < kScanTile * kCh4; i += kStreamHelpers) {
                if (i >= of.n * kCh4) break;
                const float4 xv = reinterpret_cast<const float4*>(s)[i], yv = reinterpret_cast<const float4*>(s + kY)[i], zv = reinterpret_cast<const float4*>(s + kZ)[i];
                p.out.store4(row0 + of.t + i / kCh4, c_base + my_q,
                             make_float4(fmaf(my_d.x, xv.x, yv.x) * fast_silu(zv.x), fmaf(my_d.y, xv.y, yv.y) * fast_silu(zv.y),
                                         fmaf(my_d.z, xv.z, yv.z) * fast_silu(zv.z), fmaf(my_d.w, xv.w, yv.w) * fast_silu(zv.w)));
            }
        };
        stage(0);
        stage(1);
        stage(2);
        int tile = 0;
        for (bool more = true; more; tile++) {  // once past the end, which the scanners learn of in the same way
            if (tile >= 2) bar_wait(kBarDone + (tile & 1), kAll);  // tile - 2
            cp_async_wait<2>();  // all but the next two tiles'
            bar_wait(kBarHelpers, kStreamHelpers);  // every helper's copies have landed; every helper has finished tile - 3, whose slot tile + 3 takes
            stage(tile + 3);
            more = s_tile[tile % kStreamSlots].n > 0;
            if (more) {
                float* s = smem + tile % kStreamSlots * kSlot;
#pragma unroll
                for (int i = tid; i < kScanTile * kCh4; i += kStreamHelpers) {
                    const float4 raw = reinterpret_cast<const float4*>(s + kDt)[i], xv = reinterpret_cast<const float4*>(s)[i];
                    const float4 dt = make_float4(fast_softplus(raw.x + my_bias.x), fast_softplus(raw.y + my_bias.y), fast_softplus(raw.z + my_bias.z), fast_softplus(raw.w + my_bias.w));
                    reinterpret_cast<float4*>(s + kDt)[i] = dt;
                    reinterpret_cast<float4*>(s + kDtx)[i] = make_float4(dt.x * xv.x, dt.y * xv.y, dt.z * xv.z, dt.w * xv.w);
                }
            }
            bar_arrive(kBarReady + (tile & 1), kAll);
            if (tile >= 2) finish(tile - 2);
        }
        if (tile >= 2) {  // tile - 1 was the one past the end
            bar_wait(kBarDone + (tile & 1), kAll);
            finish(tile - 2);
        }
        cp_async_wait<0>();
        return;
    }

    // ---------------- scanners ----------------
    const int ch = threadIdx.x / kLanes, part = threadIdx.x % kLanes, c = c_base + ch;
    const bool live = c < p.inner;
    // the state; what the chunk adds up to from zero, and the state it began with
    f32x2 a[kS / 2], s[kS / 2], local[kS / 2], begin[kS / 2];
    const size_t sidx = (size_t)(live ? c : 0) * kNp + part * kS;
    const size_t slot_base = (size_t)p.st.slot[seq] * p.inner * kNp;
    {
        const float* from = p.st.pos0[seq] > 0 ? p.state + slot_base + sidx : nullptr;
#pragma unroll
        for (int i = 0; i < kS / 2; i++) {
            a[i] = live ? *reinterpret_cast<const f32x2*>(p.a2 + sidx + 2 * i) : 0;
            s[i] = live && from ? *reinterpret_cast<const f32x2*>(from + 2 * i) : 0;
            local[i] = begin[i] = 0;
        }
    }
    // Four tokens at a time: what they need is requested while the four before them are computed, and before those store their y (the
    // compiler must keep loads behind stores that might be to the same place). A channel's four y end up one per lane.
    struct Four {
        float dt[4], dtx[4];
        f32x2 b[4][kS / 2], c[4][kS / 2];
    };
    const bool high = part & 2, odd = part & 1;
    const int my_token = (high ? 2 : 0) + (odd ? 1 : 0);
    float sum_dt = 0.f;  // of the chunk
    bool first = true;   // the sequence's first chunk runs from the slot: its end state is the next one's start
    for (int tile = 0;; tile++) {
        bar_wait(kBarReady + (tile & 1), kAll);
        const Tile of = s_tile[tile % kStreamSlots];
        if (of.n == 0) break;
        float* const base = smem + tile % kStreamSlots * kSlot;
        const float *sdt = base + kDt + ch, *sdtx = base + kDtx + ch, *sb = base + kB + part * kS, *sc = base + kC + part * kS;
        float* const sy = base + kY + ch + my_token * kNch;
        auto load = [&](int t0, Four& f) {
#pragma unroll
            for (int t = 0; t < 4; t++) {
                f.dt[t] = sdt[(t0 + t) * kNch];
                f.dtx[t] = sdtx[(t0 + t) * kNch];
                load_pairs<kS>(sb + (t0 + t) * kNp, f.b[t]);
                load_pairs<kS>(sc + (t0 + t) * kNp, f.c[t]);
            }
        };
        // n: tokens of the four that count (a warp-uniform number; the state does not move at the others)
        auto four = [&](int t0, const Four& f, int n) {
            float y[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (t < n) sum_dt += f.dt[t];
                const f32x2 dt2 = pair(f.dt[t], f.dt[t]), dtx2 = pair(f.dtx[t], f.dtx[t]);
                f32x2 y2 = 0;
#pragma unroll
                for (int i = 0; i < kS / 2; i++) {
                    const float2 x = unpair(mul2(dt2, a[i]));
                    const f32x2 e = pair(ex2f(x.x), ex2f(x.y)), in = mul2(dtx2, f.b[t][i]), moved = fma2(e, s[i], in), from_zero = fma2(e, local[i], in);
                    if (t < n) { s[i] = moved; local[i] = from_zero; }
                    y2 = fma2(s[i], f.c[t][i], y2);
                }
                const float2 yv = unpair(y2);
                y[t] = yv.x + yv.y;
            }
            // the upper half of the lanes takes tokens 2 and 3 over, then every second lane the odd one of each two
            const float even = (high ? y[2] : y[0]) + __shfl_xor_sync(0xffffffffu, high ? y[0] : y[2], 2);
            const float next = (high ? y[3] : y[1]) + __shfl_xor_sync(0xffffffffu, high ? y[1] : y[3], 2);
            sy[t0 * kNch] = (odd ? next : even) + __shfl_xor_sync(0xffffffffu, odd ? even : next, 1);
        };
        Four f[2];
        load(0, f[0]);
        if (of.n == kScanTile) {
#pragma unroll
            for (int t = 0; t < kScanTile; t += 4) {
                if (t + 4 < kScanTile) load(t + 4, f[(t >> 2) + 1 & 1]);
                four(t, f[t >> 2 & 1], 4);
            }
        } else {  // places of tokens past the end hold zeros
            for (int t = 0; t < of.n; t += 4) {
                four(t, f[0], of.n - t);
                if (t + 4 < of.n) load(t + 4, f[0]);
            }
        }
        bar_arrive(kBarDone + (tile & 1), kAll);
        if (of.links) {
#pragma unroll
            for (int i = 0; i < kS / 2; i++) {
                if (!first) {
                    const float2 x = unpair(mul2(pair(sum_dt, sum_dt), a[i]));
                    s[i] = fma2(pair(ex2f(x.x), ex2f(x.y)), begin[i], local[i]);
                }
                begin[i] = s[i];
                local[i] = 0;
            }
            first = false;
            sum_dt = 0.f;
        }
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < kS / 2; i++) *reinterpret_cast<f32x2*>(p.state + slot_base + sidx + 2 * i) = s[i];
    }
}

// Pass 2: end states -> start states, sequence by sequence. The first chunk ran from the slot, so its end state is exact.
__global__ void __launch_bounds__(256) selective_scan_link_kernel(const ScanParams p) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int seq = blockIdx.y;
    const int k0 = p.seq_chunk0[seq], k1 = p.seq_chunk0[seq + 1];
    const size_t per = (size_t)p.inner * p.n_pad;
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (k1 - k0 < 2 || i >= per) return;
    const int c = int(i / p.n_pad);  // the last chunk leaves no end state; what is read in its place goes nowhere
    const float a = p.a2[i];
    float s = p.st.pos0[seq] > 0 ? p.state[(size_t)p.st.slot[seq] * per + i] : 0.f;
    float end = p.part[(size_t)k0 * per + i];
    p.part[(size_t)k0 * per + i] = s;
    s = end;
    constexpr int kAhead = 8;  // chunks whose end states are requested together
    for (int kb = k0 + 1; kb < k1; kb += kAhead) {
        float e[kAhead], f[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
            const int k = min(kb + j, k1 - 1);
            e[j] = p.part[(size_t)k * per + i];
            f[j] = p.part_sum[(size_t)k * p.inner + c];
        }
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
            if (kb + j >= k1) break;
            p.part[(size_t)(kb + j) * per + i] = s;
            s = fmaf(ex2f(a * f[j]), s, e[j]);
        }
    }
}

// ---- real-gated linear recurrent unit -------------------------------------------------------------------------------
// r = sigmoid(gr + br), i = sigmoid(gi + bi), log a = -8 r softplus(lam), S <- a S + sqrt(1 - a^2) i u;
// out = out_scale * S * gelu(y + y_bias). gates [rows][...]: the products of the two block-diagonal gate matrices, block b's
// m recurrence gates followed by its m input gates.
struct LruParams {
    ingot_step st;
    const int32_t *chunk_seq, *chunk_t0, *chunk_len, *seq_chunk0;
    int n_chunks;
    const float* u; int u_ld;
    const float* gates; int gates_ld, block;
    const float *br, *bi, *sp;  // gate biases, softplus(lam)
    const float* y; int y_ld;
    const float* y_bias;
    float* state;     // [slot][width]
    float *part, *part_sum;  // [chunk][width]
    int width;
    float out_scale;
    ActOut out;
    bool whole;  // grid.y: sequences
};
template <bool kOutput, bool kExact>
__global__ void __launch_bounds__(128) gated_lru_kernel(const LruParams p) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int chunk = blockIdx.y, c = blockIdx.x * 128 + threadIdx.x;
    const bool whole = kOutput && p.whole;
    const int seq = whole ? chunk : p.chunk_seq[chunk], t0 = whole ? 0 : p.chunk_t0[chunk], len = whole ? p.st.len[seq] : p.chunk_len[chunk];
    const bool first = t0 == 0, last = t0 + len == p.st.len[seq];
    if ((!kOutput && last) || (whole && len < 1) || c >= p.width) return;
    const size_t row0 = (size_t)p.st.row_start[seq] + t0;
    const int gcol = (c / p.block) * 2 * p.block + c % p.block;
    const float br = p.br[c], bi = p.bi[c], k = -8.0f * p.sp[c], yb = kOutput ? p.y_bias[c] : 0.f;
    float* slot = p.state + (size_t)p.st.slot[seq] * p.width + c;
    float s = 0.f;
    if (kOutput && !(first && last)) s = p.part[(size_t)chunk * p.width + c];
    else if (first && p.st.pos0[seq] > 0) s = *slot;
    float sum = 0.f;
    const float* u = p.u + row0 * p.u_ld + c;
    const float* g = p.gates + row0 * p.gates_ld + gcol;
    const float* y = kOutput ? p.y + row0 * p.y_ld + c : nullptr;
    constexpr int kAhead = 8;  // tokens whose inputs are requested together
    for (int tb = 0; tb < len; tb += kAhead) {
        float gr[kAhead], gi[kAhead], uv[kAhead], yv[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
            const size_t t = min(tb + i, len - 1);
            gr[i] = g[t * p.gates_ld];
            gi[i] = g[t * p.gates_ld + p.block];
            uv[i] = u[t * p.u_ld];
            if (kOutput) yv[i] = y[t * p.y_ld];
        }
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
            if (tb + i >= len) break;
            const float log_a = k * (kExact ? sigmoidf(gr[i] + br) : fast_sigmoid(gr[i] + br));
            const float in = (kExact ? sigmoidf(gi[i] + bi) : fast_sigmoid(gi[i] + bi)) * uv[i];
            const float e = expm1f(log_a);  // a - 1; 1 - a^2 = -e (2 + e)
            s += fmaf(e, s, sqrtf(-e * (2.0f + e)) * in);
            if (kOutput) p.out.store(row0 + tb + i, c, p.out_scale * s * (kExact ? gelu_tanhf(yv[i] + yb) : fast_gelu_tanh(yv[i] + yb)));
            else sum += log_a;
        }
    }
    if (!kOutput) {
        p.part[(size_t)chunk * p.width + c] = s;
        p.part_sum[(size_t)chunk * p.width + c] = sum;
    } else if (last) {
        *slot = s;
    }
}

// The three passes in one, to the same bits: a CTA walks 32 channels of a sequence. A warp takes 8 tokens of a tile of 128, computes their decays, inputs and gates and
// keeps them; the recurrence itself - two dependent operations a token - goes from warp to warp through shared memory, while the others compute. Beside the state
// the warps hand on what the chunk adds up to from zero, its sum of log a and the state that it began with: the next chunk begins with what the link pass makes of
// those. The next tile's rows are requested before the current tile's states.
// Bound by instructions (expm1, sigmoids, square root: about 130 per value), which the passes spend twice on every value, and by the way from warp to
// warp (about 420 cycles). Against the passes over chunks (B200, calls replayed as a graph): 2048 tokens x 4096 channels 95 -> 57 us, 1000 x 4096 47 -> 30,
// 300 x 4096 28 -> 15, 2048 x 8192 179 -> 111.
constexpr int kLruRun = 8, kLruWarps = 16;
__global__ void __launch_bounds__(kLruWarps * 32) gated_lru_stream_kernel(const LruParams p) {
    __shared__ float4 s_hand[kLruWarps][32];  // to the warp after this one: state, from zero, sum of log a, begin
    INGOT_PDL_TRIGGER();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = min(blockIdx.x * 32 + lane, p.width - 1);
    const bool on = blockIdx.x * 32 + lane < p.width;
    const float br = p.br[c], bi = p.bi[c], k = -8.0f * p.sp[c], yb = p.y_bias[c];
    INGOT_PDL_WAIT();
    const int seq = gridDim.y - 1 - blockIdx.y, k0 = p.seq_chunk0[seq], k1 = p.seq_chunk0[seq + 1];  // as above
    if (k0 == k1) return;
    const int len = min(p.chunk_t0[k1 - 1] + p.chunk_len[k1 - 1], p.st.len[seq]);
    if (warp * kLruRun >= len) return;  // no tokens for this warp
    const size_t row0 = (size_t)p.st.row_start[seq];
    const int gcol = (c / p.block) * 2 * p.block + c % p.block;
    float* slot = p.state + (size_t)p.st.slot[seq] * p.width + c;
    const float* u = p.u + row0 * p.u_ld + c;
    const float* g = p.gates + row0 * p.gates_ld + gcol;
    const float* y = p.y + row0 * p.y_ld + c;
    float gr[kLruRun], gi[kLruRun], uv[kLruRun], yv[kLruRun];
    auto fetch = [&](int tile) {
#pragma unroll
        for (int i = 0; i < kLruRun; i++) {
            const size_t t = min((tile * kLruWarps + warp) * kLruRun + i, len - 1);
            gr[i] = g[t * p.gates_ld];
            gi[i] = g[t * p.gates_ld + p.block];
            uv[i] = u[t * p.u_ld];
            yv[i] = y[t * p.y_ld];
        }
    };
    const int second = k0 + 1 < k1 ? p.chunk_t0[k0 + 1] : -1;
    int chunk = k0 + 1;  // chunks before it begin before this warp's tokens
    fetch(0);
    for (int tile = 0; (tile * kLruWarps + warp) * kLruRun < len; tile++) {
        const int tb = (tile * kLruWarps + warp) * kLruRun, n = len - tb;  // tokens from here on
        unsigned begins = 0;  // bit i: a chunk begins with token i
        for (;;) {
            const int t0 = chunk + lane < k1 ? p.chunk_t0[chunk + lane] - tb : kLruRun, before = __popc(__ballot_sync(0xffffffffu, t0 < 0));
            begins = __reduce_or_sync(0xffffffffu, t0 >= 0 && t0 < kLruRun ? 1u << t0 : 0u);
            if (before <= 32 - kLruRun) break;  // the others may hold all that begin here
            chunk += before;
        }
        float log_a[kLruRun], e[kLruRun], b[kLruRun], out[kLruRun];
#pragma unroll
        for (int i = 0; i < kLruRun; i++) {
            log_a[i] = k * fast_sigmoid(gr[i] + br);
            e[i] = expm1f(log_a[i]);  // a - 1; 1 - a^2 = -e (2 + e)
            b[i] = sqrtf(-e[i] * (2.0f + e[i])) * (fast_sigmoid(gi[i] + bi) * uv[i]);
            out[i] = fast_gelu_tanh(yv[i] + yb);
            // computed here, not behind the wait below, where the compiler would put it to save registers: the other warps would wait for it in turn (4.5 times the time)
            asm volatile("" : "+f"(log_a[i]), "+f"(e[i]), "+f"(b[i]), "+f"(out[i]));
        }
        if (n > kLruWarps * kLruRun) fetch(tile + 1);
        float4 h;  // state, from zero, sum of log a, begin
        if (tile == 0 && warp == 0) {
            h = make_float4(p.st.pos0[seq] > 0 ? *slot : 0.f, 0.f, 0.f, 0.f);
        } else {
            bar_wait(warp, 64);
            h = s_hand[warp][lane];
        }
        float s[kLruRun];
        auto token = [&](int i) {
            h.x += fmaf(e[i], h.x, b[i]);
            h.y += fmaf(e[i], h.y, b[i]);
            h.z += log_a[i];
            s[i] = h.x;
        };
        auto link = [&](int i) {  // a chunk begins with token i; the first chunk ran from the slot: its end is the second one's start
            if (tb + i != second) h.x = fmaf(expf(h.z), h.w, h.y);
            h.w = h.x;
            h.y = h.z = 0.f;
        };
        if (begins & 1) link(0);
        if (begins < 2 && n >= kLruRun) {  // warp-uniform: no conditions on the way
#pragma unroll
            for (int i = 0; i < kLruRun; i++) token(i);
        } else {
#pragma unroll
            for (int i = 0; i < kLruRun; i++) {
                if (i > 0 && begins >> i & 1) link(i);
                if (i < n) token(i);
            }
        }
        if (n > kLruRun) {
            const int to = (warp + 1) % kLruWarps;
            s_hand[to][lane] = h;
            bar_arrive(to, 64);
        } else if (on) {
            *slot = h.x;
        }
#pragma unroll
        for (int i = 0; i < kLruRun; i++)
            if (i < n && on) p.out.store(row0 + tb + i, c, p.out_scale * s[i] * out[i]);
    }
}

__global__ void __launch_bounds__(128) gated_lru_link_kernel(const LruParams p) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int seq = blockIdx.y, c = blockIdx.x * 128 + threadIdx.x;
    const int k0 = p.seq_chunk0[seq], k1 = p.seq_chunk0[seq + 1];
    if (k1 - k0 < 2 || c >= p.width) return;
    float s = p.st.pos0[seq] > 0 ? p.state[(size_t)p.st.slot[seq] * p.width + c] : 0.f;
    float end = p.part[(size_t)k0 * p.width + c];
    p.part[(size_t)k0 * p.width + c] = s;
    s = end;
    constexpr int kAhead = 8;
    for (int kb = k0 + 1; kb < k1; kb += kAhead) {
        float e[kAhead], f[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
            const int k = min(kb + j, k1 - 1);
            e[j] = p.part[(size_t)k * p.width + c];
            f[j] = p.part_sum[(size_t)k * p.width + c];
        }
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
            if (kb + j >= k1) break;
            p.part[(size_t)(kb + j) * p.width + c] = s;
            s = fmaf(expf(f[j]), s, e[j]);
        }
    }
}

constexpr size_t kHalfSm = 116 * 1024;  // shared memory of which an SM has less than twice
int sm_count() {
    int dev = 0, num_sms = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? num_sms : 0;
}
// A call of single tokens (every decoded step) has one form.
ingot_scan::Form form_of(ingot_scan::Kind kind, const ingot_step* step, const ingot_scan_plan* plan, int channels, int states, int num_sms) {
    if (step->max_len == 1 || num_sms < 1) return ingot_scan::Form::chunks;
    return ingot_scan::choose(kind, {step->n_tok, step->max_len, step->n_seq, plan->max_chunks}, channels, states, num_sms).form;
}

int scan_lanes_log2(int n_state) {
    int l = 2;  // 4 lanes per channel up to 32 states, then as many as keep 8 states per lane
    while ((8 << l) < n_state) l++;
    return l;
}

// States a lane holds: an even number, so that pairs fill 64-bit registers.
int scan_states_per_lane(int n_state) {
    const int lg = scan_lanes_log2(n_state), per = ((n_state + (1 << lg) - 1) >> lg) + 1 & ~1;
    return lg > 2 && per < 6 ? 6 : per;
}

}  // namespace

extern "C" {

int ingot_causal_conv(const ingot_step* step, const float* in_dev, int in_ld, const float* in_bias_dev, const float* w_dev,
                      const float* bias_dev, int taps, int channels, int silu, float* state_dev, const ingot_act_out* out,
                      void* stream) {
    INGOT_REQUIRE(step_ok(step) && in_dev && w_dev && state_dev && out, "ingot_causal_conv: null argument or empty step");
    INGOT_REQUIRE(channels >= 1 && taps >= 1 && taps <= kMaxTaps, "ingot_causal_conv: between 1 and 16 taps");
    INGOT_REQUIRE((step->max_len + kConvRun - 1) / kConvRun <= 65535, "ingot_causal_conv: too many tokens of one sequence in one step");
    const bool four = taps >= 2 && taps <= kMaxConvTaps4 && channels % 4 == 0 && in_ld % 4 == 0 && out->ld % 4 == 0;
    // Four-channel form: runs of 8 tokens where that still is a CTA of 128 threads for every place on the GPU (about 65536 threads at the registers
    // a run of 8 takes), else of 4. A grid of the longest sequence's runs for every sequence is mostly empty CTAs where one prompt is beside many short portions:
    // 63 decoded tokens beside a prompt of 2048 of 8192 channels took 343 us with runs of 8 (169 with runs of 16, as they were), and 34 with the runs of
    // all sequences packed; of 2048 channels 86, 49 and 9. Finding one's sequence costs about a microsecond; past kPackedSeqs sequences runs of 16 bound the number of empty CTAs instead.
    constexpr int kPackedSeqs = 1024;
    auto rows = [&](int run) { return ((long long)step->max_len + run - 1) / run; };
    int run = !four ? kConvRun : (long long)step->n_tok * (channels / 4) >= 8ll * 65536 ? 8 : 4;
    const long long runs = (long long)step->n_tok / run + step->n_seq;  // at most, of all sequences
    const bool sparse = four && rows(run) * step->n_seq > 2 * runs, packed = sparse && step->n_seq <= kPackedSeqs && runs <= 65535;
    if (four && !packed) {
        if (sparse) run = kConvRun;
        while (rows(run) > 65535) run *= 2;  // 16 at most
    }
    const ConvParams p = {*step, in_dev, in_ld, in_bias_dev, w_dev, bias_dev, taps, channels, silu, state_dev, act_out(out)};
    const dim3 grid(four ? (channels + 511) / 512 : (channels + 127) / 128, unsigned(packed ? runs : rows(run)), packed ? 1u : unsigned(step->n_seq));
    auto pick = [&](auto two, auto three, auto any) { return taps == 2 ? two : taps == 3 ? three : any; };
    auto kernel = !four      ? taps == 4 ? causal_conv_kernel<4> : taps < 2 || taps > 4 ? causal_conv_kernel<0> : pick(causal_conv_kernel<2>, causal_conv_kernel<3>, causal_conv_kernel<4>)
                  : packed   ? run == 4 ? pick(causal_conv4_kernel<2, 4, true>, causal_conv4_kernel<3, 4, true>, causal_conv4_kernel<4, 4, true>)
                                        : pick(causal_conv4_kernel<2, 8, true>, causal_conv4_kernel<3, 8, true>, causal_conv4_kernel<4, 8, true>)
                  : run == 4 ? pick(causal_conv4_kernel<2, 4, false>, causal_conv4_kernel<3, 4, false>, causal_conv4_kernel<4, 4, false>)
                  : run == 8 ? pick(causal_conv4_kernel<2, 8, false>, causal_conv4_kernel<3, 8, false>, causal_conv4_kernel<4, 8, false>)
                             : pick(causal_conv4_kernel<2, 16, false>, causal_conv4_kernel<3, 16, false>, causal_conv4_kernel<4, 16, false>);
    INGOT_CUDA_TRY(ingot_launch_pdl(kernel, grid, dim3(128), 0, static_cast<cudaStream_t>(stream), p));
    return INGOT_OK;
}

int ingot_scan_state_pad(int n_state) {
    if (n_state < 1 || n_state > 256) return 0;
    return scan_states_per_lane(n_state) << scan_lanes_log2(n_state);
}

int ingot_selective_scan(const ingot_step* step, const ingot_scan_plan* plan, const float* x_dev, int x_ld, const float* dt_dev,
                         int dt_ld, const float* dt_bias_dev, const float* bc_dev, int bc_ld, int b_off, int c_off,
                         const float* z_dev, int z_ld, const float* a_log2e_dev, const float* d_dev, float* state_dev, int inner,
                         int n_state, int exact, const ingot_act_out* out, void* stream) {
    INGOT_REQUIRE(step_ok(step) && plan_ok(plan), "ingot_selective_scan: bad step or plan");
    INGOT_REQUIRE(x_dev && dt_dev && dt_bias_dev && bc_dev && z_dev && a_log2e_dev && d_dev && state_dev && out, "ingot_selective_scan: null argument");
    INGOT_REQUIRE(inner >= 4 && inner % 4 == 0 && x_ld % 4 == 0 && dt_ld % 4 == 0 && z_ld % 4 == 0 && out->ld % 4 == 0 && bc_ld % 4 == 0 && b_off % 4 == 0 && c_off % 4 == 0,
                  "ingot_selective_scan: rows and offsets must be multiples of 4 floats");
    const int n_pad = ingot_scan_state_pad(n_state);
    INGOT_REQUIRE(n_pad > 0, "ingot_selective_scan: between 1 and 256 states");
    const bool multi = plan->max_chunks > 1;
    INGOT_REQUIRE(!multi || (plan->scratch_dev && plan->scratch_floats >= (size_t)plan->n_chunks * inner * (n_pad + 1)),
                  "ingot_selective_scan: scratch too small");
    const int lg = scan_lanes_log2(n_state), n_ch = 256 >> lg;
    const int per_lane = scan_states_per_lane(n_state);
    ScanParams p = {*step, plan->chunk_seq, plan->chunk_t0, plan->chunk_len, plan->seq_chunk0, plan->n_chunks,
                    x_dev, x_ld, dt_dev, dt_ld, dt_bias_dev, bc_dev, bc_ld, b_off, c_off, z_dev, z_ld, a_log2e_dev, d_dev,
                    state_dev, plan->scratch_dev, plan->scratch_dev ? plan->scratch_dev + (size_t)plan->n_chunks * inner * n_pad : nullptr,
                    inner, n_pad, lg, act_out(out), false};
    const size_t smem = (size_t)kScanTile * (2 * (3 * n_ch + 2 * n_pad) + 2 * n_ch) * sizeof(float);
    typedef void (*Kernel)(ScanParams);
    Kernel k_end, k_out;
#define INGOT_SCAN_PICK(S, OUT)                                                                                                     \
    (exact ? (lg == 2 ? selective_scan_kernel<S, OUT, 2, true> : selective_scan_kernel<(S < 6 ? 6 : S), OUT, -1, true>)             \
           : (lg == 2 ? selective_scan_kernel<S, OUT, 2, false> : selective_scan_kernel<(S < 6 ? 6 : S), OUT, -1, false>))
#define INGOT_SCAN_CASE(S)                 \
    case S:                                \
        k_end = INGOT_SCAN_PICK(S, false); \
        k_out = INGOT_SCAN_PICK(S, true);  \
        break
    switch (per_lane) {  // more than 4 lanes: always 6 or 8 states per lane
        INGOT_SCAN_CASE(2); INGOT_SCAN_CASE(4); INGOT_SCAN_CASE(6); INGOT_SCAN_CASE(8);
        default: ingot_set_error("ingot_selective_scan: unsupported state count"); return INGOT_ERR_UNSUPPORTED;
    }
#undef INGOT_SCAN_CASE
#undef INGOT_SCAN_PICK
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid((inner + n_ch - 1) / n_ch, plan->n_chunks);
    if (smem > 48 * 1024) {
        INGOT_CUDA_TRY(cudaFuncSetAttribute(k_end, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        INGOT_CUDA_TRY(cudaFuncSetAttribute(k_out, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    }
    // More than 32 states and the exact form: the plan's chunks.
    const int num_sms = !exact && lg == 2 ? sm_count() : 0;
    const ingot_scan::Form form = form_of(ingot_scan::Kind::selective, step, plan, inner, n_pad, num_sms);
    if (form == ingot_scan::Form::stream) {
        const int ch = ingot_scan::stream_channels({step->n_tok, step->max_len, step->n_seq, plan->max_chunks}, inner, num_sms);
        const bool wide = ch == 64;
        Kernel k_stream = nullptr;
        switch (per_lane) {
            case 2: k_stream = wide ? selective_scan_stream_kernel<2, 64> : selective_scan_stream_kernel<2, 32>; break;
            case 4: k_stream = wide ? selective_scan_stream_kernel<4, 64> : selective_scan_stream_kernel<4, 32>; break;
            case 6: k_stream = wide ? selective_scan_stream_kernel<6, 64> : selective_scan_stream_kernel<6, 32>; break;
            case 8: k_stream = wide ? selective_scan_stream_kernel<8, 64> : selective_scan_stream_kernel<8, 32>; break;
        }
        const int ctas = (inner + ch - 1) / ch;
        // One CTA per SM where there are enough SMs: launched while the kernel before still holds some, two would share the first ones that come
        // free and take twice as long beside idle ones.
        const size_t need = size_t(kStreamSlots) * stream_slot_floats(ch, n_pad) * sizeof(float), bytes = (long long)ctas * step->n_seq <= num_sms ? std::max(need, kHalfSm) : need;
        INGOT_CUDA_TRY(cudaFuncSetAttribute(k_stream, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
        INGOT_CUDA_TRY(ingot_launch_pdl(k_stream, dim3(ctas, step->n_seq), dim3(ch * 4 + kStreamHelpers), bytes, s, p));
        return INGOT_OK;
    }
    if (form == ingot_scan::Form::tile && multi) {
        p.whole = true;
        INGOT_CUDA_TRY(ingot_launch_pdl(k_out, dim3(grid.x, step->n_seq), dim3(128), smem, s, p));
        return INGOT_OK;
    }
    if (multi) {
        INGOT_CUDA_TRY(ingot_launch_pdl(k_end, grid, dim3(128), smem, s, p));
        INGOT_CUDA_TRY(ingot_launch_pdl(selective_scan_link_kernel, dim3(unsigned(((size_t)inner * n_pad + 255) / 256), step->n_seq), dim3(256), 0, s, p));
    }
    INGOT_CUDA_TRY(ingot_launch_pdl(k_out, grid, dim3(128), smem, s, p));
    return INGOT_OK;
}

int ingot_gated_lru(const ingot_step* step, const ingot_scan_plan* plan, const float* u_dev, int u_ld, const float* gates_dev,
                    int gates_ld, int block, const float* r_bias_dev, const float* i_bias_dev, const float* softplus_lam_dev,
                    const float* y_dev, int y_ld, const float* y_bias_dev, float* state_dev, int width, float out_scale,
                    int exact, const ingot_act_out* out, void* stream) {
    INGOT_REQUIRE(step_ok(step) && plan_ok(plan), "ingot_gated_lru: bad step or plan");
    INGOT_REQUIRE(u_dev && gates_dev && r_bias_dev && i_bias_dev && softplus_lam_dev && y_dev && y_bias_dev && state_dev && out, "ingot_gated_lru: null argument");
    INGOT_REQUIRE(width >= 1 && block >= 1 && width % block == 0, "ingot_gated_lru: the width must be a multiple of the block size");
    const bool multi = plan->max_chunks > 1;
    INGOT_REQUIRE(!multi || (plan->scratch_dev && plan->scratch_floats >= (size_t)plan->n_chunks * width * 2), "ingot_gated_lru: scratch too small");
    LruParams p = {*step, plan->chunk_seq, plan->chunk_t0, plan->chunk_len, plan->seq_chunk0, plan->n_chunks, u_dev, u_ld, gates_dev, gates_ld,
                   block, r_bias_dev, i_bias_dev, softplus_lam_dev, y_dev, y_ld, y_bias_dev, state_dev, plan->scratch_dev,
                   plan->scratch_dev ? plan->scratch_dev + (size_t)plan->n_chunks * width : nullptr, width, out_scale, act_out(out), false};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid((width + 127) / 128, plan->n_chunks);
    const int num_sms = exact ? 0 : sm_count();
    const ingot_scan::Form form = form_of(ingot_scan::Kind::gated, step, plan, width, 1, num_sms);
    if (form == ingot_scan::Form::stream) {
        const int ctas = (width + 31) / 32;
        const size_t bytes = (long long)ctas * step->n_seq <= num_sms ? kHalfSm : 0;  // as above
        INGOT_CUDA_TRY(cudaFuncSetAttribute(gated_lru_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kHalfSm)));
        INGOT_CUDA_TRY(ingot_launch_pdl(gated_lru_stream_kernel, dim3(ctas, step->n_seq), dim3(kLruWarps * 32), bytes, s, p));
        return INGOT_OK;
    }
    if (form == ingot_scan::Form::tile && multi) {
        p.whole = true;
        INGOT_CUDA_TRY(ingot_launch_pdl(gated_lru_kernel<true, false>, dim3(grid.x, step->n_seq), dim3(128), 0, s, p));
        return INGOT_OK;
    }
    if (multi) {
        INGOT_CUDA_TRY(ingot_launch_pdl(exact ? gated_lru_kernel<false, true> : gated_lru_kernel<false, false>, grid, dim3(128), 0, s, p));
        INGOT_CUDA_TRY(ingot_launch_pdl(gated_lru_link_kernel, dim3((width + 127) / 128, step->n_seq), dim3(128), 0, s, p));
    }
    INGOT_CUDA_TRY(ingot_launch_pdl(exact ? gated_lru_kernel<true, true> : gated_lru_kernel<true, false>, grid, dim3(128), 0, s, p));
    return INGOT_OK;
}

}  // extern "C"
