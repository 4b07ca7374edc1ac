// Linear recurrences with a matrix state per head, over a ragged batch, and the gated norm their results pass through. No counterpart in
// the reference, which only has attention layers.
//
//     S_t = diag(a_t) S_(t-1) + k_t v_t^T,   y_t = S_t^T q_t (+ skip v_t)        S: n_state x n_value per head, f32
//
// The decay a_t is one number per state row - a power of a sigmoid (gated linear attention) - or one per head - exp(-rate dt) with a step
// size dt that also scales the input (state-space duality). Slots, positions and time chunks as in recurrent.cu: three passes over the chunks
// of a step, of which a sequence that is one chunk takes the last alone.
//
// Three kernels compute a chunk:
//   token by token   f32 arithmetic, the state in registers, decays through expm1: the exact form
//   a few tokens     the same arithmetic laid out for streaming the state once: decoded tokens, portions of a few
//   32 at a time     tensor cores (below): portions of prompts in the 16-bit form
//
// The tensor-core kernel. A warp owns 16 value columns and holds S^T for them as MMA accumulators, all states of the head: as they stand they
// are the A operand of the readout, so the state never leaves the registers. Let b_i be the sum of log a over tokens 1..i of a tile.
//   decays per state   m half of the tile's whole sum,  q^_i = q_i e^(b_i - m),  k^_j = k_j e^(m - b_j),  S' = e^m S (S from before the tile):
//                      y_i = S'^T q^_i + sum_(j <= i) (q^_i . k^_j) v_j,  S after the tile = e^m (S' + sum_j k^_j v_j^T). All exponents lie
//                      within +- m; a tile that decays out of that range is done in smaller parts, down to single tokens.
//   decays per head    q and k as they are, shared by the heads of a CTA as are their products:
//                      y_i = e^(b_i) S^T q_i + sum_(j <= i) (q_i . k_j) e^(b_i - b_j) dt_j v_j,  S after = e^b S + sum_j k_j (e^(b - b_j) dt_j v_j)^T.
// Sums, decays and the state are f32; the state and the scores enter products as bf16 hi + lo pairs, q^, k^ and v rounded to bf16 once.
#include <algorithm>
#include <type_traits>

#include "recurrent_common.cuh"

namespace {

struct LinearParams {
    ingot_step st;
    const int32_t *chunk_seq, *chunk_t0, *chunk_len, *seq_chunk0;
    ingot_linear_scan_in in;
    float* state;     // [slot][head][n_state][n_value]
    float* part;      // [chunk][head][n_state][n_value] end states, then start states
    float* part_sum;  // [chunk][head][n_state], or [chunk][head]: sum of log a
    float* y;
    int y_ld;
    int least, most;  // portions of least..most tokens are this launch's
    __device__ __forceinline__ int per_head() const { return in.n_state * in.n_value; }
    __device__ __forceinline__ size_t part_at(int chunk, int h) const { return ((size_t)chunk * in.n_head + h) * per_head(); }
    __device__ __forceinline__ size_t slot_at(int seq, int h) const { return ((size_t)st.slot[seq] * in.n_head + h) * per_head(); }
    // Start state of a chunk, null: zero. Pass 3 of a multi-chunk sequence takes the first chunk's from what pass 2 left too: the last
    // chunk's CTA may write the slot before this one gets to read it.
    __device__ __forceinline__ const float* start(bool output, int chunk, int seq, int h, bool first, bool last) const {
        if (output && !(first && last)) return part + part_at(chunk, h);
        return first && st.pos0[seq] > 0 ? state + slot_at(seq, h) : nullptr;
    }
};

// ---- token by token ---------------------------------------------------------------------------------------------------
// A CTA owns 32 value columns of one head over one time chunk; a warp an eighth of the states, a lane one column. Tiles of 16 tokens are
// staged in shared memory: q, k and a - 1 once per token and state.
constexpr int kScanTile = 16, kScanWarps = 8, kScanThreads = kScanWarps * 32;
template <int kR, bool kOutput>
__global__ void __launch_bounds__(kScanThreads) linear_scan_kernel(const LinearParams p) {
    extern __shared__ __align__(16) float smem[];
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int h = blockIdx.y, chunk = blockIdx.z, seq = p.chunk_seq[chunk], t0 = p.chunk_t0[chunk], len = p.chunk_len[chunk], whole = p.st.len[seq];
    const bool first = t0 == 0, last = t0 + len == whole;
    if (whole < p.least || whole > p.most || (!kOutput && last)) return;
    const int np = p.in.n_state, vp = p.in.n_value, R = np / kScanWarps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 32 + lane;
    const bool live = c < vp, per_state = p.in.decay == INGOT_DECAY_SIGMOID_POWER;
    const size_t row0 = (size_t)p.st.row_start[seq] + t0;
    float* const sq = smem;                                    // [16][np]
    float* const sk = sq + kScanTile * np;
    float* const se = sk + kScanTile * np;                     // [16][np], or [16]: a - 1
    float* const sv = se + kScanTile * (per_state ? np : 1);   // [16][32]
    float* const sp = sv + kScanTile * 32;                     // [16][8][32] parts of the result
    float* const sdt = sp + kScanTile * kScanThreads;          // [16] factor of k

    float s[kR];
    {
        const float* from = p.start(kOutput, chunk, seq, h, first, last);
#pragma unroll
        for (int r = 0; r < kR; r++) s[r] = from && live && r < R ? from[(size_t)(warp * R + r) * vp + c] : 0.f;
    }
    const float* q = p.in.q + row0 * p.in.q_ld + (size_t)(h / p.in.share) * np;
    const float* k = p.in.k + row0 * p.in.k_ld + (size_t)(h / p.in.share) * np;
    const float* v = p.in.v + row0 * p.in.v_ld + (size_t)h * vp + c;
    const float* z = p.in.z + row0 * p.in.z_ld + (per_state ? (size_t)h * np : (size_t)h);
    const float skip = kOutput && p.in.skip ? p.in.skip[h] : 0.f;
    constexpr int kSums = 2;  // n_state is at most 512
    float sum[kSums] = {0.f, 0.f};

    for (int tb = 0; tb < len; tb += kScanTile) {
        const int n_t = min(kScanTile, len - tb);
        if (tb) __syncthreads();
        if (per_state) {
#pragma unroll
            for (int i = 0; i < kSums; i++) {
                const int n = threadIdx.x + i * kScanThreads;
                if (n >= np) break;
                const float bias = p.in.bias[(size_t)h * np + n];
                for (int t = 0; t < n_t; t++) {
                    const float x = -softplusf(-(z[(size_t)(tb + t) * p.in.z_ld + n] + bias)) * p.in.power;
                    se[t * np + n] = expm1f(x);
                    sum[i] += x;
                }
            }
        } else if (threadIdx.x < n_t) {
            const float dt = softplusf(z[(size_t)(tb + threadIdx.x) * p.in.z_ld] + p.in.bias[h]), x = -p.in.rate[h] * dt;
            se[threadIdx.x] = expm1f(x);
            sdt[threadIdx.x] = dt;
            sum[0] += x;
        }
        if (!per_state) __syncthreads();  // the step sizes
        for (int i = threadIdx.x; i < n_t * np; i += kScanThreads) {
            const int t = i / np, n = i - t * np;
            sk[i] = k[(size_t)(tb + t) * p.in.k_ld + n] * (per_state ? 1.0f : sdt[t]);
            if (kOutput) sq[i] = q[(size_t)(tb + t) * p.in.q_ld + n] * p.in.q_scale;
        }
        for (int t = warp; t < n_t; t += kScanWarps) sv[t * 32 + lane] = live ? v[(size_t)(tb + t) * p.in.v_ld] : 0.f;
        __syncthreads();
        for (int t = 0; t < n_t; t++) {
            const float x = sv[t * 32 + lane];
            const float2* tk = reinterpret_cast<const float2*>(sk + t * np + warp * R);
            const float2* tq = reinterpret_cast<const float2*>(sq + t * np + warp * R);
            const float2* te = reinterpret_cast<const float2*>(se + t * np + warp * R);
            const float one = per_state ? 0.f : se[t];
            float o = 0.f;
#pragma unroll
            for (int r = 0; r < kR; r += 2) {
                if (r >= R) break;
                const float2 kk = tk[r / 2], e = per_state ? te[r / 2] : make_float2(one, one);
                s[r] += fmaf(e.x, s[r], kk.x * x);
                s[r + 1] += fmaf(e.y, s[r + 1], kk.y * x);
                if (kOutput) {
                    const float2 qq = tq[r / 2];
                    o = fmaf(s[r], qq.x, o);
                    o = fmaf(s[r + 1], qq.y, o);
                }
            }
            if (kOutput) sp[(t * kScanWarps + warp) * 32 + lane] = o;
        }
        if (kOutput) {
            __syncthreads();
            for (int t = warp; t < n_t; t += kScanWarps) {
                float o = skip * sv[t * 32 + lane];
#pragma unroll
                for (int w = 0; w < kScanWarps; w++) o += sp[(t * kScanWarps + w) * 32 + lane];
                if (live) p.y[(row0 + tb + t) * p.y_ld + (size_t)h * vp + c] = o;
            }
        }
    }
    if (!kOutput && blockIdx.x == 0) {
        if (per_state) {
#pragma unroll
            for (int i = 0; i < kSums; i++) {
                const int n = threadIdx.x + i * kScanThreads;
                if (n < np) p.part_sum[((size_t)chunk * p.in.n_head + h) * np + n] = sum[i];
            }
        } else if (warp == 0) {
            float total = sum[0];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
            if (lane == 0) p.part_sum[(size_t)chunk * p.in.n_head + h] = total;
        }
    }
    if (!live || (kOutput && !last)) return;
    float* to = kOutput ? p.state + p.slot_at(seq, h) : p.part + p.part_at(chunk, h);
#pragma unroll
    for (int r = 0; r < kR; r++)
        if (r < R) to[(size_t)(warp * R + r) * vp + c] = s[r];
}

// ---- a few tokens ------------------------------------------------------------------------------------------------------------
// Decoded tokens and portions of at most kFewTokens: bound by reading and writing the state. A CTA owns `cols` columns of one head (a power of
// two) and holds them as quads of columns, all of them requested before anything else is done.
constexpr int kFewTokens = 7, kFewThreads = 256, kFewWarps = kFewThreads / 32;
template <int kQuads>
__global__ void __launch_bounds__(kFewThreads, 4) linear_scan_few_kernel(const LinearParams p, int cols) {
    extern __shared__ __align__(16) float smem[];
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int h = blockIdx.y, seq = blockIdx.z, len = p.st.len[seq];
    if (len < p.least || len > p.most) return;
    const int np = p.in.n_state, vp = p.in.n_value, lanes = cols >> 2, c4 = threadIdx.x & (lanes - 1), r0 = threadIdx.x / lanes, step = kFewThreads / lanes;
    const int col = blockIdx.x * cols + c4 * 4;
    const bool per_state = p.in.decay == INGOT_DECAY_SIGMOID_POWER, go_on = p.st.pos0[seq] > 0;
    const size_t row0 = p.st.row_start[seq];
    float4* const state = reinterpret_cast<float4*>(p.state + p.slot_at(seq, h) + col);
    float4 s[kQuads];
#pragma unroll
    for (int j = 0; j < kQuads; j++) {
        const int r = r0 + j * step;
        s[j] = go_on && r < np ? __ldcs(state + (size_t)r * (vp / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float* const sq = smem;              // [len][np]
    float* const sk = sq + len * np;     // [len][np], times dt
    float* const se = sk + len * np;     // [len][np]: a - 1
    float* const sv = se + len * np;     // [len][cols]
    float* const so = sv + len * cols;   // [len][8][cols]
    const size_t qk = (size_t)(h / p.in.share) * np;
    for (int t = 0; t < len; t++) {
        for (int n = threadIdx.x; n < np; n += kFewThreads) {
            const float q = p.in.q[(row0 + t) * p.in.q_ld + qk + n], k = p.in.k[(row0 + t) * p.in.k_ld + qk + n];
            float x, dt = 1.f;
            if (per_state) {
                x = -softplusf(-(p.in.z[(row0 + t) * p.in.z_ld + (size_t)h * np + n] + p.in.bias[(size_t)h * np + n])) * p.in.power;
            } else {
                dt = softplusf(p.in.z[(row0 + t) * p.in.z_ld + h] + p.in.bias[h]);
                x = -p.in.rate[h] * dt;
            }
            sq[t * np + n] = q * p.in.q_scale;
            sk[t * np + n] = k * dt;
            se[t * np + n] = expm1f(x);
        }
        const int c = kFewThreads - 1 - (int)threadIdx.x;  // the threads that have no state left
        if (c < cols) sv[t * cols + c] = p.in.v[(row0 + t) * p.in.v_ld + (size_t)h * vp + blockIdx.x * cols + c];
    }
    __syncthreads();
    for (int t = 0; t < len; t++) {
        const float4 v = *reinterpret_cast<const float4*>(sv + t * cols + c4 * 4);
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < kQuads; j++) {
            const int r = r0 + j * step;
            if (r >= np) break;
            const float e = se[t * np + r], k = sk[t * np + r], q = sq[t * np + r];
            s[j].x += fmaf(e, s[j].x, k * v.x);
            s[j].y += fmaf(e, s[j].y, k * v.y);
            s[j].z += fmaf(e, s[j].z, k * v.z);
            s[j].w += fmaf(e, s[j].w, k * v.w);
            o.x = fmaf(s[j].x, q, o.x);
            o.y = fmaf(s[j].y, q, o.y);
            o.z = fmaf(s[j].z, q, o.z);
            o.w = fmaf(s[j].w, q, o.w);
        }
        for (int d = lanes; d < 32; d <<= 1) {  // lanes of a warp that hold the same columns
            o.x += __shfl_xor_sync(0xffffffffu, o.x, d);
            o.y += __shfl_xor_sync(0xffffffffu, o.y, d);
            o.z += __shfl_xor_sync(0xffffffffu, o.z, d);
            o.w += __shfl_xor_sync(0xffffffffu, o.w, d);
        }
        const int warp = threadIdx.x >> 5;
        if ((threadIdx.x & 31) < lanes) *reinterpret_cast<float4*>(so + (t * kFewWarps + warp) * cols + c4 * 4) = o;
    }
#pragma unroll
    for (int j = 0; j < kQuads; j++) {
        const int r = r0 + j * step;
        if (r < np) __stcs(state + (size_t)r * (vp / 4), s[j]);
    }
    __syncthreads();
    const float skip = p.in.skip ? p.in.skip[h] : 0.f;
    for (int i = threadIdx.x; i < len * cols; i += kFewThreads) {
        const int t = i / cols, c = i - t * cols;
        float y = skip * sv[i];
#pragma unroll
        for (int w = 0; w < kFewWarps; w++) y += so[(t * kFewWarps + w) * cols + c];
        p.y[(row0 + t) * p.y_ld + (size_t)h * vp + blockIdx.x * cols + c] = y;
    }
}

// Pass 2: end states -> start states, sequence by sequence, four values per thread. The first chunk ran from the slot, so its end state is
// exact; the last chunk leaves none.
__global__ void __launch_bounds__(256) linear_scan_link_kernel(const LinearParams p) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int h = blockIdx.y, seq = blockIdx.z, k0 = p.seq_chunk0[seq], k1 = p.seq_chunk0[seq + 1];
    const int i = (blockIdx.x * 256 + threadIdx.x) * 4, per = p.per_head();
    if (k1 - k0 < 2 || i >= per) return;
    const bool per_state = p.in.decay == INGOT_DECAY_SIGMOID_POWER;
    const size_t stride = (size_t)p.in.n_head * per, sum_stride = (size_t)p.in.n_head * (per_state ? p.in.n_state : 1);
    float* part = p.part + p.part_at(k0, h) + i;
    const float* sum = p.part_sum + k0 * sum_stride + (per_state ? (size_t)h * p.in.n_state + i / p.in.n_value : (size_t)h);
    auto at = [&](int k) { return reinterpret_cast<float4*>(part + k * stride); };
    float4 s = p.st.pos0[seq] > 0 ? *reinterpret_cast<const float4*>(p.state + p.slot_at(seq, h) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    const int n = k1 - k0 - 1;  // chunks that leave an end state
    constexpr int kAhead = 16;  // of which so many are requested together
    for (int kb = 0; kb < n; kb += kAhead) {
        float4 e[kAhead];
        float f[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
            if (kb + j >= n) break;
            e[j] = *at(kb + j);
            f[j] = sum[(kb + j) * sum_stride];
        }
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
            if (kb + j >= n) break;
            *at(kb + j) = s;
            const float a = kb + j == 0 ? 0.f : expf(f[j]);
            s = make_float4(fmaf(a, s.x, e[j].x), fmaf(a, s.y, e[j].y), fmaf(a, s.z, e[j].z), fmaf(a, s.w, e[j].w));
        }
    }
    *at(n) = s;
}

// ---- 32 tokens at a time on tensor cores ------------------------------------------------------------------------------------
constexpr int kTile = 32, kMaxWarps = 8;
constexpr float kRange = 144.0f;  // most a tile may decay by, in powers of two
// Warps of a CTA: `per_head` for each of `heads` heads that share q and k, 16 value columns each; long values take several CTAs.
struct WarpPlan {
    int per_head, heads, slices;
    WarpPlan(int n_value, int share) {
        const int tiles = n_value / 16;
        slices = (tiles + kMaxWarps - 1) / kMaxWarps;
        per_head = (tiles + slices - 1) / slices;
        heads = slices > 1 ? 1 : std::max(1, std::min(kMaxWarps / per_head, share));
    }
};
// Shared memory, offsets in bytes: everything but the number of heads is known when compiled, so that addresses are sums with constants.
template <int kN, bool kPerState>
struct MmaSmem {
    static constexpr int ld = kN + 4, v_ld = kMaxWarps * 16 + 4, op_ld = kN + 8, score_ld = kTile + 8;
    static constexpr int k = kTile * ld * 4, z = 2 * k;                           // raw q, k, z: [32][ld]
    static constexpr int v = z + (kPerState ? k : 0), v_bytes = kTile * v_ld * 4;  // [2][32][v_ld]
    static constexpr int op = v + 2 * v_bytes, plane = kTile * op_ld * 2;          // q^, k^: [32][op_ld] bf16
    static constexpr int in = op + 2 * plane, out = in + kN * 4, m = out + 2 * kN * 4, sum = m + kN * 4;
    static constexpr int head = kPerState ? sum + kN * 4 : in, head_floats = 4 * kTile;  // per head b, e^b, dt e^(total - b), dt: [4][32]
    static constexpr int score_plane = kTile * score_ld * 2;                       // per head hi, lo: [32][score_ld] bf16
    __host__ __device__ static int score(int heads) { return head + (kPerState ? 0 : heads * head_floats * 4); }
    static int bytes(int heads) { return score(heads) + heads * 2 * score_plane; }
};
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// (x, y) as a bf16 pair and what that leaves
__device__ __forceinline__ void split_bf16(float x, float y, uint32_t& hi, uint32_t& lo) {
    hi = pack_bf16(x, y);
    lo = pack_bf16(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}

template <int kN, bool kPerState, bool kOutput>
__global__ void __launch_bounds__(kMaxWarps * 32, kN <= 128 ? 2 : 1) linear_scan_mma_kernel(const LinearParams p, int per_head, int heads) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int chunk = blockIdx.z, seq = p.chunk_seq[chunk], t0 = p.chunk_t0[chunk], len = p.chunk_len[chunk], whole = p.st.len[seq];
    const bool first = t0 == 0, last = t0 + len == whole;
    if (whole < p.least || whole > p.most || (!kOutput && last)) return;
    const int np = p.in.n_state, vp = p.in.n_value, n_threads = blockDim.x, n_warps = n_threads >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j2 = (lane & 3) * 2;
    // heads h0.. of one group of heads that share q and k; this warp's head and first column
    const int runs = (p.in.share + heads - 1) / heads, group = blockIdx.y / runs, h0 = group * p.in.share + blockIdx.y % runs * heads;
    const int n_heads = min(heads, min((group + 1) * p.in.share, p.in.n_head) - h0), my = warp / per_head, h = h0 + min(my, n_heads - 1);
    const int slice0 = blockIdx.x * per_head * 16, v0 = slice0 + warp % per_head * 16;
    const bool live = my < n_heads && v0 < vp;
    typedef MmaSmem<kN, kPerState> L;
    const size_t row0 = (size_t)p.st.row_start[seq] + t0;
    const uint32_t s_base = (uint32_t)__cvta_generic_to_shared(smem_raw);
    float* const sq = reinterpret_cast<float*>(smem_raw);
    float* const sk = reinterpret_cast<float*>(smem_raw + L::k);
    float* const sz = reinterpret_cast<float*>(smem_raw + L::z);
    float* const s_in = reinterpret_cast<float*>(smem_raw + L::in);    // [kN]: what the accumulators are multiplied with before a tile,
    float* const s_out = reinterpret_cast<float*>(smem_raw + L::out);  // [2][kN]: what they lack after the last one and after this one
    float* const s_m = reinterpret_cast<float*>(smem_raw + L::m);
    float* const s_sum = reinterpret_cast<float*>(smem_raw + L::sum);
    float* const s_heads = reinterpret_cast<float*>(smem_raw + L::head);
    const float* const s_head = s_heads + my * L::head_floats;
    const int score = L::score(heads);

    const float* gq = p.in.q + row0 * p.in.q_ld + (size_t)group * np;
    const float* gk = p.in.k + row0 * p.in.k_ld + (size_t)group * np;
    const float* gv = p.in.v + row0 * p.in.v_ld + (size_t)h0 * vp + slice0;
    const float* gz = p.in.z + row0 * p.in.z_ld + (kPerState ? (size_t)h0 * np : (size_t)(h0 + min(warp, n_heads - 1)));
    const int v_cols = heads > 1 ? n_heads * vp : min(vp - slice0, n_warps * 16);
    // f(token, column) for every fourth column of the tile's rows of kQuads quads
    auto walk = [&](auto quads, auto&& f) {
        constexpr int kQuads = decltype(quads)::value;
        for (int i = threadIdx.x; i < kTile * kQuads; i += n_threads) f(i / kQuads, i % kQuads * 4);
    };
    constexpr std::integral_constant<int, kN / 4> kRow{};
    constexpr std::integral_constant<int, kMaxWarps * 4> kValues{};
    auto stage = [&](int tile) {
        float* v = reinterpret_cast<float*>(smem_raw + L::v + (tile & 1) * L::v_bytes);
        const size_t tb = (size_t)tile * kTile;
        const int left = len - int(tb);
        const float *q0 = gq + tb * p.in.q_ld, *k0 = gk + tb * p.in.k_ld, *z0 = gz + tb * p.in.z_ld, *u0 = gv + tb * p.in.v_ld;
        walk(kRow, [&](int t, int c) {
            if (c >= np) return;
            const bool on = t < left;
            const int r = on ? t : 0;
            if (kOutput) cp_async16(sq + t * L::ld + c, q0 + r * p.in.q_ld + c, on);
            cp_async16(sk + t * L::ld + c, k0 + r * p.in.k_ld + c, on);
            if (kPerState) cp_async16(sz + t * L::ld + c, z0 + r * p.in.z_ld + c, on);
        });
        walk(kValues, [&](int t, int c) {
            if (c >= n_warps * 16) return;
            const bool on = t < left && c < v_cols;
            cp_async16(v + t * L::v_ld + c, u0 + (on ? t * p.in.v_ld + c : 0), on);
        });
        cp_async_commit();
    };
    stage(0);
    // decays of whole heads: a warp per head, a lane per token
    auto next_step = [&](int tile) { return !kPerState && warp < n_heads && tile * kTile + lane < len ? gz[(size_t)(tile * kTile + lane) * p.in.z_ld] : 0.f; };
    float z_step = next_step(0), log_sum = 0.f;

    // S^T: accumulator i holds states 8 i + j2, + 1 (elements 0, 1; 2, 3) of columns v0 + g (0, 1) and v0 + g + 8 (2, 3)
    float acc[kN / 8][4];
    {
        const float* from = live ? p.start(kOutput, chunk, seq, h, first, last) : nullptr;
#pragma unroll
        for (int i = 0; i < kN / 8; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[i][e] = from && i * 8 < np ? from[(size_t)(i * 8 + j2 + (e & 1)) * vp + v0 + g + (e >> 1) * 8] : 0.f;
    }
    if (kPerState)
        for (int n = threadIdx.x; n < np; n += n_threads) {
            s_sum[n] = 0.f;
            s_out[n] = 1.f;
        }
    int turn = 0;
    const float skip = kOutput && p.in.skip ? p.in.skip[h] : 0.f;
    constexpr float kLog2e = 1.44269504f;
    const int step_head = h0 + min(warp, n_heads - 1);
    const float rate = kPerState ? p.in.power : p.in.rate[step_head] * kLog2e, head_bias = kPerState ? 0.f : p.in.bias[step_head];

    const int n_tiles = (len + kTile - 1) / kTile;
    for (int tile = 0; tile < n_tiles; tile++) {
        cp_async_wait<0>();
        __syncthreads();  // the tile is in, and every warp is done with the operands and the other value buffer
        const float* sv = reinterpret_cast<const float*>(smem_raw + L::v + (tile & 1) * L::v_bytes);
        const int n_t = min(kTile, len - tile * kTile);
        int lo = 0, width = kTile;
        while (lo < n_t) {
            const int hi = min(n_t, lo + width);
            if (lo) __syncthreads();  // the operands are free again
            bool far = false;
            if (kPerState) {
                // ---- q^, k^ and e^m of tokens lo..hi-1: a warp takes 16 states, a lane two of them and eight tokens
                const int c2 = lane & 7, oct = lane >> 3;
                for (int blk = warp; blk < np / 16; blk += n_warps) {
                    const int n = blk * 16 + c2 * 2;
                    const float2 bias = *reinterpret_cast<const float2*>(p.in.bias + (size_t)h0 * np + n);
                    float2 b[8], run = make_float2(0.f, 0.f);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int t = oct * 8 + j;
                        const bool on = t >= lo && t < hi;
                        const float2 z = *reinterpret_cast<const float2*>(sz + t * L::ld + n);
                        run.x += on ? fmaxf(fast_log2_sigmoid(z.x + bias.x) * rate, -kRange) : 0.f;
                        run.y += on ? fmaxf(fast_log2_sigmoid(z.y + bias.y) * rate, -kRange) : 0.f;
                        b[j] = run;
                    }
                    float2 upto = run;
#pragma unroll
                    for (int o = 8; o <= 16; o <<= 1) {
                        const float ux = __shfl_up_sync(0xffffffffu, upto.x, o), uy = __shfl_up_sync(0xffffffffu, upto.y, o);
                        if (lane >= o) { upto.x += ux; upto.y += uy; }
                    }
                    const float2 before = make_float2(upto.x - run.x, upto.y - run.y);  // tokens of the lanes below
                    run.x = __shfl_sync(0xffffffffu, upto.x, 24 + c2);
                    run.y = __shfl_sync(0xffffffffu, upto.y, 24 + c2);
                    far = far || run.x < -kRange || run.y < -kRange;
                    const float2 m = make_float2(0.5f * run.x, 0.5f * run.y);
                    if (oct == 0) {
                        const float2 f = make_float2(ex2f(m.x), ex2f(m.y)), lack = *reinterpret_cast<const float2*>(s_out + turn * kN + n);
                        *reinterpret_cast<float2*>(s_in + n) = make_float2(lack.x * f.x, lack.y * f.y);
                        *reinterpret_cast<float2*>(s_out + (turn ^ 1) * kN + n) = f;
                        if (!kOutput) *reinterpret_cast<float2*>(s_m + n) = m;
                    }
                    const float2 off = make_float2(before.x - m.x, before.y - m.y);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const int t = oct * 8 + j;
                        const bool on = t >= lo && t < hi;
                        const float2 d = make_float2(off.x + b[j].x, off.y + b[j].y);
                        unsigned char* to = smem_raw + L::op + (t * L::op_ld + n) * 2;
                        if (kOutput) {
                            const float2 q = *reinterpret_cast<const float2*>(sq + t * L::ld + n);
                            *reinterpret_cast<uint32_t*>(to) = on ? pack_bf16(q.x * p.in.q_scale * ex2f(d.x), q.y * p.in.q_scale * ex2f(d.y)) : 0u;
                        }
                        const float2 k = *reinterpret_cast<const float2*>(sk + t * L::ld + n);
                        *reinterpret_cast<uint32_t*>(to + L::plane) = on ? pack_bf16(k.x * ex2f(-d.x), k.y * ex2f(-d.y)) : 0u;
                    }
                }
            } else {
                // ---- q and k as they are; per head and token b, e^b, dt e^(total - b) and dt
                walk(kRow, [&](int t, int c) {
                    if (c >= np) return;
                    unsigned char* to = smem_raw + L::op + (t * L::op_ld + c) * 2;
                    if (kOutput) {
                        const float4 q = *reinterpret_cast<const float4*>(sq + t * L::ld + c);
                        *reinterpret_cast<uint2*>(to) = make_uint2(pack_bf16(q.x * p.in.q_scale, q.y * p.in.q_scale), pack_bf16(q.z * p.in.q_scale, q.w * p.in.q_scale));
                    }
                    const float4 k = *reinterpret_cast<const float4*>(sk + t * L::ld + c);
                    *reinterpret_cast<uint2*>(to + L::plane) = make_uint2(pack_bf16(k.x, k.y), pack_bf16(k.z, k.w));
                });
                if (warp < n_heads) {
                    const float dt = lane < n_t ? fast_softplus(z_step + head_bias) : 0.f;
                    float b = -rate * dt;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const float u = __shfl_up_sync(0xffffffffu, b, o);
                        if (lane >= o) b += u;
                    }
                    const float total = __shfl_sync(0xffffffffu, b, 31);
                    float* to = s_heads + warp * L::head_floats + lane;
                    to[0] = b;
                    to[kTile] = ex2f(b);
                    to[2 * kTile] = ex2f(total - b) * dt;
                    to[3 * kTile] = dt;
                    log_sum += total;
                }
            }
            if (__syncthreads_or(far && hi - lo > 1)) {  // too much decay for one go: fewer tokens
                width = (hi - lo) / 2;
                continue;
            }
            turn ^= 1;
            if (hi == n_t && tile + 1 < n_tiles) {  // the raw tile is used up
                stage(tile + 1);
                z_step = next_step(tile + 1);
            }
            if (kPerState && !kOutput)
                for (int n = threadIdx.x; n < np; n += n_threads) s_sum[n] += 2.0f * s_m[n];

            if (kOutput) {
                // ---- scores q^_i . k^_j, j <= i: a warp takes blocks of 16 tokens i and 8 tokens j
                for (int blk = warp; blk < 6; blk += n_warps) {
                    const int mi = blk < 2 ? 0 : 1, nj = blk < 2 ? blk : blk - 2;
                    if (mi * 16 >= hi) continue;
                    float c[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
                    const uint32_t a_addr = s_base + L::op + ((mi * 16 + (lane & 15)) * L::op_ld + (lane >> 4) * 8) * 2;
                    const uint32_t b_addr = s_base + L::op + L::plane + ((nj * 8 + (lane & 7)) * L::op_ld + (lane >> 3) * 8) * 2;  // two steps of 16 states at a time
#pragma unroll 4
                    for (int ks = 0; ks < np / 16; ks += 2) {
                        uint32_t a[4], b[4];
                        ldmatrix4(a, a_addr + ks * 32);
                        ldmatrix4(b, b_addr + ks * 32);
                        mma_bf16(c, a, b[0], b[1]);
                        if (ks + 1 < np / 16) {
                            ldmatrix4(a, a_addr + ks * 32 + 32);
                            mma_bf16(d, a, b[2], b[3]);
                        }
                    }
                    for (int k = 0; k < n_heads; k++) {
                        const float* hd = s_heads + k * L::head_floats;
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int i = mi * 16 + g + 8 * e, j = nj * 8 + j2;
                            float x = c[2 * e] + d[2 * e], y = c[2 * e + 1] + d[2 * e + 1];
                            if (!kPerState) {
                                const float2 bj = *reinterpret_cast<const float2*>(hd + j), dt = *reinterpret_cast<const float2*>(hd + 3 * kTile + j);
                                x *= ex2f(hd[i] - bj.x) * dt.x;
                                y *= ex2f(hd[i] - bj.y) * dt.y;
                            }
                            uint32_t sh, sl;
                            split_bf16(j <= i ? x : 0.f, j + 1 <= i ? y : 0.f, sh, sl);
                            unsigned char* to = smem_raw + score + k * 2 * L::score_plane + (i * L::score_ld + j) * 2;
                            *reinterpret_cast<uint32_t*>(to) = sh;
                            *reinterpret_cast<uint32_t*>(to + L::score_plane) = sl;
                        }
                    }
                }
            }
            float o[4][4] = {};
            if (live) {
                uint32_t va[2][4];  // (what the state takes in of) V^T as A operand, 16 tokens each
                {
                    const float* t = sv + j2 * L::v_ld + warp * 16 + g;
#pragma unroll
                    for (int s = 0; s < 2; s++) {
                        const float* a = t + s * 16 * L::v_ld;
                        float2 w0 = make_float2(1.f, 1.f), w1 = w0;
                        if (!kPerState) {
                            w0 = *reinterpret_cast<const float2*>(s_head + 2 * kTile + s * 16 + j2);
                            w1 = *reinterpret_cast<const float2*>(s_head + 2 * kTile + s * 16 + j2 + 8);
                        }
                        va[s][0] = pack_bf16(a[0] * w0.x, a[L::v_ld] * w0.y);
                        va[s][1] = pack_bf16(a[8] * w0.x, a[L::v_ld + 8] * w0.y);
                        va[s][2] = pack_bf16(a[8 * L::v_ld] * w1.x, a[9 * L::v_ld] * w1.y);
                        va[s][3] = pack_bf16(a[8 * L::v_ld + 8] * w1.x, a[9 * L::v_ld + 8] * w1.y);
                    }
                }
                // ---- y += S'^T q^; S' += k^ v^T. The accumulators hold the last tile's S', its e^m is made up for with this one's.
                const uint32_t q_addr = s_base + L::op + (((lane & 7) + ((lane >> 4) & 1) * 8) * L::op_ld + ((lane >> 3) & 1) * 8) * 2;          // B operand, tokens are columns
                const uint32_t k_addr = s_base + L::op + L::plane + (((lane & 7) + ((lane >> 3) & 1) * 8) * L::op_ld + (lane >> 4) * 8) * 2;  // B operand, tokens are rows
                const float keep = kPerState ? 1.f : s_head[kTile + kTile - 1];
#pragma unroll
                for (int i = 0; i < kN / 16; i++) {
                    if (i * 16 >= np) break;
                    float(&x)[4] = acc[2 * i];
                    float(&y)[4] = acc[2 * i + 1];
                    float2 f0 = make_float2(keep, keep), f1 = f0;
                    if (kPerState) {
                        f0 = *reinterpret_cast<const float2*>(s_in + i * 16 + j2);
                        f1 = *reinterpret_cast<const float2*>(s_in + i * 16 + 8 + j2);
                        x[0] *= f0.x; x[1] *= f0.y; x[2] *= f0.x; x[3] *= f0.y;
                        y[0] *= f1.x; y[1] *= f1.y; y[2] *= f1.x; y[3] *= f1.y;
                    }
                    if (kOutput) {
                        uint32_t sh[4], sl[4], q[4];
                        split_bf16(x[0], x[1], sh[0], sl[0]);
                        split_bf16(x[2], x[3], sh[1], sl[1]);
                        split_bf16(y[0], y[1], sh[2], sl[2]);
                        split_bf16(y[2], y[3], sh[3], sl[3]);
#pragma unroll
                        for (int t = 0; t < 2; t++) {
                            ldmatrix4(q, q_addr + t * 16 * L::op_ld * 2 + i * 32);
                            mma_bf16(o[2 * t], sh, q[0], q[1]);
                            mma_bf16(o[2 * t + 1], sh, q[2], q[3]);
                            mma_bf16(o[2 * t], sl, q[0], q[1]);
                            mma_bf16(o[2 * t + 1], sl, q[2], q[3]);
                        }
                    }
                    if (!kPerState) {
                        x[0] *= keep; x[1] *= keep; x[2] *= keep; x[3] *= keep;
                        y[0] *= keep; y[1] *= keep; y[2] *= keep; y[3] *= keep;
                    }
#pragma unroll
                    for (int s = 0; s < 2; s++) {
                        uint32_t k[4];
                        ldmatrix4_trans(k, k_addr + s * 16 * L::op_ld * 2 + i * 32);
                        mma_bf16(x, va[s], k[0], k[1]);
                        mma_bf16(y, va[s], k[2], k[3]);
                    }
                }
            }
            if (kOutput) {
                __syncthreads();  // the scores are in
                if (live) {
                    const uint32_t addr = s_base + score + my * 2 * L::score_plane + (((lane & 7) + ((lane >> 4) & 1) * 8) * L::score_ld + ((lane >> 3) & 1) * 8) * 2;
                    if (!kPerState) {
#pragma unroll
                        for (int t = 0; t < 4; t++) {
                            const float2 f = *reinterpret_cast<const float2*>(s_head + kTile + t * 8 + j2);
                            o[t][0] *= f.x; o[t][1] *= f.y; o[t][2] *= f.x; o[t][3] *= f.y;
                        }
                    }
#pragma unroll
                    for (int s = 0; s < 2; s++) {
                        if (s * 16 >= hi) break;
                        uint32_t va[4];
                        const float* a = sv + (j2 + s * 16) * L::v_ld + warp * 16 + g;
                        va[0] = pack_bf16(a[0], a[L::v_ld]);
                        va[1] = pack_bf16(a[8], a[L::v_ld + 8]);
                        va[2] = pack_bf16(a[8 * L::v_ld], a[9 * L::v_ld]);
                        va[3] = pack_bf16(a[8 * L::v_ld + 8], a[9 * L::v_ld + 8]);
#pragma unroll
                        for (int t = s; t < 2; t++) {  // tokens 16 t..; later ones do not score earlier ones
                            if (t * 16 >= hi) break;
                            uint32_t ah[4], al[4];
                            ldmatrix4(ah, addr + (t * 16 * L::score_ld + s * 16) * 2);
                            ldmatrix4(al, addr + L::score_plane + (t * 16 * L::score_ld + s * 16) * 2);
                            mma_bf16(o[2 * t], va, ah[0], ah[1]);
                            mma_bf16(o[2 * t + 1], va, ah[2], ah[3]);
                            mma_bf16(o[2 * t], va, al[0], al[1]);
                            mma_bf16(o[2 * t + 1], va, al[2], al[3]);
                        }
                    }
                    float* y = p.y + (row0 + tile * kTile + j2) * p.y_ld + (size_t)h * vp + v0 + g;
                    const float* u = sv + j2 * L::v_ld + warp * 16 + g;
                    const bool all = lo == 0 && hi == kTile;
#pragma unroll
                    for (int t = 0; t < 4; t++)
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int tok = t * 8 + (e & 1), c = (e >> 1) * 8;
                            if (all || (tok + j2 >= lo && tok + j2 < hi)) y[tok * p.y_ld + c] = kPerState ? o[t][e] : fmaf(skip, u[tok * L::v_ld + c], o[t][e]);
                        }
                }
            }
            lo = hi;
        }
    }
    if (!kOutput && blockIdx.x == 0) {
        constexpr float kLn2 = 0.69314718f;
        if (kPerState) {
            __syncthreads();
            for (int n = threadIdx.x; n < np; n += n_threads) p.part_sum[((size_t)chunk * p.in.n_head + h0) * np + n] = s_sum[n] * kLn2;
        } else if (warp < n_heads && lane == 0) {
            p.part_sum[(size_t)chunk * p.in.n_head + h0 + warp] = log_sum * kLn2;
        }
    }
    if (!live || (kOutput && !last)) return;
    float* to = kOutput ? p.state + p.slot_at(seq, h) : p.part + p.part_at(chunk, h);
#pragma unroll
    for (int i = 0; i < kN / 8; i++)
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (i * 8 < np) {
                const int n = i * 8 + j2 + (e & 1);
                to[(size_t)n * vp + v0 + g + (e >> 1) * 8] = kPerState ? acc[i][e] * s_out[turn * kN + n] : acc[i][e];
            }
}

// ---- gated norm ---------------------------------------------------------------------------------------------------------
// Per row: y = x act(gate), normed in equal parts, or x normed in equal parts and then times act(gate); the row is heads of `size` values
// stored `padded` apart. Results are the next product's operand, zeros in the padding.
struct GatedNormParams {
    ingot_gated_norm in;
    int n, part, n_rows;  // values of a row, of a part
    ActOut out;
};
__device__ __forceinline__ float gate_act(int act, bool exact, float z) {
    if (act == INGOT_GATE_SIGMOID) return exact ? sigmoidf(z) : fast_sigmoid(z);
    return exact ? siluf(z) : fast_silu(z);
}
// Parts that are whole 4-value runs of unpadded rows: kTeam threads hold a part in registers, kKeep runs each.
template <int kTeam, int kKeep>
__global__ void __launch_bounds__(256) gated_norm_kernel(const GatedNormParams p) {
    __shared__ float red[8];
    INGOT_PDL_TRIGGER();
    const int team = threadIdx.x / kTeam, i0 = threadIdx.x % kTeam, part = blockIdx.y * (256 / kTeam) + team;
    const bool on = part < p.in.parts;
    const size_t row = blockIdx.x;
    const int base = on ? part * p.part : 0;
    float4 w[kKeep], x[kKeep], z[kKeep];
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        const int i = (i0 + k * kTeam) * 4;
        w[k] = on && i < p.part ? *reinterpret_cast<const float4*>(p.in.weight + base + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    INGOT_PDL_WAIT();
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        const int i = (i0 + k * kTeam) * 4;
        const bool in = on && i < p.part;
        x[k] = in ? *reinterpret_cast<const float4*>(p.in.x + row * p.in.x_ld + base + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        z[k] = in ? *reinterpret_cast<const float4*>(p.in.gate + row * p.in.gate_ld + base + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int act = p.in.act;
    const bool exact = p.in.exact;
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        z[k] = make_float4(gate_act(act, exact, z[k].x), gate_act(act, exact, z[k].y), gate_act(act, exact, z[k].z), gate_act(act, exact, z[k].w));
        if (p.in.gate_first) x[k] = make_float4(x[k].x * z[k].x, x[k].y * z[k].y, x[k].z * z[k].z, x[k].w * z[k].w);
        ss = fmaf(x[k].x, x[k].x, ss); ss = fmaf(x[k].y, x[k].y, ss); ss = fmaf(x[k].z, x[k].z, ss); ss = fmaf(x[k].w, x[k].w, ss);
    }
#pragma unroll
    for (int o = (kTeam < 32 ? kTeam : 32) / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (kTeam > 32) {
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
        __syncthreads();
        ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) ss += red[i];
    }
    if (!on) return;
    const float inv = 1.0f / sqrtf(ss / float(p.part) + p.in.eps);
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        const int i = (i0 + k * kTeam) * 4;
        if (i >= p.part) continue;
        float4 v = make_float4(x[k].x * inv * w[k].x, x[k].y * inv * w[k].y, x[k].z * inv * w[k].z, x[k].w * inv * w[k].w);
        if (!p.in.gate_first) v = make_float4(v.x * z[k].x, v.y * z[k].y, v.z * z[k].z, v.w * z[k].w);
        p.out.store4(row, base + i, v);
    }
}
// Any sizes: a CTA per row and part.
__global__ void __launch_bounds__(256) gated_norm_any_kernel(const GatedNormParams p) {
    __shared__ float red[8];
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const size_t row = blockIdx.x;
    const int base = blockIdx.y * p.part, size = p.in.size, padded = p.in.padded;
    auto place = [&](int i) { return (base + i) / size * padded + (base + i) % size; };
    auto value = [&](int c, float& gate) {
        gate = gate_act(p.in.act, p.in.exact, p.in.gate[row * p.in.gate_ld + c]);
        const float x = p.in.x[row * p.in.x_ld + c];
        return p.in.gate_first ? x * gate : x;
    };
    float ss = 0.f, gate;
    for (int i = threadIdx.x; i < p.part; i += 256) {
        const float v = value(place(i), gate);
        ss = fmaf(v, v, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) ss += red[i];
    const float inv = 1.0f / sqrtf(ss / float(p.part) + p.in.eps);
    for (int i = threadIdx.x; i < p.part; i += 256) {
        const int c = place(i);
        float v = value(c, gate) * inv * p.in.weight[c];
        if (!p.in.gate_first) v *= gate;
        p.out.store(row, c, v);
        if ((base + i) % size == size - 1)
            for (int k = 1; k <= padded - size; k++) p.out.store(row, c + k, 0.f);
    }
}
// Without a norm: x act(gate), four columns per thread.
__global__ void __launch_bounds__(256) gated_rows_kernel(const GatedNormParams p) {
    INGOT_PDL_TRIGGER();
    INGOT_PDL_WAIT();
    const int c = (blockIdx.y * 256 + threadIdx.x) * 4;
    const size_t row = blockIdx.x;
    if (c >= p.in.heads * p.in.padded) return;
    const float4 x = *reinterpret_cast<const float4*>(p.in.x + row * p.in.x_ld + c), z = *reinterpret_cast<const float4*>(p.in.gate + row * p.in.gate_ld + c);
    const int act = p.in.act;
    const bool exact = p.in.exact;
    p.out.store4(row, c, make_float4(x.x * gate_act(act, exact, z.x), x.y * gate_act(act, exact, z.y), x.z * gate_act(act, exact, z.z), x.w * gate_act(act, exact, z.w)));
}

size_t scan_smem(const ingot_linear_scan_in& in) {
    const bool per_state = in.decay == INGOT_DECAY_SIGMOID_POWER;
    return sizeof(float) * (size_t(kScanTile) * (2 * in.n_state + (per_state ? in.n_state : 1)) + kScanTile * 32 + kScanTile * kScanThreads + kScanTile);
}
typedef void (*LinearKernel)(LinearParams);
template <bool kOutput>
LinearKernel pick_scan(int n_state) {
    const int r = n_state / kScanWarps;
    return r <= 2   ? linear_scan_kernel<2, kOutput>
           : r <= 4 ? linear_scan_kernel<4, kOutput>
           : r <= 8 ? linear_scan_kernel<8, kOutput>
           : r <= 16 ? linear_scan_kernel<16, kOutput>
           : r <= 32 ? linear_scan_kernel<32, kOutput>
                     : linear_scan_kernel<64, kOutput>;
}
// Columns a CTA of the few-tokens kernel owns, 0: it does not take these sizes. As many as leave two CTAs for every SM, at least 32; a thread
// holds up to 4 quads.
int few_columns(const ingot_linear_scan_in& in, int n_seq, int num_sms) {
    const int vp = in.n_value;
    if ((vp & (vp - 1)) != 0) return 0;
    int cols = std::min(vp, 128);
    while (cols > 16 && in.n_state * cols > 4 * 4 * kFewThreads) cols /= 2;
    while (cols > 32 && (long long)in.n_head * n_seq * (vp / cols) < 2 * num_sms) cols /= 2;
    return in.n_state * cols <= 4 * 4 * kFewThreads ? cols : 0;
}
int launch_few(const LinearParams& p, int cols, cudaStream_t s) {
    const int quads = (p.in.n_state * cols / 4 + kFewThreads - 1) / kFewThreads, len = std::min(p.most, p.st.max_len);
    const size_t smem = sizeof(float) * len * (3 * p.in.n_state + (1 + kFewWarps) * cols);
    auto kernel = quads <= 1 ? linear_scan_few_kernel<1> : quads <= 2 ? linear_scan_few_kernel<2> : linear_scan_few_kernel<4>;
    INGOT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    INGOT_CUDA_TRY(ingot_launch_pdl(kernel, dim3(p.in.n_value / cols, p.in.n_head, p.st.n_seq), dim3(kFewThreads), smem, s, p, cols));
    return INGOT_OK;
}
template <bool kOutput>
int launch_scan(const LinearParams& p, int n_chunks, cudaStream_t s) {
    const size_t smem = scan_smem(p.in);
    const LinearKernel kernel = pick_scan<kOutput>(p.in.n_state);
    INGOT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    INGOT_CUDA_TRY(ingot_launch_pdl(kernel, dim3((p.in.n_value + 31) / 32, p.in.n_head, n_chunks), dim3(kScanThreads), smem, s, p));
    return INGOT_OK;
}
template <int kN, bool kPerState, bool kOutput>
int launch_mma_sized(const LinearParams& p, int n_chunks, cudaStream_t s) {
    const WarpPlan w(p.in.n_value, kPerState ? 1 : p.in.share);
    const int groups = p.in.n_head / p.in.share, runs = (p.in.share + w.heads - 1) / w.heads, smem = MmaSmem<kN, kPerState>::bytes(w.heads);
    auto kernel = linear_scan_mma_kernel<kN, kPerState, kOutput>;
    INGOT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    INGOT_CUDA_TRY(ingot_launch_pdl(kernel, dim3(w.slices, groups * runs, n_chunks), dim3(w.per_head * w.heads * 32), size_t(smem), s, p, w.per_head, w.heads));
    return INGOT_OK;
}
template <bool kPerState, bool kOutput>
int launch_mma_decay(const LinearParams& p, int n_chunks, cudaStream_t s) {
    const int n = p.in.n_state;
    return n <= 16   ? launch_mma_sized<16, kPerState, kOutput>(p, n_chunks, s)
           : n <= 32 ? launch_mma_sized<32, kPerState, kOutput>(p, n_chunks, s)
           : n <= 64 ? launch_mma_sized<64, kPerState, kOutput>(p, n_chunks, s)
           : n <= 128 ? launch_mma_sized<128, kPerState, kOutput>(p, n_chunks, s)
                      : launch_mma_sized<256, kPerState, kOutput>(p, n_chunks, s);
}
template <bool kOutput>
int launch_mma(const LinearParams& p, int n_chunks, cudaStream_t s) {
    return p.in.decay == INGOT_DECAY_SIGMOID_POWER ? launch_mma_decay<true, kOutput>(p, n_chunks, s) : launch_mma_decay<false, kOutput>(p, n_chunks, s);
}

}  // namespace

extern "C" {

int ingot_linear_scan(const ingot_step* step, const ingot_scan_plan* plan, const ingot_linear_scan_in* in, float* state_dev, float* y_dev, int y_ld, int min_len, int impl,
                      void* stream) {
    INGOT_REQUIRE(step_ok(step) && plan_ok(plan) && in, "ingot_linear_scan: bad step or plan");
    INGOT_REQUIRE(in->q && in->k && in->v && in->z && in->bias && state_dev && y_dev, "ingot_linear_scan: null argument");
    const bool per_state = in->decay == INGOT_DECAY_SIGMOID_POWER;
    INGOT_REQUIRE(per_state || (in->decay == INGOT_DECAY_STEP && in->rate), "ingot_linear_scan: unknown decay");
    INGOT_REQUIRE(in->n_head >= 1 && in->n_head <= 65535 && in->n_state >= 16 && in->n_state % 16 == 0 && in->n_value >= 16 && in->n_value % 16 == 0 && in->share >= 1 && in->n_head % in->share == 0,
                  "ingot_linear_scan: states and values are multiples of 16, heads of the number that share");
    INGOT_REQUIRE(in->q_ld % 4 == 0 && in->k_ld % 4 == 0 && in->v_ld % 4 == 0 && (!per_state || in->z_ld % 4 == 0), "ingot_linear_scan: rows must be multiples of 4 floats");
    if (in->n_state > 512) {
        ingot_set_error("ingot_linear_scan: at most 512 states");
        return INGOT_ERR_UNSUPPORTED;
    }
    const bool multi = plan->max_chunks > 1, tensor = impl != 1 && in->n_state <= 256;
    const size_t per = (size_t)in->n_head * in->n_state * in->n_value;
    INGOT_REQUIRE(!multi || (plan->scratch_dev && plan->scratch_floats >= (size_t)plan->n_chunks * (per + (size_t)in->n_head * in->n_state)), "ingot_linear_scan: scratch too small");
    if (impl == 2 && !tensor) {
        ingot_set_error("ingot_linear_scan: the tensor-core kernel takes at most 256 states");
        return INGOT_ERR_UNSUPPORTED;
    }
    LinearParams p = {*step, plan->chunk_seq, plan->chunk_t0, plan->chunk_len, plan->seq_chunk0, *in, state_dev, plan->scratch_dev,
                      plan->scratch_dev ? plan->scratch_dev + (size_t)plan->n_chunks * per : nullptr, y_dev, y_ld, 0, 0x7fffffff};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // portions of a few tokens (one chunk each), on tensor cores from `from` tokens on, and token by token between
    static int num_sms = 0;
    if (!num_sms) {
        int dev = 0;
        INGOT_CUDA_TRY(cudaGetDevice(&dev));
        INGOT_CUDA_TRY(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev));
    }
    const int from = !tensor ? 0x7fffffff : impl == 2 ? 1 : INGOT_LINEAR_SCAN_TILE_FROM;
    const int cols = impl == 2 ? 0 : few_columns(*in, step->n_seq, num_sms);
    const int few = cols > 0 ? std::min(kFewTokens, from - 1) : 0;
    if (impl == 3 && (few == 0 || step->max_len > few)) {
        ingot_set_error("ingot_linear_scan: the kernel for few tokens takes a power of two of values, and at most " + std::to_string(kFewTokens) + " tokens");
        return INGOT_ERR_UNSUPPORTED;
    }
    auto range = [&](int least, int most) {
        LinearParams a = p;
        a.least = least;
        a.most = most;
        return a;
    };
    const bool some = few + 1 < from && min_len < from && step->max_len > few, many = step->max_len >= from;
    if (multi) {
        if (some)
            if (const int rc = launch_scan<false>(range(few + 1, from - 1), plan->n_chunks, s)) return rc;
        if (many)
            if (const int rc = launch_mma<false>(range(from, 0x7fffffff), plan->n_chunks, s)) return rc;
        INGOT_CUDA_TRY(ingot_launch_pdl(linear_scan_link_kernel, dim3((in->n_state * in->n_value + 1023) / 1024, in->n_head, step->n_seq), dim3(256), 0, s, p));
    }
    if (min_len <= few)
        if (const int rc = launch_few(range(0, few), cols, s)) return rc;
    if (some)
        if (const int rc = launch_scan<true>(range(few + 1, from - 1), plan->n_chunks, s)) return rc;
    if (many)
        if (const int rc = launch_mma<true>(range(from, 0x7fffffff), plan->n_chunks, s)) return rc;
    return INGOT_OK;
}

int ingot_gated_norm_rows(const ingot_gated_norm* norm, int n_rows, const ingot_act_out* out, void* stream) {
    INGOT_REQUIRE(norm && out && norm->x && norm->gate && n_rows >= 1, "ingot_gated_norm_rows: null argument");
    const ingot_gated_norm& g = *norm;
    INGOT_REQUIRE(g.heads >= 1 && g.size >= 1 && g.padded >= g.size && g.padded % 4 == 0 && g.x_ld % 4 == 0 && g.gate_ld % 4 == 0 && out->ld % 4 == 0,
                  "ingot_gated_norm_rows: rows must be multiples of 4 floats");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    GatedNormParams p = {g, g.heads * g.size, 0, n_rows, act_out(out)};
    if (!g.weight) {
        INGOT_CUDA_TRY(ingot_launch_pdl(gated_rows_kernel, dim3(n_rows, (g.heads * g.padded + 1023) / 1024), dim3(256), 0, s, p));
        return INGOT_OK;
    }
    INGOT_REQUIRE(g.parts >= 1 && p.n % g.parts == 0, "ingot_gated_norm_rows: the row does not form equal parts");
    p.part = p.n / g.parts;
    const int quads = p.part / 4;
    if (g.padded != g.size || p.part % 4 != 0 || quads > 2048) {
        INGOT_CUDA_TRY(ingot_launch_pdl(gated_norm_any_kernel, dim3(n_rows, g.parts), dim3(256), 0, s, p));
        return INGOT_OK;
    }
    auto run = [&](auto kernel, int team) { return ingot_launch_pdl(kernel, dim3(n_rows, (g.parts + 256 / team - 1) / (256 / team)), dim3(256), 0, s, p); };
    INGOT_CUDA_TRY(quads <= 16    ? run(gated_norm_kernel<16, 1>, 16)
                   : quads <= 32  ? run(gated_norm_kernel<32, 1>, 32)
                   : quads <= 128 ? run(gated_norm_kernel<32, 4>, 32)
                   : quads <= 256 ? run(gated_norm_kernel<256, 1>, 256)
                   : quads <= 512 ? run(gated_norm_kernel<256, 2>, 256)
                   : quads <= 1024 ? run(gated_norm_kernel<256, 4>, 256)
                                   : run(gated_norm_kernel<256, 8>, 256));
    return INGOT_OK;
}

}  // extern "C"
