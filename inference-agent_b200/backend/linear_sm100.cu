// Batched projections of CudaBackend::forward_batch on the sm_100a tensor cores:
//   out[t][r] (+)= sum_i W[r][i] * x[t][i]      W f16 [n_out][n_in] (ggml ne = [n_in, n_out]), x and out f32
// — the job of the matmul loops of the CPU reference (src/cpu_backend.cpp:39-42, 71-85 over
// ops::dot_row, src/ops.cpp:127-141) and of Metal's matmul_f16 (src/metal_backend.mm:282-322) for a
// prefill chunk of up to n_batch tokens.
//
// Precision. The reference multiplies f32 activations with widened f16 weights and accumulates in f32, and
// greedy decoding on a random-init model has to reproduce its token choices, so activations are NOT
// rounded to f16: x is split as x = hi + lo with hi = f16(x), lo = f16(x - hi), and every k-step issues two MMAs
// into the same f32 accumulator, hi*W and lo*W. The pair carries 22 significant bits while lo is a normal f16,
// i.e. for |x| above about 2^-4; below that lo falls into the f16 subnormals (spacing 2^-24), so what the split
// guarantees for every x is an ABSOLUTE error of at most 2^-25 per element (relative 3e-5 for an activation
// near 1e-3). The weights are used as stored, the products are exact, the accumulation is f32: the result
// differs from the reference only by summation order and that truncation of x.
//
// bf16 models (ingot_linear_ws_create_bf16). The same kernel on bf16 weights with the activations as one bf16 plane (plain
// bf16 products) or as a hi + lo pair (16 significant bits, for products that feed a recurrence's gates); the number of
// planes is chosen per product. Rows of any length that is a multiple of 8 are accepted (the last k-step is zero-filled
// by TMA), and a matrix may be block-diagonal: output tiles of block b then read the k_block activation columns that
// start at b * k_block.
//
// Grouped products (ingot_grouped_tc_run). One matrix per group of rows - the experts of a mixture - in one launch (up to 512 groups): the
// rows are sorted by group, group g's rows are a run of the activation matrix that starts anywhere, and its matrix is the g-th of a stack.
// CTAs list the groups that have rows from the run starts on the device; boxes that reach into the next run are multiplied along and
// not stored. The activation of an expert is folded into the epilogue, which then writes the bf16 operand of the next product.
//
// Kernels. Up to 64 rows given as a pair of planes: linear_few_kernel; everything else: linear_pair_kernel. Both put the weights on the M
// side of tcgen05.mma (kind::f16) and the rows on its N side, go through their items (output tile, row tile, k slice) persistently, and
// have 6 warps: warp 0 requests [rows][64 k] boxes of weights and planes (128-byte swizzle) with TMA, warp 1 issues the MMAs (all
// lanes walk the loop, one elected lane issues), warps 2-5 read the f32 accumulators out of tensor memory while the next item is
// multiplied. Split-k fills the GPU when there are few tiles; slices go to a scratch and are summed in slice order, by a small kernel or by the
// kernel that consumes the product, so results are reproducible. Rows past n_tok and outputs past n_out are zero-filled by TMA and not stored.
// Every mbarrier wait is bounded; on expiry the CTA raises the workspace's status word and leaves.
#include "grouped_linear.h"
#include "../csrc/sm100_ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

namespace {

using namespace ingot_sm100;

constexpr int kBK = 64;
constexpr int kSweepRows = 2048;  // rows that sweep the weight matrix together (see the tile order of linear_pair_kernel)
constexpr int kBoxBytes = 128 * kBK * 2;        // 16 KB: 128 rows x 64 f16
constexpr int kThreads = 192;
constexpr uint32_t kIdescF16 = 1u << 4;                  // f16 x f16 -> f32, both K-major; M and N are filled in
constexpr uint32_t kIdescBF16 = (1u << 7) | (1u << 10);  // bf16 x bf16 -> f32
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Programmatic dependent launch, as in the attention kernels: every kernel of the batched path lets its successor
// start early (launch_dependents at its top) and waits for its predecessor before it touches anything the predecessor
// wrote; launch latency and per-CTA set-up then overlap the predecessor's tail. INGOT_NO_PDL=1: plain stream order.
#define LINEAR_PDL_TRIGGER() asm volatile("griddepcontrol.launch_dependents;" ::: "memory")
#define LINEAR_PDL_WAIT() asm volatile("griddepcontrol.wait;" ::: "memory")
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    static const bool use_pdl = getenv("INGOT_NO_PDL") == nullptr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// One launch covers up to three weight matrices that read the same activations (q/k/v, gate/up): grid.x runs over
// the token tiles and the output tiles of all of them, tile_end[m] being the running total of tiles up to and including matrix m.
struct GemmParams {
    float* out;           // [n_tok][n_out] (single matrix only)
    float* const* out_at; // linear_few_kernel: where `out` stands instead, in device memory (null: out)
    float* partial[3];    // per matrix: [n_split][n_tok][n_out] when n_split > 1 or to_partial
    int* status;
    int n_tok, k_steps, n_split, accumulate;
    int n_out[3], tile_end[3];
    int tiles_n;
    uint32_t idesc;  // without M and N
    int rows_per_block, k_block, tiles_per_block;  // block-diagonal matrix (rows_per_block > 0, count == 1)
    // grouped: run starts [n_groups + 1] of the rows; out rows are the sorted rows
    const int32_t* group_start;
    int n_groups;
    const float* row_scale;                // epilogue: accumulator * row_scale[row] (null: none), then act
    int act;                               // 1: square of relu, 2: silu(gate) * up (INGOT_ACT_*)
    __nv_bfloat16 *out_hi, *out_lo;        // bf16 plane(s) [rows][n_out] instead of f32
    __half* out_half;                      // f16 instead of f32: row stride half_ld, block b's columns from b * half_block on
    int half_ld, half_block;
    int to_partial;  // write the slice(s) to `partial` even when there is only one (a consumer kernel sums them)
};

__device__ __forceinline__ float silu_of(float g) { return g / (1.0f + expf(-g)); }
__device__ __forceinline__ float gelu_of(float g) { return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))); }  // the tanh form

// ---- few rows ----------------------------------------------------------------------------------------------------------
//
// Products of up to kFewRows rows whose activations are a pair of planes: decoded tokens, short prompts, experts with a few rows each.
// What bounds them is reading the weights once. Tiles of 128 rows give a stage of 16 KB of weights 32 KB for activation rows that are
// mostly padding, so that 64 KB of weights are on their way per SM, and every output tile starts and drains a pipeline of its own.
// Here the weights are the M side of the MMA (128 outputs) and the rows its N side, hi and lo planes side by side (N = 2 x rows padded to
// 8; both halves of the accumulator are added on the way out, which leaves a smaller error than both planes in one: 0.85 of it over
// 2 to 64 rows by 2816 x 2048 to 32768 x 2048, and 4 to 5 % of a step less time than two narrower MMAs): a stage is 16 KB of weights and 256
// bytes per padded row, two CTAs share an SM, and a CTA goes through its share of the items (output tile, k slice, group) with one ring and two accumulators,
// so loads run on across items and into the kernel before (its weights do not depend on it).
// Measured (B200, inside a decoding step, against the 128-row tiles): 16384 x 2048 by 8 rows 13.2 us (17.3 before; 5.1 TB/s), 32768 x 2048
// by 8 rows 22.7 us (35.3; 5.9 TB/s), about 30 experts of 2816 x 2048 with a row each 45 us (84), their 2048 x 1408 down products 27 us (56).
constexpr int kFewRows = 64;  // as many as two CTAs per SM have tensor memory for: 2 accumulators x 2 planes x 64 rows = 256 columns
constexpr int kFewStages = 6, kFewGroups = 512;
constexpr int kFewSmem = 115712;  // half of what an SM has, less what is reserved per CTA
struct FewParams {
    GemmParams g;
    int rows;            // padded rows: of an activation box
    int n_stages, items; // items: the most there can be
    int tmem_cols;       // of one accumulator: a power of two, at least 2 x rows
    uint32_t idesc;
    int off_swap, off_groups, off_bar;  // shared memory behind the ring: up halves on their way to the gate halves, groups with rows
};
struct FewBars {
    uint64_t full[kFewStages], empty[kFewStages], acc_full[2], acc_empty[2];
    uint32_t tmem_base, abort_flag;
    int n_groups;
};

// Barrier of two warps that says whether all their threads passed true.
__device__ __forceinline__ bool pair_all(int barrier, bool v) {
    uint32_t r;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %2, 0;\nbar.red.and.pred p, %1, 64, q;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r) : "r"(barrier), "r"((uint32_t)v) : "memory");
    return r != 0;
}

template <bool kGrouped>
__global__ void __launch_bounds__(kThreads, 2)
linear_few_kernel(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                  const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                  const __grid_constant__ CUtensorMap map_w2, const FewParams fp) {
    const GemmParams& p = fp.g;
    extern __shared__ unsigned char smem_dyn[];
    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char* smem_al = smem_dyn + (smem_base - smem_u32(smem_dyn));
    FewBars* bars = reinterpret_cast<FewBars*>(smem_al + fp.off_bar);
    int* group_list = reinterpret_cast<int*>(smem_al + fp.off_groups);  // {group, first row, end} of the groups that have rows
    volatile uint32_t* abort_flag = &bars->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warp_u = __shfl_sync(0xffffffffu, warp, 0);
    const int n_stages = fp.n_stages, plane_bytes = fp.rows * kBK * 2, stage_bytes = kBoxBytes + 2 * plane_bytes;

    if (threadIdx.x == 0) {
        for (int s = 0; s < n_stages; s++) { mbar_init(smem_u32(&bars->full[s]), 1); mbar_init(smem_u32(&bars->empty[s]), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(smem_u32(&bars->acc_full[b]), 1); mbar_init(smem_u32(&bars->acc_empty[b]), 4); }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(2u * fp.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (kGrouped) {
        LINEAR_PDL_WAIT();  // the runs come from a kernel before
        if (warp == 0) {
            int count = 0;
            for (int g0 = 0; g0 < p.n_groups; g0 += 32) {
                const int mine = g0 + lane;
                const int a = mine < p.n_groups ? p.group_start[mine] : 0, b = mine < p.n_groups ? p.group_start[mine + 1] : 0;
                const unsigned some = __ballot_sync(0xffffffffu, b > a);
                if (b > a) {
                    int* e = group_list + 3 * (count + __popc(some & ((1u << lane) - 1)));
                    e[0] = mine; e[1] = a; e[2] = min(b, a + fp.rows);  // what tensor memory and the exchange have room for
                    if (b - a > fp.rows) atomicOr(p.status, 2);
                }
                count += __popc(some);
            }
            if (lane == 0) bars->n_groups = count;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Only now: a kernel that starts early and shares the SM must find its predecessor's tensor memory taken already.
    LINEAR_PDL_TRIGGER();
    const uint32_t tmem = bars->tmem_base;
    const int n_items = kGrouped ? bars->n_groups * p.tiles_n : fp.items;

    struct Item { int mat, n0, col_end, a_k0, m0, row_end, w_row0, k_begin, n_it, blk, split; };
    auto item_at = [&](int index) {
        Item t;
        const int tile_n = index % p.tiles_n, rest = index / p.tiles_n;  // the k slice, or the group
        t.split = kGrouped ? 0 : rest;
        t.mat = (tile_n >= p.tile_end[0]) + (tile_n >= p.tile_end[1]);
        const int n_out = t.mat == 0 ? p.n_out[0] : t.mat == 1 ? p.n_out[1] : p.n_out[2];
        t.blk = p.tiles_per_block > 0 ? tile_n / p.tiles_per_block : 0;
        t.col_end = p.tiles_per_block > 0 ? (t.blk + 1) * p.rows_per_block : n_out;
        t.a_k0 = t.blk * p.k_block;
        t.n0 = p.tiles_per_block > 0 ? t.blk * p.rows_per_block + (tile_n - t.blk * p.tiles_per_block) * 128
                                     : (tile_n - (t.mat == 0 ? 0 : t.mat == 1 ? p.tile_end[0] : p.tile_end[1])) * 128;
        t.m0 = kGrouped ? group_list[3 * rest + 1] : 0;
        t.row_end = kGrouped ? group_list[3 * rest + 2] : p.n_tok;
        t.w_row0 = kGrouped ? group_list[3 * rest] * n_out + t.n0 : t.n0;
        t.k_begin = (int)((long long)p.k_steps * t.split / p.n_split);
        t.n_it = (int)((long long)p.k_steps * (t.split + 1) / p.n_split) - t.k_begin;
        return t;
    };
    auto map_of_mat = [&](int mat) { return mat == 0 ? &map_w0 : mat == 1 ? &map_w1 : &map_w2; };

    // The weights of the first item that fit the ring are requested before the wait for the kernel before.
    const bool any = (int)blockIdx.x < n_items;
    int n_pre = 0;
    if (warp_u == 0 && any) {
        const Item t = item_at(blockIdx.x);
        n_pre = min(t.n_it, n_stages);
        if (lane == 0)
            for (int it = 0; it < n_pre; it++) {
                const uint32_t full = smem_u32(&bars->full[it]);
                mbar_expect_tx(full, stage_bytes);
                tma_load_2d(smem_base + it * stage_bytes, map_of_mat(t.mat), (t.k_begin + it) * kBK, t.w_row0, full);
            }
    }
    if (!kGrouped) LINEAR_PDL_WAIT();

    if (warp_u == 0) {
        // ---------------- TMA producer ----------------
        int done = 0, s = 0;  // k-steps requested, ring slot
        uint32_t round = 0;
        bool ok = true;
        for (int index = blockIdx.x; index < n_items && ok; index += gridDim.x) {
            const Item t = item_at(index);
            for (int it = 0; it < t.n_it && ok; it++) {
                if (lane == 0) {
                    const uint32_t full = smem_u32(&bars->full[s]), dst = smem_base + s * stage_bytes;
                    const int k = (t.k_begin + it) * kBK;
                    if (done >= n_pre) {
                        ok = mbar_wait(smem_u32(&bars->empty[s]), (round & 1) ^ 1, abort_flag, kWaitLimitNs);
                        if (ok) {
                            mbar_expect_tx(full, stage_bytes);
                            tma_load_2d(dst, map_of_mat(t.mat), k, t.w_row0, full);
                        }
                    }
                    if (ok) {
                        tma_load_2d(dst + kBoxBytes, &map_hi, t.a_k0 + k, t.m0, full);
                        tma_load_2d(dst + kBoxBytes + plane_bytes, &map_lo, t.a_k0 + k, t.m0, full);
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (ok) {
                    done++;
                    if (++s == n_stages) { s = 0; round++; }
                }
            }
        }
        if (!ok && lane == 0) {
            // copies already issued must land before the CTA's shared memory is released
            for (int it = max(0, done - n_stages); it < done; it++) {
                const uint64_t t0 = globaltimer_ns();
                while (!mbar_try_wait(smem_u32(&bars->full[it % n_stages]), (uint32_t)((it / n_stages) & 1)) && globaltimer_ns() - t0 < 100000000ull) {}
            }
        }
    } else if (warp_u == 1) {
        // ---------------- MMA issuer ----------------
        int s = 0, j = 0;
        uint32_t round = 0;
        bool ok = true;
        for (int index = blockIdx.x; index < n_items && ok; index += gridDim.x, j++) {
            const Item t = item_at(index);
            const uint32_t acc = tmem + (uint32_t)((j & 1) * fp.tmem_cols);
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars->acc_empty[j & 1]), (uint32_t)((j >> 1) & 1) ^ 1, abort_flag, kWaitLimitNs)) != 0;
            for (int it = 0; it < t.n_it && ok; it++) {
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars->full[s]), round & 1, abort_flag, kWaitLimitNs)) != 0;
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t a = smem_base + s * stage_bytes, b = a + kBoxBytes;
#pragma unroll
                    for (int ks = 0; ks < kBK / 16; ks++)
                        tc_mma_ss(acc, make_desc(a + ks * 32, 16, 1024), make_desc(b + ks * 32, 16, 1024), fp.idesc, (it > 0 || ks > 0) ? 1u : 0u);
                    tc_commit(smem_u32(&bars->empty[s]));
                    if (it == t.n_it - 1) tc_commit(smem_u32(&bars->acc_full[j & 1]));
                }
                __syncwarp();
                if (++s == n_stages) { s = 0; round++; }
            }
        }
    } else {
        // ---------------- epilogue: one thread per output, eight rows at a time ----------------
        const int lg = warp & 3;  // the tensor-memory lane group this warp may read
        float* const swap = reinterpret_cast<float*>(smem_al + fp.off_swap) + (lg >> 1) * fp.rows * 32;  // [row][32] of a gate / up pair of warps
        const bool split_k = p.n_split > 1 || p.to_partial;
        float* const out = !kGrouped && p.out_at ? *p.out_at : p.out;
        int j = 0;
        bool ok = true;
        for (int index = blockIdx.x; index < n_items && ok; index += gridDim.x, j++) {
            const Item t = item_at(index);
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars->acc_full[j & 1]), (uint32_t)((j >> 1) & 1), abort_flag, kWaitLimitNs)) != 0;
            if (kGrouped && p.act == 2) ok = pair_all(1 + (lg >> 1), ok);  // they go on, or leave, together
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)((j & 1) * fp.tmem_cols) + ((uint32_t)(lg * 32) << 16);
            const int n_out = t.mat == 0 ? p.n_out[0] : t.mat == 1 ? p.n_out[1] : p.n_out[2];
            const int col = t.n0 + lg * 32 + lane, n_rows = t.row_end - t.m0;
            auto read = [&](int c, float (&v)[8]) {  // rows c .. c + 7 of this thread's output
                float lo[8];
                tmem_ld8(acc + c, v);
                tmem_ld8(acc + fp.rows + c, lo);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] += lo[i];
            };
            auto put_pair = [&](size_t at, float x) {
                const __nv_bfloat16 h = __float2bfloat16_rn(x);
                p.out_hi[at] = h;
                if (p.out_lo) p.out_lo[at] = __float2bfloat16_rn(x - __bfloat162float(h));
            };
            if (kGrouped && p.act == 2) {
                // runs of 32 gate outputs, each followed by the 32 up outputs that go with them: one warp's lanes and the next one's
                if (lg & 1)
                    for (int c = 0; c < n_rows; c += 8) {
                        float v[8];
                        read(c, v);
#pragma unroll
                        for (int i = 0; i < 8; i++)
                            if (c + i < n_rows) swap[(c + i) * 32 + lane] = v[i];
                    }
                asm volatile("bar.sync %0, 64;" ::"r"(1 + (lg >> 1)) : "memory");
                if (!(lg & 1) && col < t.col_end) {
                    const int half_out = n_out / 2, out_col = t.n0 / 2 + (lg >> 1) * 32 + lane;
                    for (int c = 0; c < n_rows; c += 8) {
                        float v[8];
                        read(c, v);
#pragma unroll
                        for (int i = 0; i < 8; i++)
                            if (c + i < n_rows) {
                                const int row = t.m0 + c + i;
                                put_pair((size_t)row * half_out + out_col, silu_of(v[i]) * swap[(c + i) * 32 + lane] * (p.row_scale ? p.row_scale[row] : 1.0f));
                            }
                    }
                }
                asm volatile("bar.sync %0, 64;" ::"r"(1 + (lg >> 1)) : "memory");
            } else {
                float* const part = t.mat == 0 ? p.partial[0] : t.mat == 1 ? p.partial[1] : p.partial[2];
                float* const dst = (split_k ? part + (size_t)t.split * p.n_tok * n_out : out) + col;
                for (int c = 0; c < n_rows; c += 8) {
                    float v[8];
                    __syncwarp();  // lanes past the last output have left the round before early; tensor memory is read by whole warps
                    read(c, v);
                    if (col >= t.col_end) continue;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if (c + i >= n_rows) break;
                        const int row = t.m0 + c + i;
                        float x = v[i];
                        if (kGrouped) {
                            if (p.row_scale) x *= p.row_scale[row];
                            if (p.act == 1) x = x > 0.f ? x * x : 0.f;
                        }
                        if (kGrouped && p.out_hi) {
                            put_pair((size_t)row * n_out + col, x);
                        } else if (!kGrouped && p.out_half) {
                            p.out_half[(size_t)row * p.half_ld + t.blk * p.half_block + (col - t.blk * p.rows_per_block)] = __float2half_rn(fminf(fmaxf(x, -65504.f), 65504.f));
                        } else {
                            float* const d = dst + (size_t)row * n_out;
                            *d = !split_k && p.accumulate ? *d + x : x;
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->acc_empty[j & 1]));
        }
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicOr(p.status, 1);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * fp.tmem_cols) : "memory");
    }
}

// ---- many rows ---------------------------------------------------------------------------------------------------------
//
// Products of more rows (or of one plane). Bound by the tensor cores, once tiles are loaded often enough from L2 and the accumulators are
// emptied while the next tile is multiplied. Two CTAs of a cluster form a tile of 256 outputs (the M side: 128 of each CTA) by up to
// 256 rows (the N side: each CTA fetches half of them, both multiply with all), so 32 KB per SM and k-step feed 512 cycles of
// MMA, two thirds of what a 128 x 256 tile of one CTA takes. The pair goes through its share of the items (output tile, row tile, k slice) with a
// 6-stage ring and two accumulators. Rows per tile are the launch's choice (any multiple of 32; a group's rows are spread evenly over its tiles),
// so that little is multiplied for padding. A lane holds an output, so that a warp writes whole lines of a row.
// Measured (B200, inside a prompt's step, against one-CTA tiles of 128 x 256 that each start, drain and write on their own): 4096 rows by
// 28672 x 4096 603 us (807 before; 1595 TFLOP/s), by 4096 x 14336 322 us (376), by 10240 x 4096 210 us (312).
constexpr int kPairStages = 6, kPairRows = 256, kPairGroups = 512;
constexpr int kPairStageBytes = 2 * kBoxBytes;                       // W, and the activation rows of all planes
constexpr int kPairThreads = 320;                                    // 8 warps of epilogue: with 4, gated products of short rows waited for them
constexpr int kPairSwapBytes = 2 * 4 * 2 * 8 * 32 * 4;               // halves of gate / up columns on their way: [buffer][warp pair][from][8 rows][32 outputs]
struct PairParams {
    GemmParams g;
    int rows, planes;     // rows of a tile at most (grouped: 256 / planes)
    int row_tiles, items; // plain products
    int box_bytes;        // of one plane's activation box
    uint32_t idesc;       // without N
};
struct PairBars {
    uint64_t full[kPairStages], empty[kPairStages], acc_full[2], acc_empty[2];
    uint32_t tmem_base, abort_flag;
    int n_groups, n_items;
};
constexpr int kPairOffSwap = kPairStages * kPairStageBytes, kPairOffBar = kPairOffSwap + kPairSwapBytes, kPairOffGroups = kPairOffBar + 256;
constexpr int kPairSmem = kPairOffGroups + kPairGroups * 16 + 1024;  // groups: {group, first row, end, first item}
static_assert(sizeof(PairBars) <= 256 && kPairSmem <= 227 * 1024, "shared memory");

template <bool kGrouped>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
linear_pair_kernel(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                   const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                   const __grid_constant__ CUtensorMap map_w2, const PairParams pp) {
    const GemmParams& p = pp.g;
    extern __shared__ unsigned char smem_dyn[];
    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char* smem_al = smem_dyn + (smem_base - smem_u32(smem_dyn));
    PairBars* bars = reinterpret_cast<PairBars*>(smem_al + kPairOffBar);
    int4* groups = reinterpret_cast<int4*>(smem_al + kPairOffGroups);
    volatile uint32_t* abort_flag = &bars->abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warp_u = __shfl_sync(0xffffffffu, warp, 0);
    const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPairStages; s++) { mbar_init(smem_u32(&bars->full[s]), 1); mbar_init(smem_u32(&bars->empty[s]), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(smem_u32(&bars->acc_full[b]), 1); mbar_init(smem_u32(&bars->acc_empty[b]), 16); }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (kGrouped) {
        LINEAR_PDL_WAIT();  // the runs come from a kernel before
        if (warp == 0) {
            int count = 0, items = 0;
            for (int g0 = 0; g0 < p.n_groups; g0 += 32) {
                const int mine = g0 + lane;
                const int a = mine < p.n_groups ? p.group_start[mine] : 0, b = mine < p.n_groups ? p.group_start[mine + 1] : 0;
                const int n = (b - a + pp.rows - 1) / pp.rows * p.tiles_n;
                const unsigned some = __ballot_sync(0xffffffffu, b > a);
                int upto = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += v;
                }
                if (b > a) groups[count + __popc(some & ((1u << lane) - 1))] = make_int4(mine, a, b, items + upto - n);
                count += __popc(some);
                items += __shfl_sync(0xffffffffu, upto, 31);
            }
            if (lane == 0) { bars->n_groups = count; bars->n_items = items; }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the peer's barriers are there before anything is counted on them
    tc_fence_after();
    LINEAR_PDL_TRIGGER();  // tensor memory is held
    const uint32_t tmem = bars->tmem_base;
    const int n_items = kGrouped ? bars->n_items : pp.items;

    struct Item { int mat, n0, col_end, a_k0, m0, n_rows, mma_rows, w_row0, k_begin, n_it, blk, split; };
    auto item_at = [&](int index) {
        Item t;
        int tile_n, row_end;
        t.split = 0;
        if (kGrouped) {
            int lo = 0, hi = bars->n_groups - 1;  // the last group whose first item is not behind this one
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (groups[mid].w <= index) lo = mid; else hi = mid - 1;
            }
            const int4 e = groups[lo];
            const int tiles = (e.z - e.y + pp.rows - 1) / pp.rows, per = ((e.z - e.y + tiles - 1) / tiles + 31) & ~31, local = index - e.w;
            tile_n = local / tiles;  // row tiles of a group side by side: they share the weights
            t.m0 = e.y + (local - tile_n * tiles) * per;
            t.n_rows = min(per, e.z - t.m0);  // may be none: rows rounded up
            t.w_row0 = e.x * p.n_out[0];
        } else {
            const int tiles = p.tiles_n * pp.row_tiles, per_group = max(1, kSweepRows / pp.rows);
            t.split = index / tiles;
            // row tiles of about 2048 rows sweep the outputs together: what runs at a time shares weights and rows in L2
            const int local = index - t.split * tiles, grp = local / (per_group * p.tiles_n), in = local - grp * per_group * p.tiles_n;
            const int n_m = min(per_group, pp.row_tiles - grp * per_group);
            tile_n = in / n_m;
            t.m0 = (grp * per_group + in - tile_n * n_m) * pp.rows;
            row_end = p.n_tok;
            t.n_rows = min(pp.rows, row_end - t.m0);
            t.w_row0 = 0;
        }
        t.mma_rows = max(32, (t.n_rows + 31) & ~31);
        t.mat = (tile_n >= p.tile_end[0]) + (tile_n >= p.tile_end[1]);
        const int n_out = t.mat == 0 ? p.n_out[0] : t.mat == 1 ? p.n_out[1] : p.n_out[2];
        t.blk = p.tiles_per_block > 0 ? tile_n / p.tiles_per_block : 0;
        t.col_end = p.tiles_per_block > 0 ? (t.blk + 1) * p.rows_per_block : n_out;
        t.a_k0 = t.blk * p.k_block;
        t.n0 = (p.tiles_per_block > 0 ? t.blk * p.rows_per_block + (tile_n - t.blk * p.tiles_per_block) * 256
                                      : (tile_n - (t.mat == 0 ? 0 : t.mat == 1 ? p.tile_end[0] : p.tile_end[1])) * 256) + rank * 128;  // of this CTA
        t.w_row0 += t.n0;
        t.k_begin = (int)((long long)p.k_steps * t.split / p.n_split);
        t.n_it = (int)((long long)p.k_steps * (t.split + 1) / p.n_split) - t.k_begin;
        return t;
    };
    auto map_of_mat = [&](int mat) { return mat == 0 ? &map_w0 : mat == 1 ? &map_w1 : &map_w2; };
    const uint32_t stage_tx = 2 * (kBoxBytes + pp.planes * pp.box_bytes);  // of both CTAs, counted on the first one's barrier

    int n_pre = 0;
    if (warp_u == 0 && pair < n_items) {  // weights do not depend on the kernel before
        const Item t = item_at(pair);
        n_pre = min(t.n_it, kPairStages);
        if (lane == 0)
            for (int it = 0; it < n_pre; it++) {
                if (rank == 0) mbar_expect_tx(smem_u32(&bars->full[it]), stage_tx);
                tma_load_2d_pair(smem_base + it * kPairStageBytes, map_of_mat(t.mat), (t.k_begin + it) * kBK, t.w_row0, map_to_rank(smem_u32(&bars->full[it]), 0));
            }
    }
    if (!kGrouped) LINEAR_PDL_WAIT();

    if (warp_u == 0) {
        // ---------------- TMA producer of this CTA's halves ----------------
        int done = 0, s = 0;
        uint32_t round = 0;
        bool ok = true;
        for (int index = pair; index < n_items && ok; index += n_pairs) {
            const Item t = item_at(index);
            const int row = t.m0 + rank * (t.mma_rows >> 1);
            for (int it = 0; it < t.n_it && ok; it++) {
                if (lane == 0) {
                    const uint32_t full = map_to_rank(smem_u32(&bars->full[s]), 0), dst = smem_base + s * kPairStageBytes;
                    const int k = (t.k_begin + it) * kBK;
                    if (done >= n_pre) {
                        ok = mbar_wait(smem_u32(&bars->empty[s]), (round & 1) ^ 1, abort_flag, kWaitLimitNs);
                        if (ok) {
                            if (rank == 0) mbar_expect_tx(smem_u32(&bars->full[s]), stage_tx);
                            tma_load_2d_pair(dst, map_of_mat(t.mat), k, t.w_row0, full);
                        }
                    }
                    if (ok) {
                        tma_load_2d_pair(dst + kBoxBytes, &map_hi, t.a_k0 + k, row, full);
                        if (pp.planes > 1) tma_load_2d_pair(dst + kBoxBytes + (kBoxBytes >> 1), &map_lo, t.a_k0 + k, row, full);
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (ok) {
                    done++;
                    if (++s == kPairStages) { s = 0; round++; }
                }
            }
        }
        // the last arrivals on this CTA's barriers come from the first one's MMAs: they must be over before it leaves
        for (int i = 0; i < kPairStages && ok && lane == 0; i++) {
            ok = mbar_wait(smem_u32(&bars->empty[s]), (round & 1) ^ 1, abort_flag, kWaitLimitNs);
            if (++s == kPairStages) { s = 0; round++; }
        }
        if (!ok && lane == 0) {  // copies already issued must land before the CTA's shared memory is released
            const uint64_t t0 = globaltimer_ns();
            while (globaltimer_ns() - t0 < 100000000ull) {}
        }
    } else if (warp_u == 1 && rank == 0) {
        // ---------------- MMA issuer, for both ----------------
        int s = 0, j = 0;
        uint32_t round = 0;
        bool ok = true;
        for (int index = pair; index < n_items && ok; index += n_pairs, j++) {
            const Item t = item_at(index);
            const uint32_t acc = tmem + (uint32_t)((j & 1) * kPairRows), idesc = pp.idesc | ((uint32_t)(t.mma_rows >> 3) << 17);
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars->acc_empty[j & 1]), (uint32_t)((j >> 1) & 1) ^ 1, abort_flag, kWaitLimitNs)) != 0;
            tc_fence_after();
            for (int it = 0; it < t.n_it && ok; it++) {
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars->full[s]), round & 1, abort_flag, kWaitLimitNs)) != 0;
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t a = smem_base + s * kPairStageBytes, b = a + kBoxBytes;
#pragma unroll
                    for (int ks = 0; ks < kBK / 16; ks++)
                        tc_mma_pair(acc, make_desc(a + ks * 32, 16, 1024), make_desc(b + ks * 32, 16, 1024), idesc, (it > 0 || ks > 0) ? 1u : 0u);
                    if (pp.planes > 1) {
#pragma unroll
                        for (int ks = 0; ks < kBK / 16; ks++)
                            tc_mma_pair(acc, make_desc(a + ks * 32, 16, 1024), make_desc(b + (kBoxBytes >> 1) + ks * 32, 16, 1024), idesc, 1u);
                    }
                    tc_commit_pair(smem_u32(&bars->empty[s]));
                    if (it == t.n_it - 1) tc_commit_pair(smem_u32(&bars->acc_full[j & 1]));
                }
                __syncwarp();
                if (++s == kPairStages) { s = 0; round++; }
            }
        }
    } else if (warp_u >= 2) {
        // ---------------- epilogue: one thread per output, two warps for the same outputs and every second run of rows ----------------
        const int lg = warp & 3;  // the tensor-memory lane group this warp may read
        const int half = (warp - 2) >> 2, duo = 2 * half + (lg >> 1);  // duo: the warps of neighbouring outputs
        const bool split_k = p.n_split > 1 || p.to_partial;
        int j = 0;
        bool ok = true;
        for (int index = pair; index < n_items && ok; index += n_pairs, j++) {
            const Item t = item_at(index);
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars->acc_full[j & 1]), (uint32_t)((j >> 1) & 1), abort_flag, kWaitLimitNs)) != 0;
            if (p.act >= 2) ok = pair_all(1 + duo, ok);  // they go on, or leave, together
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)((j & 1) * kPairRows) + ((uint32_t)(lg * 32) << 16);
            const int n_out = t.mat == 0 ? p.n_out[0] : t.mat == 1 ? p.n_out[1] : p.n_out[2];
            const int col = t.n0 + lg * 32 + lane;
            // As soon as the last values are in registers. A release of the stores before it would wait for them at every item.
            bool drained = false;
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster_relaxed(map_to_rank(smem_u32(&bars->acc_empty[j & 1]), 0));
                drained = true;
            };
            auto put_pair = [&](size_t at, float x) {
                const __nv_bfloat16 h = __float2bfloat16_rn(x);
                p.out_hi[at] = h;
                if (p.out_lo) p.out_lo[at] = __float2bfloat16_rn(x - __bfloat162float(h));
            };
            if (p.act >= 2) {
                // Runs of 32 gate outputs, each followed by the 32 up outputs that go with them: one warp's lanes and the next one's. Of 16
                // rows each warp finishes 8: it hands the other half of its own values over.
                const bool is_up = lg & 1;
                const int half_out = n_out / 2, out_col = t.n0 / 2 + (lg >> 1) * 32 + lane;
                for (int c = half * 16, buffer = 0; c < t.n_rows; c += 32, buffer ^= 1) {
                    float v[16], x[8];
                    __syncwarp();
                    tmem_ld16(acc + c, v);
                    tmem_wait_ld();
                    if (c + 32 >= t.n_rows) release();
                    float* const swap = reinterpret_cast<float*>(smem_al + kPairOffSwap) + (buffer * 4 + duo) * 512;
#pragma unroll
                    for (int i = 0; i < 8; i++) swap[is_up * 256 + i * 32 + lane] = is_up ? v[i] : v[8 + i];
                    asm volatile("bar.sync %0, 64;" ::"r"(1 + duo) : "memory");
                    if (col >= t.col_end) continue;
                    const int row = t.m0 + c + (is_up ? 8 : 0), n = t.m0 + t.n_rows - row;
                    auto gated = [&](auto act) {
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const float other = swap[!is_up * 256 + i * 32 + lane], gate = is_up ? other : v[i], up = is_up ? v[8 + i] : other;
                            x[i] = act(gate) * up;
                        }
                    };
                    if (kGrouped || p.act == 2) gated([](float g) { return silu_of(g); });
                    else gated([](float g) { return gelu_of(g); });
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (i < n) put_pair((size_t)(row + i) * half_out + out_col, p.row_scale ? x[i] * p.row_scale[row + i] : x[i]);
                }
            } else {
                float* const part = t.mat == 0 ? p.partial[0] : t.mat == 1 ? p.partial[1] : p.partial[2];
                float* const dst = (split_k ? part + (size_t)t.split * p.n_tok * n_out : p.out) + col;
                for (int c = half * 32; c < t.n_rows; c += 64) {
                    float v[32];
                    __syncwarp();  // as above: lanes past the last output
                    tmem_ld32(acc + c, v);
                    tmem_wait_ld();
                    if (c + 64 >= t.n_rows) release();
                    if (col >= t.col_end) continue;
                    const int n = t.n_rows - c;
                    if (!kGrouped && n >= 32 && !p.out_half && (split_k || !p.accumulate)) {  // plain rows: no conditions in between
                        float* d = dst + (size_t)(t.m0 + c) * n_out;
#pragma unroll
                        for (int i = 0; i < 32; i++, d += n_out) *d = v[i];
                        continue;
                    }
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        if (i >= n) break;
                        const int row = t.m0 + c + i;
                        float x = v[i];
                        if (kGrouped) {
                            if (p.row_scale) x *= p.row_scale[row];
                            if (p.act == 1) x = x > 0.f ? x * x : 0.f;
                        }
                        if (kGrouped && p.out_hi) {
                            put_pair((size_t)row * n_out + col, x);
                        } else if (!kGrouped && p.out_half) {
                            p.out_half[(size_t)row * p.half_ld + t.blk * p.half_block + (col - t.blk * p.rows_per_block)] = __float2half_rn(fminf(fmaxf(x, -65504.f), 65504.f));
                        } else {
                            float* const d = dst + (size_t)row * n_out;
                            *d = !split_k && p.accumulate ? *d + x : x;
                        }
                    }
                }
            }
            if (!drained) release();
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync();  // neither leaves while the other may still count on its barriers or multiply from its shared memory
    if (threadIdx.x == 0 && *abort_flag) atomicOr(p.status, 1);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// out (+)= sum over the k slices, in slice order
__global__ void splitk_reduce_kernel(float* out, const float* partial, int n_split, size_t n, int accumulate) {
    LINEAR_PDL_TRIGGER();
    LINEAR_PDL_WAIT();
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    float4 acc = accumulate ? *reinterpret_cast<const float4*>(out + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < n_split; s++) {
        const float4 v = *reinterpret_cast<const float4*>(partial + (size_t)s * n + i);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    *reinterpret_cast<float4*>(out + i) = acc;
}

// How f32 activations become MMA operands: an f16 pair hi = f16(x), lo = f16(x - hi), one bf16 plane, or a bf16 pair.
enum : int { kActF16Pair = 0, kActBF16 = 1, kActBF16Pair = 2 };
template <int kAct>
__device__ __forceinline__ void store_split4(__half* hi, __half* lo, size_t i, const float (&f)[4]) {
    if (kAct == kActF16Pair) {
        __half h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            h[e] = __float2half_rn(f[e]);
            l[e] = __float2half_rn(f[e] - __half2float(h[e]));
        }
        *reinterpret_cast<uint2*>(hi + i) = *reinterpret_cast<const uint2*>(h);
        *reinterpret_cast<uint2*>(lo + i) = *reinterpret_cast<const uint2*>(l);
    } else {
        __nv_bfloat16 h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            h[e] = __float2bfloat16_rn(f[e]);
            l[e] = __float2bfloat16_rn(f[e] - __bfloat162float(h[e]));
        }
        *reinterpret_cast<uint2*>(hi + i) = *reinterpret_cast<const uint2*>(h);
        if (kAct == kActBF16Pair) *reinterpret_cast<uint2*>(lo + i) = *reinterpret_cast<const uint2*>(l);
    }
}

// x rows are x_ld floats apart, the planes' rows n; grid.y = row
template <int kAct>
__global__ void split_act_kernel(__half* hi, __half* lo, const float* x, int x_ld, int n) {
    LINEAR_PDL_TRIGGER();
    LINEAR_PDL_WAIT();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    const float4 v = *reinterpret_cast<const float4*>(x + (size_t)blockIdx.y * x_ld + i);
    const float f[4] = {v.x, v.y, v.z, v.w};
    store_split4<kAct>(hi, lo, (size_t)blockIdx.y * n + i, f);
}

// hi/lo of rmsnorm(x) = x * rsqrt(mean(x^2) + eps) * w, one CTA per token row (ops::rmsnorm, src/ops.cpp:227-232,
// with the same expression order as the standalone norm kernel, so the split sees the same f32 values).
// The mean is taken over n_mean of the row's n floats (rows zero-padded to an aligned length).
template <int kAct>
__global__ void rmsnorm_split_kernel(__half* hi, __half* lo, const float* x, const float* w, int n, int n_mean, float eps) {
    LINEAR_PDL_TRIGGER();
    LINEAR_PDL_WAIT();
    __shared__ float red[32];
    const float* xr = x + (size_t)blockIdx.x * n;
    constexpr int kKeep = 4;  // float4s of the row a thread keeps between the two passes
    float4 kept[kKeep];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        kept[k] = i < n ? *reinterpret_cast<const float4*>(xr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < kKeep; k++) { ss += kept[k].x * kept[k].x; ss += kept[k].y * kept[k].y; ss += kept[k].z * kept[k].z; ss += kept[k].w * kept[k].w; }
    for (int i = (threadIdx.x + kKeep * blockDim.x) * 4; i < n; i += blockDim.x * 4) {
        const float4 v = *reinterpret_cast<const float4*>(xr + i);
        ss += v.x * v.x; ss += v.y * v.y; ss += v.z * v.z; ss += v.w * v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) red[0] = 1.0f / sqrtf(v / float(n_mean) + eps);
    }
    __syncthreads();
    const float scale = red[0];
    auto put = [&](int i, const float4& v) {
        const float4 g = *reinterpret_cast<const float4*>(w + i);
        const float f[4] = {v.x * scale * g.x, v.y * scale * g.y, v.z * scale * g.z, v.w * scale * g.w};
        store_split4<kAct>(hi, lo, (size_t)blockIdx.x * n + i, f);
    };
#pragma unroll
    for (int k = 0; k < kKeep; k++) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        if (i < n) put(i, kept[k]);
    }
    for (int i = (threadIdx.x + kKeep * blockDim.x) * 4; i < n; i += blockDim.x * 4) put(i, *reinterpret_cast<const float4*>(xr + i));
}

// Consumers of k-slice partials [n_split][n_tok][n_out]: the sum over slices (always in slice order) is folded into
// the kernel that needs the result, so a split-k GEMM costs no reduction launch of its own.
struct Slices {
    const float* base;
    int n_split;
};
__device__ __forceinline__ float4 sum_slices(const Slices& p, size_t idx, size_t slice_elems, float4 acc) {
    for (int sl = 0; sl < p.n_split; sl++) {
        const float4 v = *reinterpret_cast<const float4*>(p.base + sl * slice_elems + idx);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    return acc;
}

// Up to three plain outputs (q, k, v): out_m = sum of its slices. grid.y selects the output.
struct FinishGroup {
    Slices in[3];
    float* out[3];
    int n_out[3];
};
__global__ void finish_group_kernel(const FinishGroup g, int n_tok) {
    LINEAR_PDL_TRIGGER();
    LINEAR_PDL_WAIT();
    const int m = blockIdx.y;
    const Slices in = m == 0 ? g.in[0] : m == 1 ? g.in[1] : g.in[2];
    float* out = m == 0 ? g.out[0] : m == 1 ? g.out[1] : g.out[2];
    const size_t n = (size_t)n_tok * (m == 0 ? g.n_out[0] : m == 1 ? g.n_out[1] : g.n_out[2]);
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    *reinterpret_cast<float4*>(out + i) = sum_slices(in, i, n, make_float4(0.f, 0.f, 0.f, 0.f));
}

// x[t][:] += sum of slices (the residual add of wo / down), then, if norm_w is given, hi/lo of rmsnorm(x[t]) for the
// next projections. One CTA per token.
// pair_rows (may be null): rows of another branch that go into the sum, token t's at row_of[t * top + k] (row_of null: t).
template <int kAct>
__global__ void finish_residual_norm_kernel(float* x, const Slices in, __half* hi, __half* lo, const float* norm_w, int n, int n_mean, int n_tok,
                                            float eps, const float* pair_rows, const int32_t* row_of, int top) {
    __shared__ float red[32];
    LINEAR_PDL_TRIGGER();
    LINEAR_PDL_WAIT();
    const size_t row = (size_t)blockIdx.x * n;
    const size_t slice = (size_t)n_tok * n;
    float ss = 0.f;
    for (int i = threadIdx.x * 4; i < n; i += blockDim.x * 4) {
        float4 v = sum_slices(in, row + i, slice, *reinterpret_cast<const float4*>(x + row + i));
        for (int k = 0; k < top; k++) {
            const float4 a = *reinterpret_cast<const float4*>(pair_rows + (row_of ? (size_t)row_of[blockIdx.x * top + k] : (size_t)blockIdx.x) * n + i);
            v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
        }
        *reinterpret_cast<float4*>(x + row + i) = v;
        ss += v.x * v.x; ss += v.y * v.y; ss += v.z * v.z; ss += v.w * v.w;
    }
    if (norm_w == nullptr) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) red[0] = 1.0f / sqrtf(v / float(n_mean) + eps);
    }
    __syncthreads();
    const float scale = red[0];
    for (int i = threadIdx.x * 4; i < n; i += blockDim.x * 4) {
        const float4 v = *reinterpret_cast<const float4*>(x + row + i), g = *reinterpret_cast<const float4*>(norm_w + i);
        const float f[4] = {v.x * scale * g.x, v.y * scale * g.y, v.z * scale * g.z, v.w * scale * g.w};
        store_split4<kAct>(hi, lo, row + i, f);
    }
}

// hi/lo of silu(sum of gate slices) * (sum of up slices)
__global__ void finish_swiglu_kernel(__half* hi, __half* lo, const Slices gate, const Slices up, size_t n) {
    LINEAR_PDL_TRIGGER();
    LINEAR_PDL_WAIT();
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 g = sum_slices(gate, i, n, z), u = sum_slices(up, i, n, z);
    const float f[4] = {g.x / (1.0f + expf(-g.x)) * u.x, g.y / (1.0f + expf(-g.y)) * u.y, g.z / (1.0f + expf(-g.z)) * u.z,
                        g.w / (1.0f + expf(-g.w)) * u.w};
    store_split4<kActF16Pair>(hi, lo, i, f);
}

// One or two bf16 planes of act(gate) * up, where one product of width 2 n holds both as runs of 32 gate columns, each followed by the 32
// up columns that go with them.
// act: 0 silu, 1 the tanh form of gelu. grid.y = row.
template <int kAct>
__global__ void finish_gated_kernel(__half* hi, __half* lo, const Slices in, int n, size_t slice, int act) {
    LINEAR_PDL_TRIGGER();
    LINEAR_PDL_WAIT();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    const size_t row = (size_t)blockIdx.y * 2 * n;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const int at = (i & ~31) * 2 + (i & 31);
    const float4 g = sum_slices(in, row + at, slice, z), u = sum_slices(in, row + at + 32, slice, z);
    const float gv[4] = {g.x, g.y, g.z, g.w}, uv[4] = {u.x, u.y, u.z, u.w};
    float f[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float t = gv[e];
        f[e] = (act == 0 ? silu_of(t) : gelu_of(t)) * uv[e];
    }
    store_split4<kAct>(hi, lo, (size_t)blockIdx.y * n + i, f);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    });
    return fn;
}

// f16 or bf16 matrix [rows][cols] row-major, boxes of box_rows rows x 64 columns, 128-byte swizzle, zero fill outside
bool make_map(CUtensorMap* map, const void* base, int rows, int cols, int box_rows = 128, bool bf16 = false) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The launch of linear_few_kernel: `rows` padded rows per activation box, `items` at most.
template <bool kGrouped>
cudaError_t launch_few(const GemmParams& g, int rows, int items, int num_sms, const CUtensorMap& hi, const CUtensorMap& lo, const CUtensorMap* const* w, cudaStream_t s) {
    FewParams p = {};
    p.g = g;
    p.rows = rows;
    p.items = items;
    p.tmem_cols = 16;  // two of them: at least 32 columns, a power of two
    while (p.tmem_cols < 2 * rows) p.tmem_cols *= 2;
    p.idesc = g.idesc | ((uint32_t)(2 * rows >> 3) << 17) | ((128u >> 4) << 24);
    const int stage = kBoxBytes + 2 * rows * kBK * 2, swap = kGrouped && g.act == 2 ? 2 * rows * 32 * 4 : 0, list = kGrouped ? 3 * 4 * std::min(g.n_groups, g.n_tok) : 0;
    const int fixed = 1024 + swap + (list + 15) / 16 * 16 + (int)sizeof(FewBars);
    p.n_stages = std::min(kFewStages, (kFewSmem - fixed) / stage);
    p.off_swap = p.n_stages * stage;
    p.off_groups = p.off_swap + swap;
    p.off_bar = p.off_groups + (list + 15) / 16 * 16;
    return launch_pdl(linear_few_kernel<kGrouped>, dim3(std::min(items, 2 * num_sms)), dim3(kThreads), (size_t)kFewSmem, s, hi, lo, *w[0], *w[1], *w[2], p);
}

// The launch of linear_pair_kernel with tiles of up to `rows` rows; `items` at most.
template <bool kGrouped>
cudaError_t launch_pair(const GemmParams& g, int rows, int planes, int box_rows, int row_tiles, int items, int num_sms, const CUtensorMap& hi, const CUtensorMap& lo,
                        const CUtensorMap* const* w, cudaStream_t s) {
    PairParams p = {};
    p.g = g;
    p.rows = rows;
    p.planes = planes;
    p.row_tiles = row_tiles;
    p.items = items;
    p.box_bytes = box_rows * kBK * 2;
    p.idesc = g.idesc | ((256u >> 4) << 24);
    return launch_pdl(linear_pair_kernel<kGrouped>, dim3(2 * std::min(items, num_sms / 2)), dim3(kPairThreads), (size_t)kPairSmem, s, hi, lo, *w[0], *w[1], *w[2], p);
}

// k slices of a product of `tiles` blocks of 128 outputs by 128 rows: enough to give every SM a block, at least 4 k-steps each. The last bits of a
// product depend on its slices, and what follows rounds them to 16 bits: the number depends on nothing but the product's size and the SMs,
// so that other tiles or another kernel leave a model's results as they are.
int k_slices(long long tiles, int k_steps, int most, int num_sms) {
    return (int)std::max(1ll, std::min({num_sms / tiles, (long long)k_steps / 4, (long long)most}));
}
long long blocks_of(int n) { return (n + 127) / 128; }

// Rows of a tile for n_tok rows against tiles_n tiles of 256 outputs in n_split slices: the least rounds of all pairs of CTAs times what one costs.
// A k-step takes a pair as long as it takes to load it, about as 256 + rows (at 256 rows that is 512 cycles, what the MMAs take), and a
// tile starts and ends for about four k-steps.
struct PairTiles { int rows, row_tiles; };
PairTiles pair_tiles(int n_tok, int tiles_n, int planes, int k_steps, int n_split, int num_sms) {
    const int pairs = num_sms / 2;
    PairTiles best = {};
    long long least = 0;
    for (int rows = kPairRows / planes; rows >= 32; rows -= 32) {
        const int row_tiles = (n_tok + rows - 1) / rows;
        const long long items = (long long)tiles_n * row_tiles * n_split, rounds = (items + pairs - 1) / pairs;
        const long long cost = rounds * ((k_steps + n_split - 1) / n_split + 4) * (256 + rows * planes);
        if (best.rows == 0 || cost < least) { best = {rows, row_tiles}; least = cost; }
    }
    return best;
}

}  // namespace

struct ingot_linear_ws {
    __half* hi = nullptr;
    __half* lo = nullptr;
    float* partial = nullptr;
    int* status = nullptr;
    size_t act_elems = 0, partial_floats = 0;  // partial_floats: per slot; kSlots slots
    int slot_split[3] = {0, 0, 0};             // slices the last GEMM into each slot produced
    int slot_out[3] = {0, 0, 0};               // and its output width
    int num_sms = 0;
    bool bf16 = false;
    int n_slots = 3;
    int planes = 2;                            // of the prepared activations
    int prepared_tok = 0, prepared_in = 0;
    std::map<std::tuple<const void*, int, int, int>, CUtensorMap> maps;  // of weight matrices and activations, by place, shape and box
};

// The map of an activation or weight buffer, made once. At most kMaxMaps are kept: make_room() before a launch looks up its own.
static constexpr size_t kMaxMaps = 65536;
static void make_room(ingot_linear_ws* ws) {
    if (ws->maps.size() > kMaxMaps) ws->maps.clear();
}
static const CUtensorMap* map_of(ingot_linear_ws* ws, const void* base, int rows, int cols, int box, bool bf16) {
    const auto key = std::make_tuple(base, rows, cols, box);
    auto it = ws->maps.find(key);
    if (it == ws->maps.end()) {
        CUtensorMap tm;
        if (!make_map(&tm, base, rows, cols, box, bf16)) return nullptr;
        it = ws->maps.emplace(key, tm).first;
    }
    return &it->second;
}

static cudaError_t set_prepared(ingot_linear_ws* ws, int n_in, int n_tok) {
    ws->prepared_tok = n_tok;
    ws->prepared_in = n_in;
    return cudaGetLastError();
}

extern "C" {

static cudaError_t ws_create(ingot_linear_ws** out, size_t act_elems, size_t partial_floats, int n_slots, bool bf16) {
    *out = nullptr;
    ingot_linear_ws* ws = new ingot_linear_ws();
    ws->act_elems = act_elems;
    ws->partial_floats = partial_floats;
    ws->n_slots = n_slots;
    ws->bf16 = bf16;
    ws->planes = bf16 ? 1 : 2;
    int dev = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&ws->num_sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = cudaMalloc(&ws->hi, ws->act_elems * 2)) != cudaSuccess || (e = cudaMalloc(&ws->lo, ws->act_elems * 2)) != cudaSuccess ||
        // zero-filled: padding columns that no producer writes must be finite, they meet zero weights
        (e = cudaMemset(ws->hi, 0, ws->act_elems * 2)) != cudaSuccess || (e = cudaMemset(ws->lo, 0, ws->act_elems * 2)) != cudaSuccess ||
        (e = cudaMalloc(&ws->partial, n_slots * ws->partial_floats * 4)) != cudaSuccess || (e = cudaMalloc(&ws->status, sizeof(int))) != cudaSuccess ||
        (e = cudaMemset(ws->status, 0, sizeof(int))) != cudaSuccess ||
        (e = cudaFuncSetAttribute(linear_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(linear_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(linear_few_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewSmem)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(linear_few_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewSmem)) != cudaSuccess) {
        cudaFree(ws->hi); cudaFree(ws->lo); cudaFree(ws->partial); cudaFree(ws->status);
        delete ws;
        return e;
    }
    *out = ws;
    return cudaSuccess;
}

// max_tok x max_in: the largest activation matrix that will be prepared; also the largest output (tokens x width).
cudaError_t ingot_linear_ws_create(ingot_linear_ws** out, int max_tok, int max_in) {
    // k-slice partials: three slots, each at least two full-width slices of the largest batch (the hi-plane and the
    // lo-plane product of a quantised matrix), 24 MB or more
    const size_t act = (size_t)max_tok * max_in;
    return ws_create(out, act, std::max((size_t)6 << 20, 2 * act), 3, false);
}

// bf16 weights: one partial slot that holds at least one slice of max_tok x max_out.
cudaError_t ingot_linear_ws_create_bf16(ingot_linear_ws** out, int max_tok, int max_in, int max_out) {
    return ws_create(out, (size_t)max_tok * max_in, std::max((size_t)6 << 20, (size_t)max_tok * max_out), 1, true);
}

void ingot_linear_ws_destroy(ingot_linear_ws* ws) {
    if (!ws) return;
    cudaFree(ws->hi); cudaFree(ws->lo); cudaFree(ws->partial); cudaFree(ws->status);
    delete ws;
}

// Whether a projection of this shape can take the tensor-core path.
int ingot_linear_tc_supported(const ingot_linear_ws* ws, int w_is_f16, int n_in, int n_out, int n_tok) {
    if (!ws || !encode_fn() || n_tok < (ws->bf16 ? 2 : 16) || n_out % 4 != 0 || (size_t)n_tok * n_in > ws->act_elems) return 0;
    return ws->bf16 ? n_in % 8 == 0 : w_is_f16 && n_in % kBK == 0;
}

// Row length the planes may have: whole k-steps of f16, any multiple of 8 of bf16.
static bool act_shape_ok(const ingot_linear_ws* ws, int n_in, int n_tok) {
    return (size_t)n_tok * n_in <= ws->act_elems && n_in % (ws->bf16 ? 8 : kBK) == 0;
}

// Splits x [n_tok][n_in] f32 into the workspace's hi/lo f16 matrices; the following ingot_linear_tc_run calls use them.
cudaError_t ingot_linear_tc_prepare(ingot_linear_ws* ws, const float* x, int n_in, int n_tok, cudaStream_t s) {
    if (!act_shape_ok(ws, n_in, n_tok) || ws->bf16) return cudaErrorInvalidValue;
    cudaError_t le = launch_pdl(split_act_kernel<kActF16Pair>, dim3((unsigned)((n_in / 4 + 255) / 256), n_tok), dim3(256), 0, s, ws->hi, ws->lo, x, n_in, n_in);
    if (le != cudaSuccess) return le;
    return set_prepared(ws, n_in, n_tok);
}

// bf16 workspace: rows of x are x_ld floats apart; planes 1 or 2.
cudaError_t ingot_linear_tc_prepare_bf16(ingot_linear_ws* ws, const float* x, int x_ld, int n_in, int n_tok, int planes, cudaStream_t s) {
    if (!act_shape_ok(ws, n_in, n_tok) || !ws->bf16 || x_ld % 4 != 0) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)((n_in / 4 + 255) / 256), n_tok);
    cudaError_t le = planes > 1 ? launch_pdl(split_act_kernel<kActBF16Pair>, grid, dim3(256), 0, s, ws->hi, ws->lo, x, x_ld, n_in)
                                : launch_pdl(split_act_kernel<kActBF16>, grid, dim3(256), 0, s, ws->hi, ws->lo, x, x_ld, n_in);
    if (le != cudaSuccess) return le;
    ws->planes = planes > 1 ? 2 : 1;
    return set_prepared(ws, n_in, n_tok);
}

// The planes themselves ([n_tok][n_in] bf16, row-contiguous) for kernels that write their output as the next product's
// operand, and the declaration that they have been (or, in stream order, will have been) written.
void ingot_linear_ws_planes(ingot_linear_ws* ws, void** hi, void** lo) { *hi = ws->hi; *lo = ws->lo; }
cudaError_t ingot_linear_tc_prepared(ingot_linear_ws* ws, int n_in, int n_tok, int planes) {
    if (!act_shape_ok(ws, n_in, n_tok) || !ws->bf16) return cudaErrorInvalidValue;
    ws->planes = planes > 1 ? 2 : 1;
    return set_prepared(ws, n_in, n_tok);
}

// The same with the producer of the activations folded in: rmsnorm(x; norm_w, eps).
cudaError_t ingot_linear_tc_prepare_norm(ingot_linear_ws* ws, const float* x, const float* norm_w, float eps, int n_in, int n_tok,
                                         cudaStream_t s) {
    if (!act_shape_ok(ws, n_in, n_tok) || ws->bf16) return cudaErrorInvalidValue;
    cudaError_t le = launch_pdl(rmsnorm_split_kernel<kActF16Pair>, dim3(n_tok), dim3(256), 0, s, ws->hi, ws->lo, x, norm_w, n_in, n_in, eps);
    if (le != cudaSuccess) return le;
    return set_prepared(ws, n_in, n_tok);
}
cudaError_t ingot_linear_tc_prepare_norm_bf16(ingot_linear_ws* ws, const float* x, const float* norm_w, float eps, int n_in, int n_mean, int n_tok,
                                              int planes, cudaStream_t s) {
    if (!act_shape_ok(ws, n_in, n_tok) || !ws->bf16) return cudaErrorInvalidValue;
    cudaError_t le = planes > 1
        ? launch_pdl(rmsnorm_split_kernel<kActBF16Pair>, dim3(n_tok), dim3(256), 0, s, ws->hi, ws->lo, x, norm_w, n_in, n_mean, eps)
        : launch_pdl(rmsnorm_split_kernel<kActBF16>, dim3(n_tok), dim3(256), 0, s, ws->hi, ws->lo, x, norm_w, n_in, n_mean, eps);
    if (le != cudaSuccess) return le;
    ws->planes = planes > 1 ? 2 : 1;
    return set_prepared(ws, n_in, n_tok);
}

// count <= 3 matrices W_m [n_out_m][n_in] in one launch; matrix m goes to `out` (count == 1, !to_partial) or as k slices to
// scratch slot first_slot + m.
// append: the slices are written behind the ones the slots already hold (all slots of the group must hold the same
// number), so that a second product - the lo plane of a quantised matrix after its hi plane - simply adds k slices
// for the consumer kernel to sum.
// rows_per_block > 0 (count == 1): block-diagonal; n_in is then the row length of one block and the prepared activations hold
// n_out / rows_per_block such blocks side by side.
static cudaError_t launch_gemm(ingot_linear_ws* ws, float* out, const void* const* w, int n_in, const int* n_out, int count,
                               int accumulate, int first_slot, bool to_partial, bool append, cudaStream_t s, int rows_per_block = 0,
                               __half* out_half = nullptr, int half_ld = 0, int half_block = 0, int gate = 0, float* const* out_at = nullptr, int* there = nullptr) {
    const int n_tok = ws->prepared_tok;
    if (rows_per_block > 0 && (count != 1 || n_out[0] % rows_per_block != 0 || rows_per_block % 4 != 0 || n_in % 8 != 0)) return cudaErrorInvalidValue;
    const int act_in = rows_per_block > 0 ? n_in * (n_out[0] / rows_per_block) : n_in;
    if (act_in != ws->prepared_in || n_tok < 1 || count < 1 || first_slot < 0 || first_slot + count > ws->n_slots || (count > 1 && !to_partial) ||
        (append && !to_partial))
        return cudaErrorInvalidValue;
    const int held = append ? ws->slot_split[first_slot] : 0;
    for (int m = 0; m < count && append; m++)
        if (ws->slot_split[first_slot + m] != held || ws->slot_out[first_slot + m] != n_out[m]) return cudaErrorInvalidValue;
    make_room(ws);
    const CUtensorMap* maps[3] = {nullptr, nullptr, nullptr};
    GemmParams p = {};
    const bool few = ws->planes > 1 && n_tok <= kFewRows;  // linear_few_kernel
    const int tile = few ? 128 : 256;
    int tiles_n = 0, fit = 1 << 30;
    long long blocks = 0;  // of 128 outputs
    for (int m = 0; m < count; m++) {
        if (!(maps[m] = map_of(ws, w[m], n_out[m], n_in, 128, ws->bf16))) return cudaErrorUnknown;
        tiles_n += rows_per_block > 0 ? n_out[m] / rows_per_block * ((rows_per_block + tile - 1) / tile) : (n_out[m] + tile - 1) / tile;
        blocks += rows_per_block > 0 ? n_out[m] / rows_per_block * blocks_of(rows_per_block) : blocks_of(n_out[m]);
        p.tile_end[m] = tiles_n;
        p.n_out[m] = n_out[m];
        p.partial[m] = ws->partial + (size_t)(first_slot + m) * ws->partial_floats + (size_t)held * n_tok * n_out[m];
        fit = std::min(fit, (int)(ws->partial_floats / ((size_t)n_tok * n_out[m])) - held);
    }
    for (int m = count; m < 3; m++) { maps[m] = maps[count - 1]; p.tile_end[m] = tiles_n; p.n_out[m] = n_out[count - 1]; p.partial[m] = p.partial[count - 1]; }
    p.tiles_n = tiles_n;
    const int k_steps = (n_in + kBK - 1) / kBK;
    if (to_partial && fit < 1) return cudaErrorInvalidValue;
    const int n_split = out_half || gate ? 1 : k_slices(blocks * blocks_of(n_tok), k_steps, fit, ws->num_sms);  // no more than the slots hold
    const PairTiles t = pair_tiles(n_tok, tiles_n, ws->planes, k_steps, n_split, ws->num_sms);
    // A batch of few tokens fetches only its own rows (whole 8-row swizzle groups). What else the boxes hold is multiplied along and never stored.
    const int box = few ? (n_tok + 7) / 8 * 8 : t.rows / 2;
    const CUtensorMap *hi = map_of(ws, ws->hi, n_tok, act_in, box, ws->bf16), *lo = ws->planes > 1 ? map_of(ws, ws->lo, n_tok, act_in, box, ws->bf16) : hi;
    if (!hi || !lo) return cudaErrorUnknown;
    p.out_half = out_half;
    p.half_ld = half_ld;
    p.half_block = half_block;
    p.out = out; p.status = ws->status;
    if (out_at && few && n_split == 1) {
        p.out_at = out_at;
        *there = 1;
    }
    p.act = gate;
    if (gate) p.out_hi = reinterpret_cast<__nv_bfloat16*>(ws->lo);
    p.n_tok = n_tok; p.k_steps = k_steps; p.n_split = n_split; p.accumulate = accumulate;
    p.to_partial = to_partial ? 1 : 0;
    p.idesc = kIdescF16 | (ws->bf16 ? kIdescBF16 : 0u);
    p.rows_per_block = rows_per_block;
    p.k_block = rows_per_block > 0 ? n_in : 0;
    p.tiles_per_block = rows_per_block > 0 ? (rows_per_block + tile - 1) / tile : 0;
    cudaError_t le = few ? launch_few<false>(p, box, tiles_n * n_split, ws->num_sms, *hi, *lo, maps, s)
                         : launch_pair<false>(p, t.rows, ws->planes, box, t.row_tiles, tiles_n * t.row_tiles * n_split, ws->num_sms, *hi, *lo, maps, s);
    if (le != cudaSuccess) return le;
    for (int m = 0; m < count; m++) {
        ws->slot_split[first_slot + m] = held + n_split;
        ws->slot_out[first_slot + m] = n_out[m];
    }
    if (!to_partial && n_split > 1) {
        const size_t n = (size_t)n_tok * n_out[0];
        le = launch_pdl(splitk_reduce_kernel, dim3((unsigned)((n / 4 + 255) / 256)), dim3(256), 0, s, out, (const float*)p.partial[0], n_split, n,
                        accumulate);
        if (le != cudaSuccess) return le;
    }
    return cudaGetLastError();
}

// out [n_tok][n_out] (+)= prepared activations x W^T, W f16 [n_out][n_in] on the device.
cudaError_t ingot_linear_tc_run(ingot_linear_ws* ws, float* out, const void* w, int n_in, int n_out, int accumulate, cudaStream_t s) {
    return launch_gemm(ws, out, &w, n_in, &n_out, 1, accumulate, 0, false, false, s);
}

// The same to *out_at (a pointer in device memory, pinned host memory behind it) where the product's own kernel can write there as it goes
// (*there = 1): few rows and no k slices; else to out. 8 rows of 32768 logits then cross PCIe while the weights stream:
// product and delivery 53 -> 40 us (2048 wide, B200).
cudaError_t ingot_linear_tc_run_to(ingot_linear_ws* ws, float* out, float* const* out_at, const void* w, int n_in, int n_out, int* there, cudaStream_t s) {
    *there = 0;
    return launch_gemm(ws, out, &w, n_in, &n_out, 1, 0, 0, false, false, s, 0, nullptr, 0, 0, 0, out_at, there);
}

// Block-diagonal product: W [n_out][k_block], output rows of block b = row / rows_per_block times the prepared columns
// b * k_block .. (b + 1) * k_block - 1.
cudaError_t ingot_linear_tc_run_blocks(ingot_linear_ws* ws, float* out, const void* w, int k_block, int n_out, int rows_per_block, cudaStream_t s) {
    return launch_gemm(ws, out, &w, k_block, &n_out, 1, 0, 0, false, false, s, rows_per_block);
}

// Plain (rows_per_block 0) or block-diagonal product with an f16 result: row t at out + t * out_ld, block b's columns from b * out_block
// on. Row lengths and blocks are multiples of 8.
cudaError_t ingot_linear_tc_run_half(ingot_linear_ws* ws, void* out, int out_ld, int out_block, const void* w, int n_in, int n_out, int rows_per_block,
                                     cudaStream_t s) {
    if (out_ld % 8 != 0 || out_block % 8 != 0 || n_out % 8 != 0 || rows_per_block % 8 != 0) return cudaErrorInvalidValue;
    return launch_gemm(ws, nullptr, &w, n_in, &n_out, 1, 0, 0, false, false, s, rows_per_block, static_cast<__half*>(out), out_ld, out_block);
}

// out f16 [n_tok][out_ld] = a W^T, both operands f16: a [a_rows][n_in] with n_tok <= a_rows, W [n_out][n_in]. Lengths are multiples of 8.
cudaError_t ingot_linear_tc_run_f16(ingot_linear_ws* ws, void* out, int out_ld, const void* a, int a_rows, int n_tok, const void* w, int n_in, int n_out, cudaStream_t s) {
    if (n_in % 8 != 0 || n_out % 8 != 0 || out_ld % 8 != 0 || n_tok < 1 || n_tok > a_rows) return cudaErrorInvalidValue;
    GemmParams p = {};
    p.tiles_n = (n_out + 255) / 256;
    p.k_steps = (n_in + kBK - 1) / kBK;
    const PairTiles t = pair_tiles(n_tok, p.tiles_n, 1, p.k_steps, 1, ws->num_sms);
    make_room(ws);
    const CUtensorMap *ma = map_of(ws, a, a_rows, n_in, t.rows / 2, false), *mw = map_of(ws, w, n_out, n_in, 128, false);
    if (!ma || !mw) return cudaErrorUnknown;
    for (int m = 0; m < 3; m++) { p.n_out[m] = n_out; p.tile_end[m] = p.tiles_n; }
    p.status = ws->status;
    p.n_tok = n_tok;
    p.n_split = 1;
    p.idesc = kIdescF16;
    p.out_half = static_cast<__half*>(out);
    p.half_ld = out_ld;
    const CUtensorMap* const maps[3] = {mw, mw, mw};
    return launch_pair<false>(p, t.rows, 1, t.rows / 2, t.row_tiles, p.tiles_n * t.row_tiles, ws->num_sms, *ma, *ma, maps, s);
}

cudaError_t ingot_grouped_tc_run(ingot_linear_ws* ws, const ingot_grouped_gemm* g, cudaStream_t s) {
    if (g->act == 2 && (g->n_out % 64 != 0 || !g->out_hi)) return cudaErrorInvalidValue;
    if (!ws->bf16 || g->n_in % 8 != 0 || g->n_out % 8 != 0 || g->n_rows < 1 || g->n_groups < 1 || g->rows_per_group < 1) return cudaErrorInvalidValue;
    const int planes = g->a_lo ? 2 : 1;
    const bool few = planes > 1 && g->rows_per_group <= kFewRows;  // as for plain products
    const int tile = few ? 128 : 256, rows = few ? (g->rows_per_group + 7) / 8 * 8 : kPairRows / planes, box = few ? rows : rows / 2;
    make_room(ws);
    const CUtensorMap* hi = map_of(ws, g->a_hi, g->n_rows, g->n_in, box, true);
    const CUtensorMap* lo = planes > 1 ? map_of(ws, g->a_lo, g->n_rows, g->n_in, box, true) : hi;
    if (!hi || !lo) return cudaErrorUnknown;
    GemmParams p = {};
    p.tiles_n = (g->n_out + tile - 1) / tile;
    for (int m = 0; m < 3; m++) { p.n_out[m] = g->n_out; p.tile_end[m] = p.tiles_n; }
    p.out = g->out;
    p.status = ws->status;
    p.n_tok = g->n_rows;
    p.k_steps = (g->n_in + kBK - 1) / kBK;
    p.n_split = 1;
    p.idesc = kIdescF16 | kIdescBF16;
    p.row_scale = g->row_scale;
    p.act = g->act;
    p.out_hi = static_cast<__nv_bfloat16*>(g->out_hi);
    p.out_lo = static_cast<__nv_bfloat16*>(g->out_lo);
    static_assert(kFewGroups == kPairGroups, "groups of a launch");
    for (int first = 0; first < g->n_groups; first += kPairGroups) {  // a CTA keeps a list of the groups
        p.group_start = g->group_start + first;
        p.n_groups = std::min(g->n_groups - first, kPairGroups);
        const CUtensorMap* w = map_of(ws, static_cast<const char*>(g->w) + (size_t)first * g->n_out * g->n_in * 2, p.n_groups * g->n_out, g->n_in, 128, true);
        if (!w) return cudaErrorUnknown;
        const CUtensorMap* const maps[3] = {w, w, w};
        const int some = std::min(p.n_groups, g->n_rows);  // groups that can have rows
        const cudaError_t le = few ? launch_few<true>(p, rows, some * p.tiles_n, ws->num_sms, *hi, *lo, maps, s)
                                   : launch_pair<true>(p, rows, planes, box, 0, (g->n_rows / rows + some) * p.tiles_n, ws->num_sms, *hi, *lo, maps, s);
        if (le != cudaSuccess) return le;
    }
    return cudaSuccess;
}

// The same product left as k slices in scratch slot 0..2 for one of the ingot_linear_tc_finish_* calls below.
cudaError_t ingot_linear_tc_run_partial(ingot_linear_ws* ws, const void* w, int n_in, int n_out, int slot, cudaStream_t s) {
    return launch_gemm(ws, nullptr, &w, n_in, &n_out, 1, 0, slot, true, false, s);
}

// The products of count <= 3 matrices that read the same prepared activations (q/k/v, gate/up), as one launch:
// matrix m is left as k slices in scratch slot m.
// append != 0: the slices are added behind those the slots hold from the call before (same widths).
cudaError_t ingot_linear_tc_run_partial_group(ingot_linear_ws* ws, const void* const* w, int n_in, const int* n_out, int count,
                                              int first_slot, int append, cudaStream_t s) {
    return launch_gemm(ws, nullptr, w, n_in, n_out, count, 0, first_slot, true, append != 0, s);
}

// The product left in `slot`: *n_slices matrices [prepared tokens][n_out] f32 to be summed in order.
const float* ingot_linear_ws_slices(const ingot_linear_ws* ws, int slot, int* n_slices) {
    *n_slices = ws->slot_split[slot];
    return ws->partial + (size_t)slot * ws->partial_floats;
}

static Slices slices_of(const ingot_linear_ws* ws, int slot) {
    return Slices{ws->partial + (size_t)slot * ws->partial_floats, ws->slot_split[slot]};
}

// outs[m] = product left in slot m, for count <= 3 outputs (q, k, v) in one launch.
cudaError_t ingot_linear_tc_finish_group(ingot_linear_ws* ws, float* const* outs, int count, cudaStream_t s) {
    if (count < 1 || count > 3) return cudaErrorInvalidValue;
    FinishGroup g = {};
    int widest = 0;
    for (int m = 0; m < count; m++) {
        g.in[m] = slices_of(ws, m);
        g.out[m] = outs[m];
        g.n_out[m] = ws->slot_out[m];
        widest = std::max(widest, ws->slot_out[m]);
    }
    const size_t n = (size_t)ws->prepared_tok * widest;
    cudaError_t le = launch_pdl(finish_group_kernel, dim3((unsigned)((n / 4 + 255) / 256), count), dim3(256), 0, s, g, ws->prepared_tok);
    if (le != cudaSuccess) return le;
    return cudaGetLastError();
}

// x += product left in `slot` (the residual add), then, with norm_w, the hi/lo activations of rmsnorm(x; norm_w, eps)
// become the prepared input of the next projections (n_in = the product's width).
cudaError_t ingot_linear_tc_finish_residual_norm(ingot_linear_ws* ws, float* x, const float* norm_w, float eps, int slot, cudaStream_t s) {
    const int n = ws->slot_out[slot], n_tok = ws->prepared_tok;
    if (n % 4 != 0 || (norm_w && !act_shape_ok(ws, n, n_tok)) || ws->bf16) return cudaErrorInvalidValue;
    cudaError_t le = launch_pdl(finish_residual_norm_kernel<kActF16Pair>, dim3(n_tok), dim3(256), 0, s, x, slices_of(ws, slot), ws->hi, ws->lo, norm_w, n, n, n_tok, eps, (const float*)nullptr, (const int32_t*)nullptr, 0);
    if (le != cudaSuccess) return le;
    return norm_w ? set_prepared(ws, n, n_tok) : cudaGetLastError();
}
// pair_rows (null: none): x[t] also takes in the rows row_of[t * top + k] of it.
cudaError_t ingot_linear_tc_finish_residual_norm_bf16(ingot_linear_ws* ws, float* x, const float* norm_w, float eps, int n_mean, int planes,
                                                      const float* pair_rows, const int32_t* row_of, int top, cudaStream_t s) {
    if (!pair_rows) top = 0;
    const int n = ws->slot_out[0], n_tok = ws->prepared_tok;
    if (n % 4 != 0 || (norm_w && !act_shape_ok(ws, n, n_tok)) || !ws->bf16) return cudaErrorInvalidValue;
    cudaError_t le = planes > 1
        ? launch_pdl(finish_residual_norm_kernel<kActBF16Pair>, dim3(n_tok), dim3(256), 0, s, x, slices_of(ws, 0), ws->hi, ws->lo, norm_w, n, n_mean, n_tok, eps, pair_rows, row_of, top)
        : launch_pdl(finish_residual_norm_kernel<kActBF16>, dim3(n_tok), dim3(256), 0, s, x, slices_of(ws, 0), ws->hi, ws->lo, norm_w, n, n_mean, n_tok, eps, pair_rows, row_of, top);
    if (le != cudaSuccess) return le;
    ws->planes = planes > 1 ? 2 : 1;
    return norm_w ? set_prepared(ws, n, n_tok) : cudaGetLastError();
}

// The bf16 operand act(gate) * up of the next product, from W whose rows are runs of 32 gate rows, each followed by the 32 up rows that go
// with them (n_out: both). act: 0 silu, 1 the tanh form of gelu; planes: of the operand. With one plane in and out the accumulators
// become the operand on their way out, in the plane that is not read (the lo plane; the two then change places): 4096 rows of 28672
// wide results took 150 us more to write in f32 and to read again (B200). Otherwise, and where k slices fill the GPU, through slot 0.
cudaError_t ingot_linear_tc_run_gated_bf16(ingot_linear_ws* ws, const void* w, int n_in, int n_out, int act, int planes, cudaStream_t s) {
    const int n = n_out / 2, n_tok = ws->prepared_tok;
    if (!ws->bf16 || n_out % 64 != 0 || !act_shape_ok(ws, n, n_tok)) return cudaErrorInvalidValue;
    if (ws->planes == 1 && planes == 1 && k_slices(blocks_of(n_out) * blocks_of(n_tok), (n_in + kBK - 1) / kBK, 1 << 20, ws->num_sms) == 1) {
        const cudaError_t e = launch_gemm(ws, nullptr, &w, n_in, &n_out, 1, 0, 0, false, false, s, 0, nullptr, 0, 0, 2 + act);
        if (e != cudaSuccess) return e;
        std::swap(ws->hi, ws->lo);
        return set_prepared(ws, n, n_tok);
    }
    const cudaError_t e = launch_gemm(ws, nullptr, &w, n_in, &n_out, 1, 0, 0, true, false, s);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)((n / 4 + 255) / 256), n_tok);
    cudaError_t le = planes > 1
        ? launch_pdl(finish_gated_kernel<kActBF16Pair>, grid, dim3(256), 0, s, ws->hi, ws->lo, slices_of(ws, 0), n, (size_t)n_tok * 2 * n, act)
        : launch_pdl(finish_gated_kernel<kActBF16>, grid, dim3(256), 0, s, ws->hi, ws->lo, slices_of(ws, 0), n, (size_t)n_tok * 2 * n, act);
    if (le != cudaSuccess) return le;
    ws->planes = planes > 1 ? 2 : 1;
    return set_prepared(ws, n, n_tok);
}

// hi/lo of silu(slot_gate) .* slot_up become the prepared input of the next projection.
cudaError_t ingot_linear_tc_finish_swiglu(ingot_linear_ws* ws, int slot_gate, int slot_up, cudaStream_t s) {
    const int n_in = ws->slot_out[slot_gate], n_tok = ws->prepared_tok;
    const size_t n = (size_t)n_tok * n_in;
    if (ws->slot_out[slot_up] != n_in || n > ws->act_elems || n_in % kBK != 0) return cudaErrorInvalidValue;
    cudaError_t le = launch_pdl(finish_swiglu_kernel, dim3((unsigned)((n / 4 + 255) / 256)), dim3(256), 0, s, ws->hi, ws->lo, slices_of(ws, slot_gate), slices_of(ws, slot_up), n);
    if (le != cudaSuccess) return le;
    return set_prepared(ws, n_in, n_tok);
}

int* ingot_linear_ws_status_dev(ingot_linear_ws* ws) { return ws->status; }

// The status word: non-zero after a bounded wait expired (bit 0) or a group was longer than rows_per_group said (bit 1; its other rows are
// left out) in some launch since the last call. Synchronises the device.
int ingot_linear_ws_status(ingot_linear_ws* ws) {
    int v = 0;
    if (cudaMemcpy(&v, ws->status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (v) cudaMemset(ws->status, 0, sizeof(int));
    return v;
}

}  // extern "C"
