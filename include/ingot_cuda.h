/* ingot_cuda.h — C ABI of the B200 (sm_100a) attention path for the Ingot inference engine.
 *
 * The library replaces, for a Backend implementation, the per-layer attention stage that sits
 * between the Q/K/V projections and the output projection of Ingot's forward pass:
 *     rope(q), rope(k) -> KV-cache append -> causal GQA attention
 * (CPU reference: src/cpu_backend.cpp:43-69; Metal reference: src/metal_backend.mm:443-445).
 *
 * Conventions
 *   - Every entry point returns an int status (INGOT_OK == 0); nothing throws or aborts.
 *   - Pointers named *_dev are device pointers on the device the cache was created on; pointers
 *     named *_host are host pointers. `stream` is a cudaStream_t passed as void* (NULL = default
 *     stream). Calls are asynchronous on `stream` unless stated otherwise.
 *   - head_dim is 128 (the reference's flash kernels are specialised the same way,
 *     src/metal_backend.mm:340,361). Query heads are grouped onto KV heads as h / (n_head / n_head_kv)
 *     (src/cpu_backend.cpp:29,53).
 *   - Query / output activations are row-major [token][head][128].
 *   - The KV cache is f16 (as the Metal reference's, src/metal_backend.mm:197-198). Layouts:
 *       contiguous: K and V each [n_layer][n_head_kv][n_ctx][128]            (one sequence)
 *       paged:      K and V each [n_layer][n_blocks][n_head_kv][16][128]     (16-token blocks,
 *                   any number of sequences, each described by a row of a block table)
 *   - The cache is a pure function of (layer, position): positions may be rewritten in any order
 *     and the caller owns the notion of sequence length (src/main.cpp:295,374-375 rewind `pos`
 *     without telling the backend).
 *   - Scratch. The decode, prefill and host-buffer calls keep scratch on the handle, sized on first use and
 *     grown when a later call needs more (nothing is ever freed before ingot_kv_destroy). Growing
 *     allocates device memory, which is not allowed while a stream is being captured: run a call once
 *     eagerly with the largest shape before capturing it into a CUDA graph. Graphs captured earlier stay
 *     valid across a later growth.
 *   - A handle belongs to the device that was current at ingot_kv_create; calls with another device
 *     current are rejected with INGOT_ERR_INVALID.
 */
#ifndef INGOT_CUDA_H
#define INGOT_CUDA_H

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

enum {
    INGOT_OK = 0,
    INGOT_ERR_INVALID = 1,      /* bad argument (null pointer, range, unsupported shape) */
    INGOT_ERR_CUDA = 2,         /* a CUDA runtime/driver call failed; see ingot_last_error() */
    INGOT_ERR_UNSUPPORTED = 3,  /* shape or dtype outside what the kernels are built for */
    INGOT_ERR_NOMEM = 4,
    INGOT_ERR_DEVICE = 5        /* a kernel reported a problem through its status word */
};

enum { INGOT_F32 = 0, INGOT_F16 = 1, INGOT_BF16 = 2 };
enum { INGOT_KV_CONTIGUOUS = 0, INGOT_KV_PAGED = 1 };
#define INGOT_BLOCK_TOKENS 16
#define INGOT_HEAD_DIM 128

typedef struct ingot_kv ingot_kv;

/* Human-readable text for a status code / for the last failure on the calling thread. */
const char* ingot_status_string(int status);
const char* ingot_last_error(void);
/* Library build: compiled architecture string, e.g. "sm_100a". */
const char* ingot_build_arch(void);
/* Build variant: "" for the production library, "bounds-check" for the build whose kernels range-check every
 * offset they compute (see ingot_kv_test_shrink_extent). */
const char* ingot_build_flags(void);

/* ---- KV cache ------------------------------------------------------------------------------
 * Replaces the cache the reference backends own (src/backend.h:1; CPU: src/cpu_backend.h:23,
 * src/cpu_backend.cpp:18-19; Metal: src/metal_backend.mm:197-198).
 * capacity = n_ctx positions (contiguous) or number of 16-token blocks (paged).
 * max_seqs = most sequences one decode call will carry (sizes the split-KV scratch); 1 for a
 * single-sequence backend. Allocates on the current device. Synchronous. */
int ingot_kv_create(ingot_kv** out, int layout, int n_layer, int n_head_kv, int head_dim, int capacity,
                    int max_seqs);
void ingot_kv_destroy(ingot_kv* kv);
/* Device base pointers of one layer's K / V storage (layouts above), e.g. to import a cache. */
void* ingot_kv_k_dev(ingot_kv* kv, int layer);
void* ingot_kv_v_dev(ingot_kv* kv, int layer);
size_t ingot_kv_layer_bytes(const ingot_kv* kv);
/* Reads and clears the device status word (0 = no kernel reported a problem). Synchronises `stream`. */
int ingot_kv_status(ingot_kv* kv, void* stream, int* status_out);
/* TEST HOOK (no reference counterpart): with stall_ms > 0 the tcgen05 prefill kernel launched for this handle
 * issues no K/V copies and bounds its waits at stall_ms milliseconds, so that every wait runs out, the kernel
 * returns normally and status bit 4 is raised; 0 restores normal operation. Lets a test exercise the
 * bounded-wait exit without hanging or faulting anything. */
int ingot_kv_test_stall_prefill(ingot_kv* kv, int stall_ms);
/* TEST HOOK of the bounds-check build (no reference counterpart; no effect in the production library): the
 * kernels' range checks treat each cache layer as only `elems` f16 elements long (0 restores the real extent).
 * Accesses beyond that - which are inside the real allocation - are then skipped and raise status bit 8, which
 * shows that the checks are live without any access ever leaving a buffer. */
int ingot_kv_test_shrink_extent(ingot_kv* kv, size_t elems);

/* ---- K1: fused RoPE + K/V append -------------------------------------------------------------
 * Replaces ops::rope on q and k plus the cache memcpy (src/ops.cpp:243-255,
 * src/cpu_backend.cpp:43-49); on Metal: rope + rope_k_to_cache + to_half
 * (shaders/kernels.metal:256-282,779-782; src/metal_backend.mm:324-334,395-409).
 * For each token t in [0, n_tok): position p = positions_dev ? positions_dev[t] : pos0 + t.
 *   q_dev  [n_tok][n_head][128]   f32, may be NULL (no query work);  rotated q is written as f16
 *          to q_out_dev [n_tok][n_head][128].
 *   k_dev, v_dev [n_tok][n_head_kv][128] f32; rotated k and raw v are written as f16 into the cache
 *          at position p.
 *   inv_freq_dev [64] f32: Model::rope_inv_freq (src/model.cpp:59-69). Rotation is on adjacent
 *          pairs (x[2i], x[2i+1]) by angle float(p) * inv_freq[i], in f32.
 * Paged caches: token t belongs to sequence s = seq_ids_dev ? seq_ids_dev[t] : 0 and its block is
 * block_tables_dev[s * max_blocks_per_seq + p / 16]. Contiguous caches ignore those arguments. */
int ingot_rope_kv_append(ingot_kv* kv, int layer, const float* q_dev, void* q_out_dev, const float* k_dev,
                         const float* v_dev, const float* inv_freq_dev, int n_head, int pos0, int n_tok,
                         const int32_t* positions_dev, const int32_t* seq_ids_dev,
                         const int32_t* block_tables_dev, int max_blocks_per_seq, void* stream);

/* Import of already-rotated f16 K/V rows [n_tok][n_head_kv][128] into the cache at positions
 * pos0..pos0+n_tok-1 of one sequence (block_table_dev: that sequence's row, paged only).
 * No reference counterpart on the CPU path (its cache is f32); mirrors the layout transform of
 * the Metal KV store (src/metal_backend.mm:395-409) without the arithmetic. */
int ingot_kv_import_f16(ingot_kv* kv, int layer, const void* k_f16_dev, const void* v_f16_dev, int pos0,
                        int n_tok, const int32_t* block_table_dev, void* stream);

/* ---- K3: split-KV flash decoding -------------------------------------------------------------
 * Replaces the attention lambda for one-token queries (src/cpu_backend.cpp:51-69) and Metal's
 * attn_decode_g3 + attn_combine (shaders/kernels.metal:428-516; src/metal_backend.mm:340-360).
 * n_seq sequences, one query token each:
 *   q_dev   [n_seq][n_head][128]  q_dtype in {F32, F16, BF16}, already rotated
 *   out_dev [n_seq][n_head][128]  out_dtype in {F32, F16}
 *   seq_lens_dev [n_seq] int32: keys 0..len-1 of each sequence are attended (len >= 1).
 *          NULL with n_seq == 1 means the single length max_seq_len.
 *   max_seq_len: host-side upper bound of every length (sizes the launch grid). A device length beyond what the grid covers is
 *          clamped and raises bit 0 of the status word.
 *   block_tables_dev [n_seq][max_blocks_per_seq]: paged caches only.
 * chunk_keys: keys per split (multiple of 16), or 0 to let the library choose. */
int ingot_attn_decode(ingot_kv* kv, int layer, const void* q_dev, int q_dtype, void* out_dev, int out_dtype,
                      int n_head, int n_seq, const int32_t* seq_lens_dev, int max_seq_len,
                      const int32_t* block_tables_dev, int max_blocks_per_seq, int chunk_keys, void* stream);

/* The same for `layer_count` consecutive layers in one call, with the same lengths and block tables:
 * q_dev [layer_count][n_seq][n_head][128], out_dev likewise. This is the shape of the reference's
 * decode-attention microbenchmark, which encodes every layer's attention for one token into one
 * command buffer (src/metal_backend.mm:594-649, src/main.cpp:441-449). The layers are independent, so the
 * split CTAs of all of them form ONE grid (no launch boundary between layers) and a second launch merges the
 * split partials; ingot_attn_decode is the same with layer_count 1. */
int ingot_attn_decode_layers(ingot_kv* kv, int layer_begin, int layer_count, const void* q_dev, int q_dtype,
                             void* out_dev, int out_dtype, int n_head, int n_seq, const int32_t* seq_lens_dev,
                             int max_seq_len, const int32_t* block_tables_dev, int max_blocks_per_seq,
                             int chunk_keys, void* stream);

/* Decode for callers that cannot allocate device memory (no counterpart in the reference).
 * Meant for code that lives inside somebody else's memory budget: a plugin that is only ever handed
 * pre-allocated buffers, a component of a serving loop where cudaMalloc/cudaFree are banned because
 * they synchronise the device, or a process whose allocator is a fixed pool. This entry point takes
 * raw device pointers, needs no ingot_kv handle, and calls no cudaMalloc, cudaFree or allocating
 * library routine: the split-KV partials go to a fixed 2.06 MiB array that is part of the library
 * image (each GPU that loads the library holds it until the process exits).
 *   k_dev, v_dev  one layer of a contiguous f16 cache, [n_head_kv][n_ctx][128] (the caller's memory)
 *   q_dev   [n_head][128]  q_dtype in {F32, F16, BF16}, already rotated;  out_dev [n_head][128] F32 or F16
 *   n_keys  keys 0..n_keys-1 are attended (1 <= n_keys <= n_ctx); one sequence per call
 * Limits: n_head <= 64 and n_head / n_head_kv <= 8; larger calls are rejected with INGOT_ERR_INVALID
 * (use ingot_attn_decode). The first call on each device resolves the array's device address; make
 * that call before starting any stream capture. All calls on a device share the one array and it keeps
 * the previous call's contents (nothing in it needs clearing: every partial a call reads was written by
 * that same call), so two calls whose kernels can overlap on the GPU — different streams without an
 * ordering between them — race; keep them in one stream or order them with events. */
int ingot_attn_decode_noalloc(const void* k_dev, const void* v_dev, int n_ctx, int n_head_kv, const void* q_dev,
                              int q_dtype, void* out_dev, int out_dtype, int n_head, int n_keys, int chunk_keys,
                              void* stream);

/* ---- K2: causal GQA flash-attention prefill / chunked prefill -----------------------------------
 * Replaces n_tok iterations of the attention lambda (src/backend.h:16-20 + src/cpu_backend.cpp:51-69)
 * and Metal's attn_prefill (shaders/kernels.metal:518-633; src/metal_backend.mm:361-372).
 * Query token i (0 <= i < n_tok) sits at position q_pos0 + i and attends to keys 0..q_pos0+i, which
 * must already be in the cache (append first).
 *   q_dev   [n_tok][n_head][128]  q_dtype in {F32, F16, BF16}, already rotated
 *   out_dev [n_tok][n_head][128]  out_dtype in {F32, F16}
 *   block_table_dev: the sequence's block-table row (paged caches), else NULL.
 * impl: 0 = library's choice, 1 = force the warp-MMA kernel, 2 = force the tcgen05/TMEM/TMA kernel. */
int ingot_attn_prefill(ingot_kv* kv, int layer, const void* q_dev, int q_dtype, void* out_dev, int out_dtype,
                       int n_head, int q_pos0, int n_tok, const int32_t* block_table_dev, int impl,
                       void* stream);

/* K2 with the gather of head outputs fused into its epilogue, for a prefill sharded by KV head over
 * the GPUs of one NVLink/NVSwitch box (no counterpart in the reference, which is single-device; it
 * replaces "attn_prefill, then an all-gather of the head outputs"). This GPU's cache holds n_head_kv / N
 * KV heads and q_dev its n_head query heads [n_tok][n_head][128]. Every output row is written, by
 * plain stores from the kernel's epilogue, to each of the n_out (<= 8) buffers in out_ptrs — this GPU's
 * own and its peers' (peer-mapped device pointers, e.g. from symmetric memory) — in the token-major
 * layout [n_tok][out_n_head][128] at head index out_head0 + local head. When every rank has run it
 * and the ranks have synchronised (a barrier on the stream), each buffer holds all heads. tcgen05
 * kernel, contiguous caches only. out_ptrs is a host array read during the call. */
int ingot_attn_prefill_gather(ingot_kv* kv, int layer, const void* q_dev, int q_dtype, void* const* out_ptrs, int n_out,
                              int out_dtype, int n_head, int out_n_head, int out_head0, int q_pos0, int n_tok,
                              void* stream);

/* The same with completion signalling, so that no collective is needed as the cross-GPU barrier. Each GPU owns an
 * array of 32-bit counters, zero-initialised, one per source GPU, mapped into every peer (symmetric memory).
 * signal_ptrs[i] is the counter array that lives beside out_ptrs[i]; src_index is this GPU's slot in those arrays.
 * When the last CTA of this call's grid has finished - all stores to all destinations issued and fenced at
 * system scope - it adds 1 to counter src_index of every destination (red.release.sys). The consumer side is
 * ingot_gather_wait on the destination GPU: a one-CTA kernel on `stream` that waits until each of its n_src
 * counters is non-zero, takes the signal back off (so the counters need no reset between calls) and returns;
 * work queued behind it on the stream then sees every source's rows. The wait is bounded by timeout_ms: a source
 * that never signals raises status bit 4 (read it with ingot_kv_status) instead of hanging the GPU.
 * The destination buffers of call n+1 must not be reused before the consumers of call n are done with them
 * (alternate two buffers, or order the calls otherwise): the signal only says "written", not "read".
 * No counterpart in the reference. tcgen05 kernel, contiguous caches only. */
int ingot_attn_prefill_gather_signal(ingot_kv* kv, int layer, const void* q_dev, int q_dtype, void* const* out_ptrs,
                                     void* const* signal_ptrs, int n_out, int src_index, int out_dtype, int n_head,
                                     int out_n_head, int out_head0, int q_pos0, int n_tok, void* stream);
int ingot_gather_wait(ingot_kv* kv, void* counters_dev, int n_src, int timeout_ms, void* stream);

/* ---- Several GPUs from one process (no counterpart in the reference, which is single-device) ---------------
 * A handle that shards a long prefill by KV head over the first n_dev GPUs of this machine: it enables peer
 * access, creates on every GPU a cache shard with n_head_kv / n_dev heads (ingot_mg_kv(dev): fill it with
 * ingot_rope_kv_append / ingot_kv_import_f16 with that device current, that GPU's heads only), a token-major
 * destination buffer [n_ctx][n_head][128] (ingot_mg_out(dev)) and a counter array, and a stream (ingot_mg_stream).
 * ingot_mg_prefill runs ingot_attn_prefill_gather_signal on every GPU (q_dev[d]: GPU d's query heads
 * [n_tok][n_head / n_dev][128], on GPU d) and the bounded ingot_gather_wait behind it, synchronises, and returns
 * INGOT_OK when every GPU's buffer holds all heads of rows q_pos0..q_pos0+n_tok-1 (stored from row 0 of the buffer),
 * or INGOT_ERR_DEVICE if a wait for a peer ran out after timeout_ms. Needs peer access between all pairs. */
typedef struct ingot_mg ingot_mg;
int ingot_mg_create(ingot_mg** out, int n_dev, int n_layer, int n_head, int n_head_kv, int n_ctx, int out_dtype);
void ingot_mg_destroy(ingot_mg* mg);
ingot_kv* ingot_mg_kv(ingot_mg* mg, int dev);
void* ingot_mg_out(ingot_mg* mg, int dev);
void* ingot_mg_stream(ingot_mg* mg, int dev);
int ingot_mg_prefill(ingot_mg* mg, int layer, const void* const* q_dev, int q_dtype, int q_pos0, int n_tok, int timeout_ms);
/* One token of the one sequence of a CONTIGUOUS cache, K1 and K3 in one launch: q_dev [n_head][128], k_dev and v_dev
 * [n_head_kv][128] are the f32 projections of the token at position `pos`; the kernel rotates q and k
 * (src/ops.cpp:243-255), writes the K/V row of that position to the cache and attends over keys 0..pos
 * (src/cpu_backend.cpp:43-69 for one token), out_dev [n_head][128] f32 or f16. Bit-identical to ingot_rope_kv_append
 * followed by ingot_attn_decode. key_count_dev: null, or a device int32 holding pos + 1 (then `pos` is ignored and
 * max_seq_len bounds it, for CUDA graphs that are replayed at growing positions). */
int ingot_rope_append_decode(ingot_kv* kv, int layer, const float* q_dev, const float* k_dev, const float* v_dev,
                             const float* inv_freq_dev, void* out_dev, int out_dtype, int n_head, const int32_t* key_count_dev,
                             int pos, int max_seq_len, void* stream);

/* Prefill attention with the queries and the output in HOST memory and the cache resident on the device (the keys of
 * positions 0 .. q_pos0+n_tok-1 are in the cache already, e.g. after ingot_rope_kv_append or ingot_kv_import_f16):
 * q_host [n_tok][n_head][128] (f32, f16 or bf16) in, out_host [n_tok][n_head][128] (f32 or f16) out. The rows are
 * processed in chunks of chunk_tokens tokens (0: three full waves of CTAs, 4693 tokens at 24/8 heads) so that the copy of the next chunk in, the attention of the
 * current one and the copy of the previous one out overlap (copy streams of the handle's own; the caller's stream
 * carries the kernels and, at the end, waits for the last copy out). Asynchronous: synchronise `stream` before
 * reading out_host. Host buffers should be pinned. Not capturable into a CUDA graph. block_table_dev as for
 * ingot_attn_prefill. Replaces: a host-side loop over src/cpu_backend.cpp:51-69 for a block of tokens whose q rows
 * live in host memory. */
int ingot_attn_prefill_host(ingot_kv* kv, int layer, const void* q_host, int q_dtype, void* out_host, int out_dtype,
                            int n_head, int q_pos0, int n_tok, const int32_t* block_table_dev, int chunk_tokens,
                            void* stream);

/* Length-balanced assignment of n_seq sequences (key counts lens[]) to n_ranks GPUs for the sequence-sharded
 * batched decode: longest first, each to the least loaded rank (ties to the lower rank). rank_of_seq[i] receives
 * the rank of sequence i. Pure host code. */
int ingot_lpt_assign(const int32_t* lens, int n_seq, int n_ranks, int32_t* rank_of_seq);

/* ---- Host-buffer convenience call ---------------------------------------------------------------
 * One layer of the reference's attention stage with HOST inputs/outputs, as a CPU-side caller sees
 * it (q,k,v from the projections in; attention output for the wo projection out):
 * copies q/k/v f32 rows host->device, runs K1 then K3 (n_tok == 1) or K2 (n_tok > 1) on a contiguous
 * cache at positions pos0..pos0+n_tok-1, copies the f32 output device->host. All on `stream`,
 * asynchronous: call ingot_stream_sync (or cudaStreamSynchronize) before reading out_host.
 * Host buffers should be pinned for the copies to overlap. inv_freq_dev is a device pointer.
 * A single token whose q, k, v and output rows are all pinned, mapped and 16-byte aligned takes no copies: kernels read and write
 * the rows where they are. As with the copies, the input rows may change and the output rows hold the results once `stream` has been
 * synchronised, not before. */
int ingot_attn_layer_host(ingot_kv* kv, int layer, const float* q_host, const float* k_host, const float* v_host,
                          float* out_host, const float* inv_freq_dev, int n_head, int pos0, int n_tok,
                          void* stream);
/* The same for `layer_count` consecutive layers starting at `layer_begin` in one call, as the
 * reference's attention microbenchmark drives its backend (every layer's attention for one step,
 * src/metal_backend.mm:594-649): host arrays are [layer_count][n_tok][heads][128], one slice per layer.
 * If k_host directly follows q_host and v_host directly follows k_host in memory, rows that are copied travel in one copy. */
int ingot_attn_layers_host(ingot_kv* kv, int layer_begin, int layer_count, const float* q_host, const float* k_host,
                           const float* v_host, float* out_host, const float* inv_freq_dev, int n_head, int pos0,
                           int n_tok, void* stream);
int ingot_stream_sync(void* stream);

/* ---- Recurrent mixers and shared-row attention over a ragged batch ---------------------------------
 * No counterpart in the reference, whose models are attention-only with one sequence per call. A step carries, for each of
 * n_seq sequences, its next len tokens; the tokens are rows 0..n_tok-1 of every activation matrix, sequence after sequence.
 * All arrays are device memory (the struct itself is host memory, read during the call). */
typedef struct ingot_step {
    int n_tok, n_seq;
    int max_len;               /* host-side upper bound of len[] (sizes the launch grids) */
    const int32_t* row_seq;    /* [n_tok] sequence (index within the step) of each row */
    const int32_t* row_start;  /* [n_seq] first row */
    const int32_t* len;        /* [n_seq] */
    const int32_t* pos0;       /* [n_seq] position of the first token; 0 starts from the zero state whatever the slot holds */
    const int32_t* slot;       /* [n_seq] state slot */
} ingot_step;

/* Time chunks of a step for the recurrences: every sequence's len tokens cut into runs, sequence after sequence. */
typedef struct ingot_scan_plan {
    int n_chunks;
    int max_chunks;             /* most chunks any one sequence has: 1 = no chunk needs another's end state */
    const int32_t* chunk_seq;   /* [n_chunks] */
    const int32_t* chunk_t0;    /* [n_chunks] first token, counted from the sequence's first in this step */
    const int32_t* chunk_len;   /* [n_chunks] */
    const int32_t* seq_chunk0;  /* [n_seq + 1] */
    float* scratch_dev;         /* partial states; see the entry points for its size. May be null if max_chunks is 1 */
    size_t scratch_floats;
} ingot_scan_plan;

/* Where a kernel leaves an activation matrix [n_tok][ld]: f32 rows, and / or a bf16 plane, or a bf16 hi + lo pair (the
 * operands of the projection kernels). Null pointers are skipped. */
typedef struct ingot_act_out {
    float* f32;
    void *hi, *lo;
    int ld;
} ingot_act_out;

/* Per-channel causal convolution with carried history:
 *   out[t][c] = act(bias[c] + sum_j w[c][j] (in[t - (taps-1) + j][c] + in_bias[c])), zeros before position 0; act: none (silu 0), silu (1), or
 * silu from the hardware 2^x unit (2).
 * state_dev [slot][taps-1][channels]: the last taps-1 inputs (in + in_bias), oldest first; read and replaced. 1 <= taps <= 16.
 * in rows are in_ld floats apart; in_bias and bias may be null. */
int ingot_causal_conv(const ingot_step* step, const float* in_dev, int in_ld, const float* in_bias_dev, const float* w_dev,
                      const float* bias_dev, int taps, int channels, int silu, float* state_dev, const ingot_act_out* out,
                      void* stream);

/* States per channel as stored: n_state rounded up (at least to a multiple of 8); 0 if n_state is not supported (1..256). */
int ingot_scan_state_pad(int n_state);
/* Selective scan: with dt = softplus(dt_dev + dt_bias), per channel c and state n
 *   S[c][n] <- exp(dt A[c][n]) S[c][n] + dt x[c] B[n];  y[c] = sum_n S[c][n] C[n] + D[c] x[c];  out[c] = y[c] * silu(z[c]).
 * a_log2e_dev [inner][pad] = A * log2(e), zeros in the padding; B and C are the n_state columns at b_off / c_off of the rows of
 * bc_dev (pad columns are read, the ones beyond n_state must be finite). state_dev [slot][inner][pad] f32, read and replaced.
 * exact: decays through expm1, softplus and silu from expf / log1pf, instead of the hardware 2^x (see csrc/recurrent.cu).
 * Scratch: n_chunks * inner * (pad + 1) floats. inner, row lengths and offsets are multiples of 4. */
int ingot_selective_scan(const ingot_step* step, const ingot_scan_plan* plan, const float* x_dev, int x_ld, const float* dt_dev,
                         int dt_ld, const float* dt_bias_dev, const float* bc_dev, int bc_ld, int b_off, int c_off,
                         const float* z_dev, int z_ld, const float* a_log2e_dev, const float* d_dev, float* state_dev, int inner,
                         int n_state, int exact, const ingot_act_out* out, void* stream);

/* Real-gated linear recurrent unit with its output gate:
 *   r = sigmoid(g_r + r_bias), i = sigmoid(g_i + i_bias), log a = -8 r softplus(lam),
 *   S <- a S + sqrt(1 - a^2) i u;  out = out_scale * S * gelu_tanh(y + y_bias).
 * gates_dev rows hold, for each block of `block` channels, its g_r and then its g_i. state_dev [slot][width] f32, read and
 * replaced. exact: activations from expf / tanhf instead of the hardware 2^x unit. Scratch: 2 * n_chunks * width floats. */
int ingot_gated_lru(const ingot_step* step, const ingot_scan_plan* plan, const float* u_dev, int u_ld, const float* gates_dev,
                    int gates_ld, int block, const float* r_bias_dev, const float* i_bias_dev, const float* softplus_lam_dev,
                    const float* y_dev, int y_ld, const float* y_bias_dev, float* state_dev, int width, float out_scale,
                    int exact, const ingot_act_out* out, void* stream);

/* ---- Linear recurrences with a matrix state per head --------------------------------------------------
 * S_t = diag(a_t) S_(t-1) + k_t v_t^T, y_t = S_t^T q_t + skip v_t, S from zero at position 0. Decays (z: a raw product, z + bias):
 *   SIGMOID_POWER  one per state: a = sigmoid(z + bias) ^ power; bias [n_head][n_state]
 *   STEP           one per head: dt = softplus(z + bias), a = exp(-rate dt), and the input is dt k v^T; bias, rate [n_head] */
enum { INGOT_DECAY_SIGMOID_POWER = 0, INGOT_DECAY_STEP = 1 };
typedef struct ingot_linear_scan_in {
    int n_head, n_state, n_value;       /* states and values of a head as stored: multiples of 16, zero-padded; at most 512 states */
    int share;                          /* heads that share q and k: head h reads columns (h / share) * n_state.. of their rows */
    int decay;                          /* INGOT_DECAY_* */
    float q_scale, power;
    const float *q, *k, *v, *z;         /* rows q_ld.. floats apart (multiples of 4); v [head][n_value], z [head][n_state] or [head] */
    int q_ld, k_ld, v_ld, z_ld;
    const float *bias, *rate, *skip;    /* skip [n_head], may be null */
} ingot_linear_scan_in;
#define INGOT_LINEAR_SCAN_TILE_FROM 8
/* y [n_tok][y_ld], head h at column h * n_value. state_dev [slot][n_head][n_state][n_value] f32, read and replaced. min_len: a lower bound
 * of len[]. impl: 0 = library's choice (16-bit form: tensor cores for portions from INGOT_LINEAR_SCAN_TILE_FROM tokens on, up to 256
 * states), 1 = token by token in f32 (the exact form), 2 = tensor cores, 3 = the f32 kernel for portions of a few tokens (at most 7, a
 * power of two of values), which 0 and 1 use too. Chunks of the plan hold at least 8 tokens but for a sequence's last. Scratch: n_chunks * n_head * n_state * (n_value + 1) floats. */
int ingot_linear_scan(const ingot_step* step, const ingot_scan_plan* plan, const ingot_linear_scan_in* in, float* state_dev, float* y_dev, int y_ld,
                      int min_len, int impl, void* stream);
/* out = norm(x act(gate)) or norm(x) act(gate): rows of `heads` heads of `size` values stored `padded` apart (a multiple of 4), the RMS norm
 * over `parts` equal runs of the heads * size values, weight [heads * padded] (null: no norm). exact: activations from expf instead of the
 * hardware 2^x unit. The padding of x and gate holds finite numbers; that of the result is zero if x's or the weight's is. */
enum { INGOT_GATE_SILU = 0, INGOT_GATE_SIGMOID = 1 };
typedef struct ingot_gated_norm {
    const float *x, *gate, *weight;
    int x_ld, gate_ld, heads, size, padded, parts, act, gate_first, exact;
    float eps;
} ingot_gated_norm;
int ingot_gated_norm_rows(const ingot_gated_norm* norm, int n_rows, const ingot_act_out* out, void* stream);

/* Shared-row cache: one row per token and KV head is key and value at once (the value is the projection itself, the key the
 * projection normalised over all KV heads), paged in 16-position blocks, with causal or chunk-local visibility.
 * chunk > 0: position i sees j <= i of its own run of `chunk` positions counted from position 0; page of position p =
 * (p / chunk) * ceil(chunk / 16) + (p % chunk) / 16. chunk 0: plain causal, page p / 16. Rows [page][n_head_kv][16][head_dim]
 * f32 or f16 (head_dim a multiple of 4, <= 512, zero-padded heads allowed). Allocates on the current device; synchronous. */
typedef struct ingot_skv ingot_skv;
int ingot_skv_create(ingot_skv** out, int n_layer, int n_head_kv, int head_dim, int dtype, int chunk, int n_blocks);
void ingot_skv_destroy(ingot_skv* kv);
/* Pages that positions 0..n_positions-1 of one sequence span. */
int ingot_skv_pages(int chunk, int n_positions);
/* Row length to create an f16 cache with for heads of this size (the layout the tensor-core kernels take). */
int ingot_skv_row_length(int head_size);
/* The device status word itself, for callers that read several of them with their own copies. */
int* ingot_skv_status_dev(ingot_skv* kv);
/* Reads and clears the device status word (bit 2: a block-table entry outside the pool; the access was skipped). */
int ingot_skv_status(ingot_skv* kv, void* stream, int* status_out);
/* Query / key normalisation and append: columns q_off.. (n_head * head_dim) and k_off.. (n_head_kv * head_dim) of proj_dev's rows
 * (f32, proj_ld apart) are the projections, heads padded to head_dim with zeros, head_size their true size. Writes the cache rows
 * of the step's positions, and q_out_dev [n_tok][n_head][head_dim] in the cache's type: q / rms(q) * q_norm * k_norm, the key norm
 * weight folded in. q_norm_dev [n_head * head_dim], k_norm_dev [n_head_kv * head_dim], zero in the padding.
 * tables_dev [n_seq][max_blocks]: blocks of the step's sequences, entry 0 of a row being page first_page_dev[seq] (null: page 0). */
int ingot_skv_append(ingot_skv* kv, int layer, const ingot_step* step, const float* proj_dev, int proj_ld, int q_off, int k_off,
                     int n_head, int head_size, const float* q_norm_dev, const float* k_norm_dev, float eps, void* q_out_dev,
                     const int32_t* tables_dev, const int32_t* first_page_dev, int max_blocks, void* stream);
/* Softmax over the visible keys of every row (appended before), scores = q . k_row / rms(k) * scale; out[t][h * out_dim + d] =
 * out_scale * result for d < out_dim. impl: 0 = library's choice (tensor cores for f16 rows of the lengths
 * ingot_skv_row_length returns up to 256), 1 = the plain f32-arithmetic kernel, 2 = the warp-level tensor-core
 * kernel, 3 = the tcgen05 kernel (rows of 128 values). */
int ingot_skv_attend(ingot_skv* kv, int layer, const ingot_step* step, const void* q_dev, int n_head, int out_dim, float scale,
                     float out_scale, const ingot_act_out* out, const int32_t* tables_dev, const int32_t* first_page_dev, int max_blocks, int impl, void* stream);

/* The same cache for rows that are keys as they stand (no per-key scale), with a window that slides along: position i sees
 * i - window + 1 .. i (window 0: the whole past), page of position p = p / 16. row_length a multiple of 4, <= 1024. */
int ingot_skv_create_window(ingot_skv** out, int n_layer, int n_head_kv, int row_length, int dtype, int window, int n_blocks);

/* ---- Latent attention -------------------------------------------------------------------------------
 * One row per token for all heads: a normalised latent c (rank columns) and a rotated key part (rot columns), in a window-form
 * cache with one KV head. Lengths are as stored (padded with zeros); rank_count is the latent's true length. */
typedef struct ingot_latent_shape {
    int n_head, dim, rot;      /* per head: unrotated and rotated query columns, stored side by side */
    int rank, rank_count;
    int rot_dims;              /* rotated values, even, <= rot: i with i + rot_dims / 2; the rest of the part passes unchanged */
    float rot_gain;            /* factor of cosines and sines */
} ingot_latent_shape;
/* Columns q_off.. of proj_dev's rows: n_head x [dim | rot]; columns latent_off..: [rank | rot], the latent not yet normalised.
 * Writes the cache rows of the step's positions, the rotated query parts into q_rows_dev [n_tok][n_head][row length] (cache type;
 * may be null) and the unrotated query parts to q_plain [n_tok][n_head * dim]. turns_dev [rot_dims / 2]: turns per position
 * (base^(-2 i / rot_dims) / 2 pi). norm_dev [rank], zero in the padding. Tables as for ingot_skv_append.
 * From token long_from on the queries go to q_long_dev instead, f16 [n_tok][n_head][long_dim | long_rot], both parts zero-padded (the
 * operand of ingot_latent_attend_expanded; f16 caches only); null: no token does. */
int ingot_latent_append(ingot_skv* kv, int layer, const ingot_step* step, const float* proj_dev, int proj_ld, int q_off, int latent_off,
                        const ingot_latent_shape* shape, const float* norm_dev, float eps, const double* turns_dev, const ingot_act_out* q_plain,
                        void* q_rows_dev, void* q_long_dev, int long_from, int long_dim, int long_rot, const int32_t* tables_dev,
                        const int32_t* first_page_dev, int max_blocks, void* stream);
/* Latent queries f32 [n_tok][n_head * rank] into the first rank columns of the query rows. */
int ingot_latent_queries(const ingot_skv* kv, const float* q_dev, int n_tok, int n_head, int rank, void* q_rows_dev, void* stream);
/* out [n_tok][n_head * rank]: sum over the visible keys of softmax(q_row . row * scale) times the first rank columns of the row;
 * sink_dev [n_head] (may be null): one more term of each head's softmax sum, exp(sink), without a value. impl: 0 = library's choice, 1 = the plain f32-arithmetic
 * kernel, 2 = the warp-level tensor-core kernel (f16 rows, row length a multiple of 32, rank a multiple of 16 and at most 512), 3 =
 * the tcgen05 kernel (single tokens; f16 rows, row length a multiple of 64 and at least rank rounded up to 128, rank at most 512). */
int ingot_latent_attend(ingot_skv* kv, int layer, const ingot_step* step, const void* q_rows_dev, int n_head, int rank, float scale,
                        const float* sink_dev, const ingot_act_out* out, const int32_t* tables_dev, const int32_t* first_page_dev, int max_blocks,
                        int impl, void* stream);

/* The same for long portions, on keys and values computed from the cached latents (f16, tcgen05). For each sequence of the step
 * the keys it sees - positions key_pos .. the portion's last - are rows key0, key0 + 1, .. of two buffers.
 * ingot_latent_gather fetches them from the cache: latents [key][rank], rotated parts [key][rot_ld] (zero-padded); max_keys: the
 * most any sequence of the step has. The expansion of the latents is a product (ingot_linear_tc_run_f16 of the backend). */
int ingot_latent_gather(ingot_skv* kv, int layer, const ingot_step* step, const int32_t* key0_dev, const int32_t* key_pos_dev,
                        int max_keys, int rank, int rot, void* latent_dev, void* rotated_dev, int rot_ld, const int32_t* tables_dev,
                        const int32_t* first_page_dev, int max_blocks, void* stream);
typedef struct ingot_latent_expansion {
    const void* q;              /* f16 [q_rows][n_head][dim | rot], row t = token t of the step */
    const void* kv;             /* f16 [key_rows][n_head][dim | v]: unrotated keys and values */
    const void* rotated;        /* f16 [key_rows][rot] */
    long long q_rows, key_rows; /* rows of the buffers (all of them hold finite numbers) */
    int n_head, dim, rot, v;    /* padded parts: multiples of 64, dim + rot <= 256, v <= 128 */
    const int32_t *key0, *key_pos; /* device, per sequence */
    const float* gate;          /* may be null: the result times sigmoid(z), z at gate[t * gate_ld + column of the result] */
    int gate_ld;                /* a multiple of 4 */
} ingot_latent_expansion;
/* out [n_tok][n_head * out_dim], out_dim <= v. */
int ingot_latent_attend_expanded(ingot_skv* kv, const ingot_step* step, const ingot_latent_expansion* x, float scale,
                                 const float* sink_dev, int out_dim, const ingot_act_out* out, void* stream);

/* ---- Grouped-query attention over joined rows -------------------------------------------------------
 * A window-form cache whose rows are [key | value] of one token and KV head side by side, in plain page order. */
int ingot_skv_create_joined(ingot_skv** out, int n_layer, int n_head_kv, int row_length, int dtype, int window, int n_blocks);
/* RMS norm of queries and keys before rotation: none, over each head with one weight [dim] for all, or over the whole projection with a
 * weight [heads][dim]. Weights are zero in the padding. */
enum { INGOT_QK_NORM_NONE = 0, INGOT_QK_NORM_HEAD = 1, INGOT_QK_NORM_ALL = 2 };
typedef struct ingot_gqa_shape {
    int n_head, n_head_kv;
    int dim, vdim;   /* stored columns of a query / key and of a value head, zero-padded; dim + vdim is the row length */
    int dim_count;   /* true size of a query / key head */
    int rot_dims;    /* rotated values of a head, even: pairs (2 i, 2 i + 1); the rest passes unchanged */
    int norm;        /* INGOT_QK_NORM_* */
} ingot_gqa_shape;
/* Columns q_off.. (n_head * dim), k_off.. (n_head_kv * dim) and v_off.. (n_head_kv * vdim) of proj_dev's rows. Writes the cache rows of the
 * step's positions and the queries, q_out_dev [n_tok][n_head][dim] in the cache's type. turns_dev [rot_dims / 2]: turns per position;
 * cosine and sine are multiplied by rot_gain. first_values_dev [n_tok][n_head_kv * vdim] (null: nothing is mixed): store_first != 0
 * stores the values there, else they become (1 - mix) v + mix * stored before they are cached. Tables as for ingot_skv_append. */
int ingot_gqa_append(ingot_skv* kv, int layer, const ingot_step* step, const float* proj_dev, int proj_ld, int q_off, int k_off, int v_off,
                     const ingot_gqa_shape* shape, const float* q_norm_dev, const float* k_norm_dev, float eps, const double* turns_dev, float rot_gain,
                     float* first_values_dev, int store_first, float mix, void* q_out_dev, const int32_t* tables_dev, const int32_t* first_page_dev,
                     int max_blocks, void* stream);
/* out [n_tok][n_head * vdim]: the softmax average of the visible values, scores q . k * scale. sink_dev [n_head] (may be null): one more
 * term exp(sink) of a head's softmax sum. gate_dev (may be null): the result times sigmoid(z), z at gate_dev[t * gate_ld + ...], one per
 * head or one per result column. impl: 0 = library's choice, 1 = the plain f32-arithmetic kernel, 2 = the warp-level tensor-core kernel
 * with split keys (f16, sizes that are multiples of 16 and at most 256), 3 = the tcgen05 kernel (f16, sizes that are multiples of 16,
 * keys at most 256, values at most 128, scale > 0), which 0 takes for portions of several tokens when the step's sequences, each as long
 * as the longest, have INGOT_GQA_LONG_ROWS (token, head) pairs. The step may be some sequences of a larger one: n_seq and the per-sequence
 * arrays are theirs, n_tok and the rows those of the whole. */
#define INGOT_GQA_LONG_ROWS 2560
int ingot_gqa_attend(ingot_skv* kv, int layer, const ingot_step* step, const void* q_dev, const ingot_gqa_shape* shape, float scale, const float* sink_dev,
                     const float* gate_dev, int gate_ld, int gate_per_head, const ingot_act_out* out, const int32_t* tables_dev, const int32_t* first_page_dev,
                     int max_blocks, int impl, void* stream);

/* ---- Mixture of experts -----------------------------------------------------------------------------
 * Pair p = token * top + k is a token's k-th expert; rows are the pairs sorted by expert, in token order within one. */
enum { INGOT_ACT_NONE = 0, INGOT_ACT_RELU2 = 1, INGOT_ACT_SILU_GATED = 2 };  /* RELU2: the square of relu; SILU_GATED: silu(gate) * up */
/* The top experts of each token by logit (the lower index of equal ones) with sigmoid(logit) as weight, and their sorting:
 * expert_of, weight_of, row_of [n_tok * top] by pair, pair_of, row_weight [n_tok * top] by row, group_start [n_expert + 1]. */
int ingot_moe_route(const float* logits_dev, int ld, int n_tok, int n_expert, int top, int32_t* expert_of_dev, float* weight_of_dev,
                    int32_t* group_start_dev, int32_t* row_of_dev, int32_t* pair_of_dev, float* row_weight_dev, void* stream);
/* Routers over n_expert experts and n_identity identity experts behind them (whose output is the token's own input): scores are the softmax
 * of all the logits, choices the `top` largest of score + correction within the `keep` best of `groups` equal runs of neighbours (a run is
 * as good as its best choice), weights the scores of the chosen over their sum (+ 1e-20), times scale. At most 1024 outputs. */
typedef struct ingot_moe_router {
    int n_expert, n_identity, top, groups, keep;
    float scale;
    const float* correction;  /* device, [n_expert + n_identity]; may be null */
} ingot_moe_router;
/* As ingot_moe_route. Pairs of identity experts have no row: row_of is -1, their weights add up in self_gain_dev [n_tok], and only the
 * first group_start[n_expert] rows exist. shared_gain_dev [n_tok] (may be null): sigmoid of the logit behind the router's. */
int ingot_moe_route_grouped(const ingot_moe_router* router, const float* logits_dev, int ld, int n_tok, int32_t* expert_of_dev, float* weight_of_dev,
                            int32_t* group_start_dev, int32_t* row_of_dev, int32_t* pair_of_dev, float* row_weight_dev, float* self_gain_dev,
                            float* shared_gain_dev, void* stream);
/* The same without a router: table_dev [vocabulary][top] holds each token id's experts (0..n_expert-1; one that is named twice counts twice), tokens_dev
 * [n_tok] the ids; every pair weighs `weight`. expert_of and weight_of may be left unwritten. */
int ingot_moe_route_table(const int32_t* table_dev, const int32_t* tokens_dev, int n_tok, int n_expert, int top, float weight, int32_t* expert_of_dev,
                          float* weight_of_dev, int32_t* group_start_dev, int32_t* row_of_dev, int32_t* pair_of_dev, float* row_weight_dev, void* stream);
/* bf16 planes [n_rows][n] of the rows from planes [n_tok][n] of the tokens (lo may be null). n a multiple of 8. n_rows_dev (may be null):
 * how many of the n_rows rows exist. */
int ingot_moe_gather(void* hi_dev, void* lo_dev, const void* src_hi_dev, const void* src_lo_dev, const int32_t* pair_of_dev, int n_rows,
                     const int32_t* n_rows_dev, int top, int n, void* stream);
/* out[row] = act(row_weight[row] * W_e x), W bf16 [n_expert][n_out][n_in], f32 arithmetic. x row of a row: its token's
 * (pair_of_dev given) or its own; row_weight_dev may be null. SILU_GATED: out[row] = row_weight[row] * silu(gate) * up, n_out a multiple of
 * 32, W [n_expert][2 n_out][n_in] with each 32 gate rows followed by the 32 up rows of the same outputs. */
int ingot_moe_linear(float* out_dev, const void* w_dev, const float* x_dev, int x_ld, int n_in, int n_out, int n_expert, int n_rows,
                     const int32_t* group_start_dev, const int32_t* pair_of_dev, int top, const float* row_weight_dev, int act, void* stream);
/* x [n_tok][n] += the sum of each token's rows of [n_tok * top][n] (row_of_dev null, top 1: its own). */
int ingot_moe_add(float* x_dev, const float* rows_dev, const int32_t* row_of_dev, int n_tok, int top, int n, void* stream);

/* ---- Diagnostics ----------------------------------------------------------------------------------
 * HBM read-bandwidth probe: what the reference's `bwtest` verb measures (src/main.cpp:450-455,
 * MetalBackend::bandwidth_test src/metal_backend.mm:533-592 with the bw_fill / bw_sum kernels,
 * shaders/kernels.metal:949-991). Allocates `bytes` on the current device, fills them, then times a kernel
 * that only reads them with 16-byte streaming loads, `reps` times; *best_seconds receives the fastest pass
 * (bandwidth = bytes / *best_seconds). Synchronous. Sizes beyond the L2 (126 MB) measure HBM. */
int ingot_hbm_read_probe(size_t bytes, int reps, double* best_seconds, void* stream);

#ifdef __cplusplus
}
#endif
#endif /* INGOT_CUDA_H */
