// What the layers of a model folder are written in: projections (with the norm of their input or the residual add of their
// output folded in), scratch activations, weight upload, state and cache groups; and the interfaces of a layer's two parts.
//
// Precision. Weights are bf16. In the 16-bit form the tensor-core products take bf16 activations (a hi + lo pair where the
// product feeds a recurrence's gates or step sizes, and in small batches) and accumulate in f32; everything between products - residual stream,
// norms, scores and softmax, gates, recurrent states, router scores - is f32, and single tokens multiply f32 activations. In the f32 form
// every product is f32 FMA on widened weights and the attention cache is f32.
//
// Padding. Every vector is stored with a length that is a multiple of 8 (heads and gate blocks each padded on their own):
// padded weight rows and columns are zero, so padded activations are zero and only means need the true count.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <numeric>
#include <string>
#include <utility>
#include <vector>

#include "block_pool.h"
#include "cuda_util.h"
#include "grouped_linear.h"
#include "ingot_cuda.h"
#include "model_registry.h"
#include "residual_norm.h"
#include "weight_streamer.h"
#include "../csrc/scan_routes.h"

extern "C" {
cudaError_t ingot_support_embed_rows_bf16(float* out, const void* table, int n_in, int n_rows_table, const int32_t* rows_dev, int n_rows,
                                          float scale, int* status_dev, cudaStream_t s);
cudaError_t ingot_support_embed_sum_bf16(float* out, float* copy, const void* table, int n_rows_table, const int32_t* rows_dev, const void* table2,
                                         int n_rows_table2, const int32_t* rows2_dev, int n_in, int n_rows, float scale, int* status_dev, cudaStream_t s);
cudaError_t ingot_support_concat_rows(float* f32, void* hi, void* lo, const float* a, const float* b, int n, int n_rows, cudaStream_t s);
cudaError_t ingot_support_deliver(float* const* dst_at, const float* src, int src_ld, int n, int rows, int* status, int* const* words, int n_words, cudaStream_t s);
cudaError_t ingot_support_fetch(void* dst, const void* src, size_t n, cudaStream_t s);
cudaError_t ingot_support_softcap(float* x, size_t n, float cap, cudaStream_t s);
cudaError_t ingot_support_rmsnorm_rows(float* out, const float* x, const float* w, const int32_t* rows_dev, int n_rows, int n, int n_mean,
                                       float eps, cudaStream_t s);
cudaError_t ingot_support_linear_bf16(float* out, const void* w, const float* x, int x_ld, int n_in, int n_out, int rows_per_block,
                                      int n_tok, int accumulate, cudaStream_t s);
cudaError_t ingot_support_gemv_bf16(float* out, const void* w, int n_out, int n_in, const float* x, const float* norm_w, float eps, int n_mean,
                                    int gated, int act, int accumulate, cudaStream_t s);
cudaError_t ingot_support_gated_act(float* out, const float* in, int n_rows, int n, int act, cudaStream_t s);
struct ingot_linear_ws;
cudaError_t ingot_linear_ws_create_bf16(ingot_linear_ws** out, int max_tok, int max_in, int max_out);
void ingot_linear_ws_destroy(ingot_linear_ws* ws);
int* ingot_linear_ws_status_dev(ingot_linear_ws* ws);
const float* ingot_linear_ws_slices(const ingot_linear_ws* ws, int slot, int* n_slices);
void ingot_linear_ws_planes(ingot_linear_ws* ws, void** hi, void** lo);
cudaError_t ingot_linear_tc_prepared(ingot_linear_ws* ws, int n_in, int n_tok, int planes);
cudaError_t ingot_linear_tc_prepare_bf16(ingot_linear_ws* ws, const float* x, int x_ld, int n_in, int n_tok, int planes, cudaStream_t s);
cudaError_t ingot_linear_tc_prepare_norm_bf16(ingot_linear_ws* ws, const float* x, const float* norm_w, float eps, int n_in, int n_mean, int n_tok,
                                              int planes, cudaStream_t s);
cudaError_t ingot_linear_tc_run(ingot_linear_ws* ws, float* out, const void* w, int n_in, int n_out, int accumulate, cudaStream_t s);
cudaError_t ingot_linear_tc_run_to(ingot_linear_ws* ws, float* out, float* const* out_at, const void* w, int n_in, int n_out, int* there, cudaStream_t s);
cudaError_t ingot_linear_tc_run_blocks(ingot_linear_ws* ws, float* out, const void* w, int k_block, int n_out, int rows_per_block, cudaStream_t s);
cudaError_t ingot_linear_tc_run_partial(ingot_linear_ws* ws, const void* w, int n_in, int n_out, int slot, cudaStream_t s);
cudaError_t ingot_linear_tc_run_half(ingot_linear_ws* ws, void* out, int out_ld, int out_block, const void* w, int n_in, int n_out, int rows_per_block,
                                     cudaStream_t s);
cudaError_t ingot_linear_tc_run_f16(ingot_linear_ws* ws, void* out, int out_ld, const void* a, int a_rows, int n_tok, const void* w, int n_in, int n_out,
                                    cudaStream_t s);
cudaError_t ingot_linear_tc_finish_residual_norm_bf16(ingot_linear_ws* ws, float* x, const float* norm_w, float eps, int n_mean, int planes,
                                                      const float* pair_rows, const int32_t* row_of, int top, cudaStream_t s);
cudaError_t ingot_linear_tc_run_gated_bf16(ingot_linear_ws* ws, const void* w, int n_in, int n_out, int act, int planes, cudaStream_t s);
}

inline constexpr int kMinTcTokens = 2;  // from two tokens on, a product on the tensor cores streams the weights once, whatever rows are padding

// Up to this many tokens a product is bound by streaming the weights, so the activations go in as a hi + lo pair at no cost: a
// decoded token's logits then hardly depend on whether it is alone (f32 activations) or in a batch.
inline constexpr int kPairTokens = 64;

inline int round_up(int v, int q) { return (v + q - 1) / q * q; }

inline int get_int(const Json& j, const char* key, int lo = 1, int hi = 1 << 28) {
    const int64_t v = j.at(key).integer();
    if (v < lo || v > hi) throw std::runtime_error(std::string("model config: \"") + key + "\" is out of range");
    return int(v);
}
inline float get_float(const Json& j, const char* key) { return float(j.at(key).number()); }
inline bool has(const Json& j, const char* key) { return j.has(key) && !j.at(key).is_null(); }

// A kind of grouped-query attention layer: what the design fixes about it; its sizes, rotation, window and value mixing come from the
// configuration.
enum class OutputGate { none, per_head, per_value };
struct AttentionKind {
    const char* type;  // name in the configuration
    int qk_norm;       // INGOT_QK_NORM_*
    bool sink;
    OutputGate gate;
};

// The same for latent attention.
struct LatentKind {
    bool sink = true;
    bool gate = false;    // the heads side by side times sigmoid(W_g h)
    bool paired = false;  // rotation of neighbouring values instead of value i with value i + dims / 2
};

// What a design fixes and its configuration does not say.
struct Design {
    float norm_offset = 0.f;     // the norms' weights are stored around this: x / rms(x) * (norm_offset + w)
    bool centred = false;        // norms over the residual are layer norms with a bias (tensor NAME.b) instead of RMS norms
    bool sandwich = false;       // a part's result is normed too before the residual sum (tensors norm1b, norm2b)
    bool parallel = false;       // a layer adds mixer(norm1 x) + ff(norm2 x), both of the same x, instead of one after the other
    bool tied_head = false;      // the output matrix is the embedding table
    int act = 1;                 // of gated feed-forwards: 0 silu, 1 the tanh form of gelu
    bool gated_experts = false;  // experts are gated (silu) and weighed by a softmax router, instead of squared-relu ones by sigmoid scores
    bool table_experts = false;  // gated experts without a router: a table gives every token id its own, all of equal weight
    bool loop_step = false;      // a pass of the loop begins by adding a vector of its own, instead of a product of x and the embedding
    std::vector<AttentionKind> attention = {};
    LatentKind latent = {};
};

// A norm over the residual's length as it is uploaded: RMS (over the whole row or in groups), or centred if it has a bias. With `conv`, what
// is read through it is h + conv(h), h the normed rows: a causal convolution per channel over the sequence (the taps hold the sum).
struct Norm : ingot_norm {
    float *conv = nullptr, *conv_state = nullptr;
    int pass = 0;  // of the loop: whose state the convolution goes on from
    Norm() : ingot_norm{nullptr, nullptr, 1} {}
    explicit operator bool() const { return w != nullptr; }
    Norm of_pass(int p) const {
        Norm n = *this;
        n.pass = p;
        return n;
    }
    bool apart() const { return b || groups > 1 || conv; }  // taken by a launch of its own: products only fold in plain RMS norms
    bool operator==(const Norm& o) const { return w == o.w; }
};
// The norms around one part of a layer: of its input, of its result before the residual sum (may be none), and the one that reads the
// residual stream next (none: something else happens to it first).
struct Norms { Norm in, post, next; };

// A dimension of n groups of `size` values, each stored with `padded` places.
struct Groups {
    int n, size, padded;
    int count() const { return n * size; }
    int width() const { return n * padded; }
};
inline Groups flat(int size) { return {1, size, round_up(size, 8)}; }

// A bf16 matrix on the device, [n_out][n_in] row-major, both padded. rows_per_block > 0: block-diagonal, n_in per block.
struct Matrix {
    void* data = nullptr;
    int n_out = 0, n_in = 0, rows_per_block = 0;
    const void* rows_from(int r) const { return static_cast<const char*>(data) + size_t(r) * n_in * 2; }
};

// One tensor's place in a matrix: its logical rows (from row src_row0 on; groups src_stride rows apart, 0: side by side) and columns
// go to r0 + row groups, c0 + column groups.
struct Part {
    std::string name;
    std::vector<int64_t> shape;
    Groups rows, cols;
    int r0 = 0, c0 = 0, src_row0 = 0, src_stride = 0;
};

enum Buf { kProj, kConv, kStateIn, kDt, kGates, kMix, kGateUp, kMid, kNormed, kQuery, kQueryPlain, kQueryLong, kLatent, kValue, kRouter, kExpertIn, kExpertMid, kExpertOut,
           kBranch, kConcat, kFirstValue, kConvIn, kBufCount };

// The step as the launches see it.
struct StepCtx {
    ingot_step st = {};
    // Time chunks, by LayerOps::scan_plan: one part for all sequences of the step, or one for the short ones and one for the others.
    struct ScanPart { ingot_step st; ingot_scan_plan plan; };
    std::vector<std::vector<ScanPart>> plans;
    const int32_t* lens = nullptr;  // host copy of st.len; sequences come in ascending order of it
    const int32_t* tokens = nullptr;  // device: the token id of each row
    bool tc = false;  // products on the tensor cores (16-bit form, more than one token)
    int planes = 1;   // bf16 planes an activation is given as there
};

// Shared-row attention caches of equal shape and visibility live in one handle with one page pool.
struct CacheGroup {
    int kv_heads, dim, chunk, window;  // visibility: own chunk, sliding window (one of them 0), or the whole past
    enum Form { scaled, plain, joined } form;  // rows with a key scale of their own (ingot_skv_create), without (ingot_skv_create_window), [key | value]
    int n_layer = 0;
    ingot_skv* kv = nullptr;
    BlockPool pool;
    int pages_per_chunk = 0;
    const int32_t *tables = nullptr, *first_page = nullptr;  // device, of the current step
    int width = 0;
    // Portions that run on keys expanded per head (latent attention): from how many tokens on (0: none), how many keys at a time, and
    // of the current step the first sequence that does, the runs of sequences that are expanded together, and where their keys go.
    int expand_from = 0, key_rows = 0, first_long = 0;
    struct Expansion { int seq0, n_seq, n_keys, most_keys; };
    std::vector<Expansion> expansions;
    const int32_t *key0 = nullptr, *key_pos = nullptr;       // device, per sequence
    int page(int pos) const { return ingot_skv_pages(chunk, pos + 1) - 1; }
    int first_visible(int pos) const { return chunk > 0 ? pos / chunk * chunk : window > 0 && pos >= window ? pos - window + 1 : 0; }
    bool forgets() const { return chunk > 0 || window > 0; }  // pages fall out of sight for good
    int pages_seen() const { return chunk > 0 ? pages_per_chunk : (window + INGOT_BLOCK_TOKENS - 2) / INGOT_BLOCK_TOKENS + 1; }  // at most, by one token
};

// What a feed-forward branch leaves for the residual sum: rows of the residual's length, token t's at row_of[t * top + k].
struct Branch {
    const float* rows = nullptr;
    const int32_t* row_of = nullptr;  // null: row t
    int top = 1;
};

class LayerOps {
public:
    LayerOps(const ModelDir& dir, const EngineOptions& opt, const Design& design, int max_step) : dir(dir), opt(opt), design(design), max_step(max_step) {
        cuda_check(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
    }
    ~LayerOps() {
        cudaStreamSynchronize(stream);
        ingot_linear_ws_destroy(ws);
        for (void* p : allocs_) cudaFree(p);
        cudaStreamDestroy(stream);
    }

    // ---- construction ----
    void* alloc(size_t bytes, bool zero = false) {
        void* p = nullptr;
        cuda_check(cudaMalloc(&p, std::max<size_t>(bytes, 16)), "cudaMalloc");
        allocs_.push_back(p);
        if (zero) cuda_check(cudaMemset(p, 0, std::max<size_t>(bytes, 16)), "cudaMemset");
        return p;
    }
    void need(Buf b, int columns) { columns_[b] = std::max(columns_[b], columns); }
    void need_keys(size_t latents, size_t rotated, size_t expanded) {
        const size_t bytes[3] = {latents, rotated, expanded};
        for (int i = 0; i < 3; i++) key_bytes_[i] = std::max(key_bytes_[i], bytes[i]);
    }
    void tc_shape(int n_in, int n_out) { tc_in_ = std::max(tc_in_, n_in); tc_out_ = std::max(tc_out_, n_out); }
    void allocate() {
        for (int b = 0; b < kBufCount; b++) bufs_[b] = columns_[b] ? static_cast<float*>(alloc(size_t(max_step) * columns_[b] * 4, true)) : nullptr;
        for (int i = 0; i < 3; i++) keys_[i] = key_bytes_[i] ? alloc(key_bytes_[i], true) : nullptr;
        if (!opt.f32 && max_step >= kMinTcTokens) cuda_check(ingot_linear_ws_create_bf16(&ws, max_step, tc_in_, tc_out_), "linear workspace");
        loader_.finish();
        cuda_check(cudaDeviceSynchronize(), "model upload");
    }
    float* upload(const std::vector<float>& v) {
        float* d = static_cast<float*>(alloc(v.size() * 4));
        cuda_check(cudaMemcpy(d, v.data(), v.size() * 4, cudaMemcpyHostToDevice), "cudaMemcpy");
        return d;
    }
    // A vector tensor with each group padded with zeros.
    std::vector<float> host_vector(const std::string& name, const std::vector<int64_t>& shape, Groups g) {
        const std::vector<float> v = tensor_f32(dir.tensor(name, shape));
        if (int(v.size()) != g.count()) throw std::runtime_error("model: tensor " + name + " does not have " + std::to_string(g.count()) + " values");
        std::vector<float> out(size_t(g.width()), 0.f);
        for (int i = 0; i < g.n; i++) std::copy(v.begin() + i * g.size, v.begin() + (i + 1) * g.size, out.begin() + i * g.padded);
        return out;
    }
    float* vector(const std::string& name, const std::vector<int64_t>& shape, Groups g) { return upload(host_vector(name, shape, g)); }
    float* vector(const std::string& name, int n) { return vector(name, {n}, flat(n)); }
    // A norm over the residual stream as the design stores it (RMS weights around norm_offset, or weight and bias); its result times `gain`.
    Norm norm(const std::string& name, float gain = 1.f) {
        Norm n;
        n.groups = norm_groups;
        auto load = [&](const std::string& tensor, float offset) {
            std::vector<float> v = host_vector(tensor, {width}, flat(width));
            for (int i = 0; i < width; i++) v[size_t(i)] = (v[size_t(i)] + offset) * gain;
            return upload(v);
        };
        n.w = load(name, design.norm_offset);
        if (design.centred) n.b = load(name + ".b", 0.f);
        return n;
    }
    // The norm a part of a layer reads the residual stream through, with the input convolution (tensor `conv_name`) where there is one.
    Norm input_norm(const std::string& name, const std::string& conv_name) {
        Norm n = norm(name);
        if (input_taps == 0) return n;
        const int d = round_up(width, 8);
        const std::vector<float> w = tensor_f32(dir.tensor(conv_name, {width, input_taps}));
        std::vector<float> padded(size_t(d) * input_taps, 0.f);
        std::copy(w.begin(), w.end(), padded.begin());
        for (int c = 0; c < width; c++) padded[size_t(c) * input_taps + size_t(input_taps) - 1] += 1.f;
        n.conv = upload(padded);
        n.conv_state = state(size_t(input_taps - 1) * d);
        need(kConvIn, d);
        return n;
    }
    float scalar(const std::string& name) {
        const TensorView& t = dir.tensor(name);
        if (t.elems() != 1) throw std::runtime_error("model: tensor " + name + " is not one number");
        return tensor_f32(t)[0];
    }
    const TensorView& bf16(const std::string& name, const std::vector<int64_t>& shape) const {
        const TensorView& t = dir.tensor(name, shape);
        if (t.dtype != "BF16") throw std::runtime_error("model: tensor " + name + " has type " + t.dtype + ", expected BF16");
        return t;
    }
    // grouped: a stack of matrices for ingot_grouped_tc_run, whose results do not pass through the workspace
    Matrix matrix(int n_out, int n_in, const std::vector<Part>& parts, int rows_per_block = 0, bool grouped = false) {
        std::vector<uint16_t> host(size_t(n_out) * n_in, 0);
        for (const Part& p : parts) {
            const TensorView& t = bf16(p.name, p.shape);
            const int stride = p.src_stride ? p.src_stride : p.rows.size;
            if (t.elems() < int64_t(p.src_row0 + (p.rows.n - 1) * stride + p.rows.size) * p.cols.count() || t.elems() % p.cols.count() != 0)
                throw std::runtime_error("model: tensor " + p.name + " has an unexpected size");
            const int nr = p.rows.count();
            for (int r = 0; r < nr; r++) {
                uint16_t* dst = host.data() + size_t(p.r0 + r / p.rows.size * p.rows.padded + r % p.rows.size) * n_in + p.c0;
                const unsigned char* src = t.data + size_t(p.src_row0 + r / p.rows.size * stride + r % p.rows.size) * p.cols.count() * 2;
                for (int g = 0; g < p.cols.n; g++) memcpy(dst + g * p.cols.padded, src + size_t(g) * p.cols.size * 2, size_t(p.cols.size) * 2);
            }
        }
        return matrix(host, n_out, n_in, rows_per_block, grouped);
    }
    Matrix matrix(const std::vector<uint16_t>& host, int n_out, int n_in, int rows_per_block, bool grouped = false) {
        Matrix m;
        m.n_out = n_out;
        m.n_in = n_in;
        m.rows_per_block = rows_per_block;
        m.data = alloc(host.size() * 2);
        loader_.copy(m.data, host.data(), host.size() * 2);
        weight_bytes += host.size() * 2;
        if (!grouped) tc_shape(rows_per_block > 0 ? n_in * (n_out / rows_per_block) : n_in, n_out);
        return m;
    }
    Matrix matrix(const std::string& name, Groups rows, Groups cols) {
        return matrix(rows.width(), cols.width(), {Part{name, {rows.count(), cols.count()}, rows, cols}});
    }

    // ---- the step ----
    float* buf(Buf b) const { return bufs_[b]; }
    void* keys(int i) const { return keys_[i]; }  // 0 latents, 1 rotated parts, 2 expanded keys and values
    // Output of a kernel that feeds a product: the operand planes on the tensor-core path (and f32 rows if `keep`), else f32.
    ingot_act_out operand(const StepCtx& s, float* f32, int ld, bool keep, int planes = 0) const {
        ingot_act_out o = {};
        o.ld = ld;
        if (!s.tc || keep) o.f32 = f32;
        if (s.tc) {
            ingot_linear_ws_planes(ws, &o.hi, &o.lo);
            if (std::max(planes, s.planes) < 2) o.lo = nullptr;
        }
        return o;
    }
    void operand_ready(const StepCtx& s, int n_in, int planes = 0) const {
        if (s.tc) cuda_check(ingot_linear_tc_prepared(ws, n_in, s.st.n_tok, std::max(planes, s.planes)), "operand");
    }
    static bool streams(const Matrix& w) { return w.n_in % 256 == 0 && w.n_in <= 12032 && w.rows_per_block == 0; }

    // out [n_tok][w.n_out] = W norm(x)
    void norm_project(const StepCtx& s, float* out, const Matrix& w, const Norm& norm) {
        if (s.tc) {
            prepare_norm(s, w, norm);
            cuda_check(ingot_linear_tc_run(ws, out, w.data, w.n_in, w.n_out, 0, stream), "projection");
        } else if (s.st.n_tok == 1 && streams(w) && !norm.apart()) {
            cuda_check(ingot_support_gemv_bf16(out, w.data, w.n_out, w.n_in, x, norm.w, eps, width, 0, 0, 0, stream), "projection");
        } else {
            norm_rows(s, norm);
            project(s, out, w, buf(kNormed), w.n_in);
        }
    }
    // out = W in. Tensor-core path: the operand planes must hold `in` (operand_ready).
    void project(const StepCtx& s, float* out, const Matrix& w, const float* in, int in_ld) {
        if (s.tc) {
            if (w.rows_per_block > 0) cuda_check(ingot_linear_tc_run_blocks(ws, out, w.data, w.n_in, w.n_out, w.rows_per_block, stream), "block projection");
            else cuda_check(ingot_linear_tc_run(ws, out, w.data, w.n_in, w.n_out, 0, stream), "projection");
        } else if (s.st.n_tok == 1 && streams(w) && w.n_out > 2048) {  // few rows: ingot_support_linear_bf16 gives each a CTA
            cuda_check(ingot_support_gemv_bf16(out, w.data, w.n_out, w.n_in, in, nullptr, 0.f, w.n_in, 0, 0, 0, stream), "projection");
        } else {
            cuda_check(ingot_support_linear_bf16(out, w.data, in, in_ld, w.n_in, w.n_out, w.rows_per_block, s.st.n_tok, 0, stream), "projection");
        }
    }
    // Tensor-core path: f32 rows become the operand planes.
    void prepare_rows(const StepCtx& s, const float* in, int in_ld, int n_in, int planes = 0) const {
        cuda_check(ingot_linear_tc_prepare_bf16(ws, in, in_ld, n_in, s.st.n_tok, std::max(planes, s.planes), stream), "operand");
    }
    // The same for f32 rows that are not in the planes yet.
    void project_rows(const StepCtx& s, float* out, const Matrix& w, const float* in, int in_ld, int planes) {
        if (s.tc) prepare_rows(s, in, in_ld, w.n_in, planes);
        project(s, out, w, in, in_ld);
    }
    // x += post(W in); n.next: the norm that the following product reads x through, folded into the same kernel.
    void project_residual(const StepCtx& s, const Matrix& w, const float* in, const Norms& n) {
        if (n.post || n.next.apart()) {
            ingot_residual_norm r = {};
            product(s, w, in, r);
            finish(s, r, n);
            add_branch(s);
            return;
        }
        norm_ready_ = Norm();
        if (s.tc) {
            cuda_check(ingot_linear_tc_run_partial(ws, w.data, w.n_in, w.n_out, 0, stream), "output projection");
            cuda_check(ingot_linear_tc_finish_residual_norm_bf16(ws, x, n.next.w, eps, width, s.planes, branch_.rows, branch_.row_of, branch_.top, stream), "residual");
            norm_ready_ = n.next;
            branch_ = Branch();
            return;
        }
        if (s.st.n_tok == 1 && streams(w)) {
            cuda_check(ingot_support_gemv_bf16(x, w.data, w.n_out, w.n_in, in, nullptr, 0.f, w.n_in, 0, 0, 1, stream), "output projection");
        } else {
            cuda_check(ingot_support_linear_bf16(x, w.data, in, w.n_in, w.n_in, w.n_out, 0, s.st.n_tok, 1, stream), "output projection");
        }
        add_branch(s);
    }
    // W in as the product of a residual sum (finish): slices in the workspace, or rows of kBranch.
    void product(const StepCtx& s, const Matrix& w, const float* in, ingot_residual_norm& r) {
        if (s.tc) {
            cuda_check(ingot_linear_tc_run_partial(ws, w.data, w.n_in, w.n_out, 0, stream), "output projection");
            r.product = ingot_linear_ws_slices(ws, 0, &r.n_slices);
        } else {
            project(s, buf(kBranch), w, in, w.n_in);
            r.product = buf(kBranch);
            r.n_slices = 1;
        }
    }
    // x += post(the terms of r), and next(x) for the part that follows.
    void finish(const StepCtx& s, ingot_residual_norm& r, const Norms& n) {
        norm_ready_ = Norm();
        r.post = n.post;
        if (n.next.apart()) r.next = n.next;  // plain RMS norms are folded into the products that read through them
        residual_norm(s, r, n.next);
        if (n.next.apart()) norm_ready_ = n.next;
    }
    // next: the norm r.next was taken from, if it has one
    void residual_norm(const StepCtx& s, ingot_residual_norm& r, const Norm& next) {
        r.x = x;
        r.n = round_up(width, 8);
        r.n_mean = width;
        r.n_rows = s.st.n_tok;
        r.eps = eps;
        const bool joined = r.next.w && conv_joins(s, next);
        if (joined) {
            r.conv = next.conv;
            r.conv_state = conv_state(next);
            r.taps = input_taps;
            r.slot = s.st.slot;
            r.pos0 = s.st.pos0;
        }
        if (r.next.w && next.conv && !joined) {
            r.out = buf(kConvIn);
        } else if (r.next.w) {
            const ingot_act_out o = operand(s, buf(kNormed), r.n, false);
            r.out = o.f32;
            r.hi = o.hi;
            r.lo = o.lo;
        }
        cuda_check(ingot_residual_norm_run(&r, stream), "residual");
        if (r.next.w && (!next.conv || joined)) operand_ready(s, r.n);
    }
    // Steps of single tokens: the launch that takes the norm does its input convolution too.
    bool conv_joins(const StepCtx& s, const Norm& norm) const { return norm.conv && s.st.max_len == 1 && input_taps <= 4; }
    float* conv_state(const Norm& norm) const { return norm.conv_state + size_t(norm.pass) * size_t(opt.max_seqs) * size_t(input_taps - 1) * size_t(round_up(width, 8)); }
    // x += v, one vector for all rows; `next` is the norm that is read then.
    void add_vector(const StepCtx& s, const float* v, const Norm& next) {
        norm_ready_ = Norm();
        shift_ = v;
        if (next.apart()) return;  // goes into that norm's launch
        ingot_residual_norm r = {};
        r.shift = std::exchange(shift_, nullptr);
        residual_norm(s, r, Norm());
    }
    // A feed-forward that runs beside the mixer leaves its result here; the mixer's project_residual takes it in.
    void set_branch(const Branch& b) { branch_ = b; }
    // The same without a mixer to join: x += branch.
    void add_branch(const StepCtx& s) {
        if (!branch_.rows) return;
        ingot_check(ingot_moe_add(x, branch_.rows, branch_.row_of, s.st.n_tok, branch_.top, round_up(width, 8), stream));
        branch_ = Branch();
        norm_ready_ = Norm();
    }
    // x = W [x; x0], two residual-length rows side by side
    void project_concat(const StepCtx& s, const Matrix& w, const float* x0) {
        const int n = round_up(width, 8);
        ingot_act_out o = operand(s, buf(kConcat), 2 * n, false);
        cuda_check(ingot_support_concat_rows(o.f32, o.hi, o.lo, x, x0, n, s.st.n_tok, stream), "concatenation");
        operand_ready(s, 2 * n);
        project(s, x, w, buf(kConcat), 2 * n);
        norm_ready_ = Norm();
    }
    // kMid (or the operand planes) = act(W_gate h) * (W_up h), h = norm(x); w holds runs of 32 gate rows, each followed by its up rows
    void gated_project(const StepCtx& s, const Matrix& w, const Norm& norm) {
        if (s.tc) prepare_norm(s, w, norm);
        else if (norm.apart() || !(s.st.n_tok == 1 && streams(w))) norm_rows(s, norm);
        gated_project_normed(s, w, norm);
    }
    // The same when the planes, or kNormed, hold h (single tokens read x through an RMS norm themselves).
    void gated_project_normed(const StepCtx& s, const Matrix& w, const Norm& norm) {
        const int ff = w.n_out / 2;
        if (s.tc) {
            cuda_check(ingot_linear_tc_run_gated_bf16(ws, w.data, w.n_in, w.n_out, design.act, s.planes, stream), "gate / up");
        } else if (s.st.n_tok == 1 && streams(w)) {
            cuda_check(ingot_support_gemv_bf16(buf(kMid), w.data, ff, w.n_in, norm.apart() ? buf(kNormed) : x, norm.apart() ? nullptr : norm.w, eps, width, 1, design.act, 0, stream), "gate / up");
        } else {
            cuda_check(ingot_support_linear_bf16(buf(kGateUp), w.data, buf(kNormed), w.n_in, w.n_in, w.n_out, 0, s.st.n_tok, 0, stream), "gate / up");
            cuda_check(ingot_support_gated_act(buf(kMid), buf(kGateUp), s.st.n_tok, ff, design.act, stream), "gate");
        }
    }
    void begin() { norm_ready_ = Norm(); branch_ = Branch(); shift_ = nullptr; }
    // Without tensor cores: kNormed = norm(x).
    void norm_rows(const StepCtx& s, const Norm& norm) {
        if (norm.apart()) {
            norm_now(s, norm);
            return;
        }
        cuda_check(ingot_support_rmsnorm_rows(buf(kNormed), x, norm.w, nullptr, s.st.n_tok, round_up(width, 8), width, eps, stream), "rmsnorm");
    }
    // Tensor-core path: the planes hold norm(x).
    void prepare_norm(const StepCtx& s, const Matrix& w, const Norm& norm) {
        if (norm.apart()) {
            norm_now(s, norm);
            return;
        }
        const bool ready = norm_ready_ == norm && norm;  // the kernel that finished x already normalised it for this product
        norm_ready_ = Norm();
        if (!ready) cuda_check(ingot_linear_tc_prepare_norm_bf16(ws, x, norm.w, eps, w.n_in, width, s.st.n_tok, s.planes, stream), "rmsnorm");
    }
    // A norm of its own (Norm::apart), unless the kernel that finished x took it, and the input convolution.
    void norm_now(const StepCtx& s, const Norm& norm) {
        const bool ready = norm_ready_ == norm;
        norm_ready_ = Norm();
        if (!ready) {
            ingot_residual_norm r = {};
            r.next = norm;
            r.shift = std::exchange(shift_, nullptr);
            residual_norm(s, r, norm);
        }
        if (!norm.conv || conv_joins(s, norm)) return;
        const int n = round_up(width, 8);
        const ingot_act_out o = operand(s, buf(kNormed), n, false);
        ingot_check(ingot_causal_conv(&s.st, buf(kConvIn), n, nullptr, norm.conv, nullptr, input_taps, n, 0, conv_state(norm), &o, stream));
        operand_ready(s, n);
    }

    const ModelDir& dir;
    const EngineOptions opt;
    const Design design;
    const int max_step;
    cudaStream_t stream = nullptr;
    ingot_linear_ws* ws = nullptr;
    float* x = nullptr;  // residual stream [n_tok][round_up(width, 8)]
    int width = 0;
    float eps = 0.f;
    int norm_groups = 1, input_taps = 0;  // equal groups of the norms over the residual; taps of the input convolutions (0: none)
    int passes = 1;  // of the layer under construction: each pass of a loop has a state and a cache of its own
    int pass = 0;    // the one that runs
    size_t weight_bytes = 0;
    std::vector<std::unique_ptr<CacheGroup>> caches;
    Groups mixed_values = {0, 0, 0};  // the values that layers mix with the first such layer's (kFirstValue): heads and sizes; none so far

    // The group a layer's caches belong to; *layer: the first of its `passes` caches there.
    CacheGroup* cache_group(int kv_heads, int dim, int chunk, int window, CacheGroup::Form form, int* layer) {
        CacheGroup* g = nullptr;
        for (auto& c : caches)
            if (c->kv_heads == kv_heads && c->dim == dim && c->chunk == chunk && c->window == window && c->form == form) g = c.get();
        if (!g) {
            caches.push_back(std::make_unique<CacheGroup>());
            g = caches.back().get();
            g->kv_heads = kv_heads; g->dim = dim; g->chunk = chunk; g->window = window; g->form = form;
        }
        *layer = g->n_layer;
        g->n_layer += passes;
        return g;
    }
    // Time chunks for a recurrence: threads that one chunk occupies (they size the chunks of a step), floats of scratch that it needs. The
    // number of the plan in StepCtx::plans; equal mixers share one. kind: of the recurrences over channels in 16-bit form (scan_routes.h), whose
    // short sequences may go in a call of their own, with their channels and states per channel; Kind::none for the others.
    struct PlanRequest { int threads; size_t scratch; ingot_scan::Kind kind; int channels, states; };
    size_t scan_plan(int threads, size_t scratch, ingot_scan::Kind kind = ingot_scan::Kind::none, int channels = 0, int states = 0) {
        for (size_t i = 0; i < plans_.size(); i++)
            if (plans_[i].threads == threads && plans_[i].kind == kind && plans_[i].channels == channels && plans_[i].states == states) {
                plans_[i].scratch = std::max(plans_[i].scratch, scratch);
                return i;
            }
        plans_.push_back({threads, scratch, kind, channels, states});
        return plans_.size() - 1;
    }
    const std::vector<PlanRequest>& plans() const { return plans_; }
    // Recurrent state of a layer: `floats` per sequence slot, for every pass; and the running pass's.
    float* state(size_t floats) { return static_cast<float*>(alloc(size_t(opt.max_seqs) * floats * size_t(passes) * 4, true)); }
    float* at_pass(float* state, size_t floats) const { return state + size_t(pass) * size_t(opt.max_seqs) * floats; }

private:
    WeightStreamer loader_;
    std::vector<void*> allocs_;
    int columns_[kBufCount] = {};
    float* bufs_[kBufCount] = {};
    int tc_in_ = 8, tc_out_ = 8;
    size_t key_bytes_[3] = {0, 0, 0};
    void* keys_[3] = {nullptr, nullptr, nullptr};
    Branch branch_;
    std::vector<PlanRequest> plans_;
    Norm norm_ready_;  // the norm x has been prepared with
    const float* shift_ = nullptr;  // to be added to x by the launch that takes the next norm
};

// ---- layers ----------------------------------------------------------------------------------------------------------

class Mixer {
public:
    virtual ~Mixer() = default;
    // x += post(mixer(in(x))) + the branch set beside it; norms as in LayerOps::project_residual.
    virtual void run(LayerOps& ops, const StepCtx& s, const Norms& n) = 0;
};

class FeedForward {
public:
    virtual ~FeedForward() = default;
    // x += post(ff(in(x))), after the mixer
    virtual void run(LayerOps& ops, const StepCtx& s, const Norms& n) = 0;
    // ff(norm(x)) as a branch beside the mixer (LayerOps::set_branch); runs before the mixer does
    virtual void branch(LayerOps& ops, const StepCtx& s, const Norm& norm) = 0;
};

// One function per kind; a further kind is a class in a file of its own and a line in make_mixer / make_feed_forward
// (hybrid_backend.cpp).
std::unique_ptr<Mixer> make_selective_scan(LayerOps& ops, const Json& config, const std::string& prefix);
std::unique_ptr<Mixer> make_gated_linear(LayerOps& ops, const Json& config, const std::string& prefix);
std::unique_ptr<Mixer> make_state_space(LayerOps& ops, const Json& config, const std::string& prefix);
std::unique_ptr<Mixer> make_parallel(LayerOps& ops, const Json& config, const std::string& prefix);
std::unique_ptr<Mixer> make_latent_attention(LayerOps& ops, const Json& config, const std::string& prefix);
std::unique_ptr<Mixer> make_grouped_attention(LayerOps& ops, const AttentionKind& kind, const Json& config, const std::string& prefix);
std::unique_ptr<FeedForward> make_gated_feed_forward(LayerOps& ops, const Json& config, const std::string& prefix);
std::unique_ptr<FeedForward> make_mixture(LayerOps& ops, const Json& config, const std::string& prefix);
