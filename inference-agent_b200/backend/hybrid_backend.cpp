// Decoder-only models whose layers are listed one by one in their configuration, each with a mixer of its own kind - recurrent,
// attention, or several side by side - and an optional feed-forward ("Besudra", "Banevik", "Silevik", "Gatuzen" and designs like them).
//
// Reading guide.
//   layer_ops.h     what layers are written in (LayerOps), and the interfaces Mixer and FeedForward: weights, per-sequence state and
//                   launches of one kind each. LayerOps picks the kernel by the number of tokens: weight-streaming GEMV for one
//                   token, tcgen05 GEMM for more (f32 kernels in the 32-bit form).
//   recurrent_layers.cpp, latent_layers.cpp, attention_layers.cpp, feed_forward.cpp   the kinds. A new one is a class there plus a line
//                   in make_mixer() or make_feed_forward().
//   HybridBackend   the step: one ragged batch of portions of several sequences, state slots and cache pages, the loop over layers
//                   (some of which may run several times, each pass with a state of its own), logits. A Design is what a model
//                   family fixes; everything else comes from its configuration.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "layer_ops.h"

namespace {

std::unique_ptr<Mixer> make_mixer(const std::string& type, LayerOps& ops, const Json& config, const std::string& prefix) {
    if (type == "mamba1") return make_selective_scan(ops, config, prefix);
    if (type == "mamba2") return make_state_space(ops, config, prefix);
    if (type == "gla") return make_gated_linear(ops, config, prefix);
    if (type == "parallel") return make_parallel(ops, config, prefix);
    if (type == "latent_attention") return make_latent_attention(ops, config, prefix);
    for (const AttentionKind& kind : ops.design.attention)
        if (type == kind.type) return make_grouped_attention(ops, kind, config, prefix);
    throw std::runtime_error("model config: unknown layer type \"" + type + "\"");
}

std::unique_ptr<FeedForward> make_feed_forward(LayerOps& ops, const Json& config, const std::string& prefix) {
    const std::string& kind = config.at("kind").str();
    if (kind == "dense") return make_gated_feed_forward(ops, config, prefix);
    if (kind == "moe") return make_mixture(ops, config, prefix);
    throw std::runtime_error("model config: unknown feed-forward kind \"" + kind + "\"");
}

// ---- the model -------------------------------------------------------------------------------------------------------

class HybridBackend : public ModelBackend {
public:
    HybridBackend(const ModelDir& dir, const EngineOptions& opt, const Design& design)
        : design_(design), ops_(dir, opt, design, opt.max_step_tokens > 0 ? opt.max_step_tokens : opt.max_tokens), max_seqs_(opt.max_seqs), max_ctx_(opt.max_tokens) {
        if (opt.max_tokens < 1 || opt.max_seqs < 1) throw std::runtime_error("engine: needs at least one token and one sequence");
        int device = 0;
        cuda_check(cudaGetDevice(&device), "cudaGetDevice");
        cuda_check(cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, device), "device attribute");
        const Json& c = dir.config();
        n_vocab_ = get_int(c, "vocab");
        ops_.width = get_int(c, "width");
        ops_.eps = get_float(c.at("norm"), "eps");
        if (has(c.at("norm"), "groups")) ops_.norm_groups = get_int(c.at("norm"), "groups", 1, ops_.width);
        if (ops_.width % ops_.norm_groups != 0) throw std::runtime_error("model config: \"width\" is not a multiple of \"norm.groups\"");
        if (ops_.norm_groups > 1 && design.centred) throw std::runtime_error("model config: this design's norms have no groups");
        if (has(c, "canon")) ops_.input_taps = get_int(c.at("canon"), "taps", 1, 16);
        const float residual = has(c, "residual_mult") ? get_float(c, "residual_mult") : 1.f;  // rides on the norms of the parts' results
        if (residual != 1.f && !design.sandwich) throw std::runtime_error("model config: this design has no \"residual_mult\"");
        const Groups d = flat(ops_.width);
        ops_.x = static_cast<float*>(ops_.alloc(size_t(ops_.max_step) * d.padded * 4, true));
        ops_.need(kNormed, d.padded);
        if (design.sandwich) ops_.need(kBranch, d.padded);
        ops_.tc_shape(d.padded, round_up(n_vocab_, 8));
        embed_ = ops_.matrix("embed", flat(n_vocab_), d);
        if (has(c, "embedding") && has(c.at("embedding"), "scale")) embed_scale_ = get_float(c.at("embedding"), "scale");
        if (has(c, "embedding") && has(c.at("embedding"), "bigram")) {
            const Json& b = c.at("embedding").at("bigram");
            bigram_buckets_ = get_int(b, "buckets");
            bigram_prev_ = b.at("mul_prev").integer();
            bigram_cur_ = b.at("mul_cur").integer();
            bigram_ = ops_.matrix("bigram", Groups{1, bigram_buckets_ + 1, bigram_buckets_ + 1}, d);
        }
        const auto& layers = c.at("layers").items();
        if (has(c, "loop")) {
            const Json& l = c.at("loop");
            loop_start_ = size_t(get_int(l, "start", 0, int(layers.size())));
            loop_stop_ = size_t(get_int(l, "stop", 0, int(layers.size())));
            loop_times_ = get_int(l, "times");
            if (loop_stop_ <= loop_start_) throw std::runtime_error("model config: the loop has no layers");
        }
        size_t table_bytes = ops_.weight_bytes;  // read row by row, not once per step
        if (loop_times_ > 0 && design.loop_step) {
            loop_step_ = ops_.vector("loop.step", {loop_times_, ops_.width}, {loop_times_, ops_.width, d.padded});
        } else if (loop_times_ > 0) {
            loop_in_ = ops_.matrix(d.padded, 2 * d.padded, {Part{"loop.in", {ops_.width, 2 * ops_.width}, d, {2, ops_.width, d.padded}}});
            x0_ = static_cast<float*>(ops_.alloc(size_t(ops_.max_step) * d.padded * 4, true));
            ops_.need(kConcat, 2 * d.padded);
        }
        for (size_t i = 0; i < layers.size(); i++) {
            const std::string p = "l" + std::to_string(i) + ".";
            Layer L;
            L.type = layers[i].at("type").str();
            ops_.passes = in_loop(i) ? loop_times_ : 1;
            L.norm1 = ops_.input_norm(p + "norm1", p + "canon1");
            if (design.sandwich) L.norm1b = ops_.norm(p + "norm1b", residual);
            L.mixer = make_mixer(L.type, ops_, layers[i].at("mixer"), p + "mix.");
            if (layers[i].has("mlp") && !layers[i].at("mlp").is_null()) {
                L.norm2 = ops_.input_norm(p + "norm2", p + "canon2");
                if (design.sandwich) L.norm2b = ops_.norm(p + "norm2b", residual);
                L.mlp = make_feed_forward(ops_, layers[i].at("mlp"), p + "mlp.");
            }
            layers_.push_back(std::move(L));
        }
        // a factor of the logits rides on the norm before them
        final_norm_ = ops_.norm("final.norm", has(c, "logit_scale") ? get_float(c, "logit_scale") : 1.f);
        if (design.tied_head) {
            head_ = embed_;
            table_bytes -= size_t(embed_.n_out) * embed_.n_in * 2;
        } else {
            head_ = ops_.matrix("head", flat(n_vocab_), d);
        }
        if (has(c, "logit_softcap")) softcap_ = get_float(c, "logit_softcap");
        weight_bytes_ = ops_.weight_bytes - table_bytes;
        // the layers as they run, pass after pass
        for (size_t i = 0; i < layers_.size();) {
            if (i != loop_start_ || loop_times_ == 0) { runs_.push_back({i++, 0, false}); continue; }
            for (int pass = 0; pass < loop_times_; pass++)
                for (size_t j = loop_start_; j < loop_stop_; j++) runs_.push_back({j, pass, j == loop_start_});
            i = loop_stop_;
        }
        for (auto& g : ops_.caches) {
            g->pages_per_chunk = g->chunk > 0 ? (g->chunk + INGOT_BLOCK_TOKENS - 1) / INGOT_BLOCK_TOKENS : 0;
            // the pool holds max_tokens tokens of live sequences however they are spread over max_seqs of them
            // (whole chunks, and one begun chunk and one begun page per sequence)
            const long long whole = g->chunk > 0 ? (long long)(max_ctx_ / g->chunk) * g->pages_per_chunk : 0, pages = (long long)max_ctx_ / INGOT_BLOCK_TOKENS + max_seqs_;
            long long blocks = g->chunk > 0 ? whole + std::min(pages, (long long)max_seqs_ * g->pages_per_chunk) : pages;
            // behind a window only what it covers is held, besides the tokens of the step itself
            if (g->window > 0) blocks = std::min(pages, (long long)max_seqs_ * (g->pages_seen() + 2) + ops_.max_step / INGOT_BLOCK_TOKENS);
            if (blocks > (1 << 26)) throw std::runtime_error("engine: cache pool too large");
            const int dtype = opt.f32 ? INGOT_F32 : INGOT_F16;
            if (g->form == CacheGroup::scaled && g->window > 0) throw std::runtime_error("engine: no cache form for scaled rows behind a window");
            ingot_check(g->form == CacheGroup::scaled  ? ingot_skv_create(&g->kv, g->n_layer, g->kv_heads, g->dim, dtype, g->chunk, int(blocks))
                        : g->form == CacheGroup::plain ? ingot_skv_create_window(&g->kv, g->n_layer, g->kv_heads, g->dim, dtype, g->window, int(blocks))
                                                       : ingot_skv_create_joined(&g->kv, g->n_layer, g->kv_heads, g->dim, dtype, g->window, int(blocks)));
            g->pool = BlockPool(int(blocks), max_seqs_, ingot_skv_pages(g->chunk, max_ctx_));
        }
        embed_status_ = static_cast<int*>(ops_.alloc(sizeof(int), true));
        ops_.allocate();
        cuda_check(cudaMallocHost(&status_host_, kMaxStatus * sizeof(int)), "cudaMallocHost");
        cuda_check(cudaEventCreate(&ev0_), "cudaEventCreate");
        cuda_check(cudaEventCreate(&ev1_), "cudaEventCreate");
        lens_.assign(size_t(max_seqs_), 0);
        last_token_.assign(size_t(max_seqs_), 0);
        status_words_.push_back(embed_status_);
        if (ops_.ws) status_words_.push_back(ingot_linear_ws_status_dev(ops_.ws));
        for (auto& g : ops_.caches) status_words_.push_back(ingot_skv_status_dev(g->kv));
        if (status_words_.size() > kMaxStatus) throw std::runtime_error("engine: too many cache groups");
    }
    ~HybridBackend() override {
        cudaStreamSynchronize(ops_.stream);
        drop_graphs();
        for (auto& g : ops_.caches) ingot_skv_destroy(g->kv);
        cudaFree(meta_dev_);
        cudaFree(logits_dev_);
        cudaFree(scan_scratch_dev_);
        cudaFreeHost(meta_host_);
        cudaFreeHost(logits_);
        cudaFreeHost(status_host_);
        if (ev0_) cudaEventDestroy(ev0_);
        if (ev1_) cudaEventDestroy(ev1_);
    }

    const float* forward_multi(const int32_t* tokens, const int32_t* seq_ids, const int32_t* positions, int n) override {
        static const int32_t zero = 0;
        std::vector<StepEntry> e(size_t(std::max(n, 0)));
        for (int i = 0; i < n; i++) e[size_t(i)] = StepEntry{seq_ids[i], positions[i], tokens + i, 1, &zero, 1};
        return forward_step(e.data(), n, n_vocab_);
    }

    const float* forward_step(const StepEntry* entries, int n, int n_vocab) override {
        float* const into = std::exchange(into_, nullptr);
        if (n_vocab != n_vocab_) throw std::runtime_error("engine: vocabulary size mismatch");
        Step step = check(entries, n);
        reserve_pages(entries, n);
        reserve_logits(step.n_want);
        float* const logits = into ? into : logits_;
        const StepCtx s = lay_out_step(entries, n, step, logits);
        // Steps of single decoded tokens are the same launches every time but for what the metadata says: captured once per
        // batch size and reach (Step::reach) and replayed. The first such step of a size runs eagerly.
        const bool replay = step.decode && !tap_ && use_graphs_;
        const std::pair<int, int> key(n, step.reach);
        cuda_check(cudaEventRecord(ev0_, ops_.stream), "cudaEventRecord");
        if (replay && graphs_.count(key) && graphs_[key].exec) {
            cuda_check(cudaGraphLaunch(graphs_[key].exec, ops_.stream), "cudaGraphLaunch");
        } else if (replay && graphs_[key].seen++ > 0) {
            cuda_check(cudaStreamBeginCapture(ops_.stream, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
            try {
                encode(s, step);
            } catch (...) {
                cudaGraph_t dead = nullptr;
                cudaStreamEndCapture(ops_.stream, &dead);
                if (dead) cudaGraphDestroy(dead);
                throw;
            }
            cuda_check(cudaStreamEndCapture(ops_.stream, &graphs_[key].graph), "cudaStreamEndCapture");
            cuda_check(cudaGraphInstantiate(&graphs_[key].exec, graphs_[key].graph, 0), "cudaGraphInstantiate");
            cuda_check(cudaGraphLaunch(graphs_[key].exec, ops_.stream), "cudaGraphLaunch");
        } else {
            encode(s, step);
        }
        if (step.n_want > kDeliveredRows)
            cuda_check(cudaMemcpy2DAsync(logits, size_t(n_vocab_) * 4, logits_dev_, size_t(head_.n_out) * 4, size_t(n_vocab_) * 4, size_t(step.n_want),
                                         cudaMemcpyDeviceToHost, ops_.stream), "D2H logits");
        cuda_check(cudaEventRecord(ev1_, ops_.stream), "cudaEventRecord");
        cuda_check(cudaStreamSynchronize(ops_.stream), "step");
        cudaEventElapsedTime(&last_ms_, ev0_, ev1_);
        for (size_t i = 0; i < status_words_.size(); i++)
            if (status_host_[i]) {
                const int word = status_host_[i];
                cudaMemset(status_words_[i], 0, sizeof(int));
                throw std::runtime_error("engine: a kernel reported status " + std::to_string(word));
            }
        for (int i = 0; i < n; i++) {
            const int seq = entries[i].seq_id, next = entries[i].pos0 + entries[i].n_tokens;
            lens_[size_t(seq)] = next;
            last_token_[size_t(seq)] = entries[i].tokens[entries[i].n_tokens - 1];
            // pages of chunks that lie wholly in the past, or behind the window, can never be seen again
            for (auto& g : ops_.caches)
                if (g->forgets() && next < max_ctx_) g->pool.release(seq, 0, g->page(g->first_visible(next)));
        }
        return step.n_want ? logits : nullptr;
    }
    bool step_into(float* rows) override {
        into_ = rows;
        return true;
    }

    void release_sequence(int seq_id) override {
        if (seq_id < 0 || seq_id >= max_seqs_) throw std::runtime_error("engine: sequence id out of range");
        lens_[size_t(seq_id)] = 0;
        for (auto& g : ops_.caches) g->pool.release(seq_id);
    }
    int max_seqs() const override { return max_seqs_; }
    int n_ctx_per_seq() const override { return max_ctx_; }
    int max_portion() const override { return ops_.max_step; }
    int max_step_tokens() const override { return ops_.max_step; }
    int n_vocab() const override { return n_vocab_; }
    void tap_residuals(std::vector<float>* out) override { tap_ = out; }
    size_t weight_bytes() const override { return weight_bytes_; }
    float last_step_ms() const override { return last_ms_; }
    std::string describe() const override {
        std::map<std::string, int> kinds;
        for (const Layer& l : layers_) kinds[l.type]++;
        std::string t = std::to_string(layers_.size()) + " layers (";
        bool first = true;
        for (const auto& [k, v] : kinds) { t += (first ? "" : ", ") + std::to_string(v) + " " + k; first = false; }
        return t + "), width " + std::to_string(ops_.width) + ", vocabulary " + std::to_string(n_vocab_) + ", " + (ops_.opt.f32 ? "float32" : "bfloat16");
    }

private:
    struct Layer {
        std::string type;
        Norm norm1, norm1b, norm2, norm2b;  // before and after the mixer, before and after the feed-forward
        std::unique_ptr<Mixer> mixer;
        std::unique_ptr<FeedForward> mlp;
    };
    struct Run {
        size_t layer;
        int pass;
        bool entry;  // first layer of a pass of the loop
    };
    struct Step {
        int n_tok = 0, max_len = 0, n_want = 0;
        bool decode = true;           // one token of every sequence, its logits wanted
        int reach = 0;                // decoding: pages of the longest sequence, rounded up to a power of two (block tables are this wide)
        const int32_t* want_rows = nullptr;  // device
        const int32_t* tokens = nullptr;     // device
        const int32_t* bigrams = nullptr;    // device: rows of the bigram table
        int first_want = 0;           // host copy of want_rows[0]
        size_t pieces = 0;            // of 16 bytes: the metadata
        float* const* logits_at = nullptr;   // device: where the wanted rows go (pinned host memory)
    };
    struct Graph {
        int seen = 0;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
    };
    static constexpr size_t kMaxStatus = 64;
    static constexpr int kDeliveredRows = 64;  // more rows leave by the copy engine: megabytes, whatever the start costs

    bool in_loop(size_t i) const { return loop_times_ > 0 && i >= loop_start_ && i < loop_stop_; }

    Step check(const StepEntry* entries, int n) const {
        if (n < 1 || n > max_seqs_) throw std::runtime_error("engine: batch size out of range");
        Step step;
        std::vector<char> seen(size_t(max_seqs_), 0);
        for (int i = 0; i < n; i++) {
            const StepEntry& e = entries[i];
            if (e.seq_id < 0 || e.seq_id >= max_seqs_) throw std::runtime_error("engine: sequence id out of range");
            if (seen[size_t(e.seq_id)]++) throw std::runtime_error("engine: a sequence appears twice in one step");
            if (e.n_tokens < 1) throw std::runtime_error("engine: empty portion");
            if (e.pos0 < 0 || e.pos0 > max_ctx_ - e.n_tokens) throw std::runtime_error("context window exceeded");
            // a recurrent state only exists at the end of what has been run: go on from there, or start again
            if (e.pos0 != 0 && e.pos0 != lens_[size_t(e.seq_id)]) throw std::runtime_error("engine: a sequence must continue where it stands or restart at 0");
            for (int t = 0; t < e.n_tokens; t++)
                if (e.tokens[t] < 0 || e.tokens[t] >= n_vocab_) throw std::runtime_error("token id out of range");
            for (int w = 0; w < e.n_want; w++)
                if (e.want[w] < 0 || e.want[w] >= e.n_tokens) throw std::runtime_error("engine: wanted place outside the portion");
            step.n_tok += e.n_tokens;
            step.max_len = std::max(step.max_len, e.n_tokens);
            step.n_want += e.n_want;
            step.decode = step.decode && e.n_tokens == 1 && e.n_want == 1;
            while (step.reach * INGOT_BLOCK_TOKENS < e.pos0 + e.n_tokens) step.reach = std::max(8, step.reach * 2);
        }
        if (step.n_tok > ops_.max_step) throw std::runtime_error("engine: more tokens than a step may carry");
        return step;
    }

    void reserve_pages(const StepEntry* entries, int n) {
        for (int i = 0; i < n; i++)
            for (auto& g : ops_.caches) {
                if (entries[i].pos0 == 0) g->pool.release(entries[i].seq_id);  // a restart leaves what it held
                g->pool.ensure(entries[i].seq_id, g->page(g->first_visible(entries[i].pos0)), g->page(entries[i].pos0 + entries[i].n_tokens - 1));
            }
    }

    // INGOT_SCAN_THREADS: threads per SM the chunks of a recurrence aim for (tuning).
    // Length of the time chunks of a recurrence one token-chunk of which occupies `threads` threads: as few chunks as fill the GPU.
    // Longer ones if the sequences' ends would make it more chunks than that (a second round of CTAs).
    int chunk_tokens(const std::vector<StepEntry>& entries, int n_tok, int threads) const {
        const int chunks = std::max(1, num_sms_ * scan_threads_per_sm_ / std::max(threads, 1)), even = std::max(32, round_up((n_tok + chunks - 1) / chunks, 16));
        for (int length = even; length < 2 * even; length += std::max(16, even / 16 / 16 * 16)) {
            int count = 0;
            for (const StepEntry& e : entries)
                if (e.n_tokens > 32) count += (e.n_tokens + length - 1) / length;
            if (count <= chunks) return length;
        }
        return even;
    }

    // The step's metadata, in pinned host memory (the step's first launch fetches it), and where each part of it will be on the device.
    StepCtx lay_out_step(const StepEntry* asked, int n, Step& step, float* logits) {
        // Sequences run in ascending order of their portions, so that decoded tokens and short portions are the first rows and a
        // mixer can treat them apart from long ones.
        std::vector<int> order(static_cast<size_t>(n));
        for (int i = 0; i < n; i++) order[size_t(i)] = i;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return asked[a].n_tokens < asked[b].n_tokens; });
        std::vector<StepEntry> entries;
        std::vector<int> place(static_cast<size_t>(n));
        for (int i = 0; i < n; i++) {
            entries.push_back(asked[order[size_t(i)]]);
            place[size_t(order[size_t(i)])] = i;
        }
        std::vector<int32_t>& m = meta_;
        m.clear();
        auto mark = [&] { while (m.size() % 4) m.push_back(0); return m.size(); };
        const size_t o_logits = mark();
        m.resize(m.size() + sizeof(logits) / sizeof(int32_t));
        memcpy(m.data() + o_logits, &logits, sizeof(logits));
        const size_t o_tok = mark();
        for (int i = 0; i < n; i++) m.insert(m.end(), entries[i].tokens, entries[i].tokens + entries[i].n_tokens);
        const size_t o_bigram = mark();
        if (bigram_.data)
            for (int i = 0; i < n; i++)
                for (int t = 0; t < entries[i].n_tokens; t++) {
                    const bool first = entries[i].pos0 + t == 0;
                    const int64_t prev = first ? 0 : t > 0 ? entries[i].tokens[t - 1] : last_token_[size_t(entries[i].seq_id)];
                    m.push_back(first ? bigram_buckets_ : bigram_row(prev, entries[i].tokens[t]));
                }
        const size_t o_rowseq = mark();
        for (int i = 0; i < n; i++) m.insert(m.end(), size_t(entries[i].n_tokens), i);
        const size_t o_start = mark();
        for (int i = 0, r = 0; i < n; r += entries[i].n_tokens, i++) m.push_back(r);
        const size_t o_len = mark();
        for (int i = 0; i < n; i++) m.push_back(entries[i].n_tokens);
        const size_t o_pos = mark();
        for (int i = 0; i < n; i++) m.push_back(entries[i].pos0);
        const size_t o_slot = mark();
        for (int i = 0; i < n; i++) m.push_back(entries[i].seq_id);
        const size_t o_want = mark();
        for (int i = 0; i < n; i++)
            for (int w = 0; w < asked[i].n_want; w++) m.push_back(m[o_start + size_t(place[size_t(i)])] + asked[i].want[w]);
        rows_asked_.clear();
        for (int i = 0; i < n; i++)
            for (int t = 0; t < asked[i].n_tokens; t++) rows_asked_.push_back(m[o_start + size_t(place[size_t(i)])] + t);
        lens_sorted_.assign(m.begin() + long(o_len), m.begin() + long(o_len) + n);
        step.first_want = step.n_want ? m[o_want] : 0;
        struct PlanAt { int seq0, seq1; size_t seq, t0, len, first; int n_chunks, max_chunks; };  // of sequences seq0 .. seq1 - 1
        auto plan = [&](int seq0, int seq1, int chunk) {
            PlanAt p = {};
            p.seq0 = seq0;
            p.seq1 = seq1;
            std::vector<int32_t> seq, t0, len, first;
            for (int i = seq0; i < seq1; i++) {
                first.push_back(int32_t(seq.size()));
                for (int t = 0; t < entries[i].n_tokens; t += chunk) {
                    seq.push_back(i - seq0);
                    t0.push_back(t);
                    len.push_back(std::min(chunk, entries[i].n_tokens - t));
                }
                p.max_chunks = std::max(p.max_chunks, int(seq.size()) - first.back());
            }
            first.push_back(int32_t(seq.size()));
            p.n_chunks = int(seq.size());
            p.seq = mark(); m.insert(m.end(), seq.begin(), seq.end());
            p.t0 = mark(); m.insert(m.end(), t0.begin(), t0.end());
            p.len = mark(); m.insert(m.end(), len.begin(), len.end());
            p.first = mark(); m.insert(m.end(), first.begin(), first.end());
            return p;
        };
        std::vector<std::vector<PlanAt>> plans;
        for (const auto& r : ops_.plans()) {
            const int chunk = chunk_tokens(entries, step.n_tok, r.threads);  // of the whole step, however it is cut: results do not depend on that
            auto load = [&](int a, int b) {
                const int longest = b > a ? lens_sorted_[size_t(b) - 1] : 0;
                return ingot_scan::Load{std::accumulate(lens_sorted_.begin() + a, lens_sorted_.begin() + b, 0ll), longest, b - a, (longest + chunk - 1) / chunk};
            };
            const int cut = r.kind == ingot_scan::Kind::none ? 0 : int(std::upper_bound(lens_sorted_.begin(), lens_sorted_.end(), ingot_scan::kShort) - lens_sorted_.begin());
            if (cut > 0 && ingot_scan::apart(r.kind, load(0, n), load(0, cut), load(cut, n), r.channels, r.states, num_sms_)) plans.push_back({plan(0, cut, chunk), plan(cut, n, chunk)});
            else plans.push_back({plan(0, n, chunk)});
        }
        struct TableAt { size_t first, table, key0, key_pos; };
        std::vector<TableAt> table_at;
        for (auto& g : ops_.caches) {
            const size_t o_first = mark();
            int width = 1;
            for (int i = 0; i < n; i++) {
                const int first = g->page(g->first_visible(entries[i].pos0));
                width = std::max(width, g->page(entries[i].pos0 + entries[i].n_tokens - 1) - first + 1);
                m.push_back(first);
            }
            // the same at every step that replays the same launches
            if (step.decode) width = std::min({g->forgets() ? g->pages_seen() : step.reach, step.reach, g->pool.pages_per_seq()});
            const size_t o_table = mark();
            for (int i = 0; i < n; i++) {
                const int first = m[o_first + size_t(i)];
                const int32_t* row = g->pool.row(entries[i].seq_id);
                for (int k = 0; k < width; k++) m.push_back(first + k < g->pool.pages_per_seq() ? row[first + k] : -1);
            }
            g->width = width;
            const size_t o_key0 = mark();
            plan_expansions(*g, entries);
            for (int i = 0, row = 0, b = 0; i < n; i++) {  // key rows count from 0 in each run of sequences that are expanded together
                if (i >= g->first_long && g->expansions[size_t(b)].seq0 + g->expansions[size_t(b)].n_seq <= i) { b++; row = 0; }
                m.push_back(row);
                if (i >= g->first_long) row += keys_seen(*g, entries[size_t(i)]);
            }
            const size_t o_key_pos = mark();
            for (int i = 0; i < n; i++) m.push_back(g->first_visible(entries[size_t(i)].pos0));
            table_at.push_back({o_first, o_table, o_key0, o_key_pos});
        }
        mark();
        if (m.size() > meta_cap_) {
            drop_graphs();
            cudaFree(meta_dev_);
            cudaFreeHost(meta_host_);
            meta_dev_ = meta_host_ = nullptr;
            meta_cap_ = std::max<size_t>(m.size() * 2, 65536);
            cuda_check(cudaMalloc(&meta_dev_, meta_cap_ * 4), "cudaMalloc(step metadata)");
            cuda_check(cudaMallocHost(&meta_host_, meta_cap_ * 4), "cudaMallocHost(step metadata)");
        }
        memcpy(meta_host_, m.data(), m.size() * 4);
        step.pieces = m.size() / 4;
        step.logits_at = reinterpret_cast<float* const*>(meta_dev_ + o_logits);

        StepCtx s;
        s.st.n_tok = step.n_tok;
        s.st.n_seq = n;
        s.st.max_len = step.max_len;
        s.st.row_seq = meta_dev_ + o_rowseq;
        s.st.row_start = meta_dev_ + o_start;
        s.st.len = meta_dev_ + o_len;
        s.st.pos0 = meta_dev_ + o_pos;
        s.st.slot = meta_dev_ + o_slot;
        s.lens = lens_sorted_.data();
        step.tokens = s.tokens = meta_dev_ + o_tok;
        step.bigrams = meta_dev_ + o_bigram;
        step.want_rows = meta_dev_ + o_want;
        size_t floats = 0;  // one scratch for all: mixers run one after the other
        for (size_t i = 0; i < plans.size(); i++)
            for (const PlanAt& at : plans[i])
                if (at.max_chunks > 1) floats = std::max(floats, ops_.plans()[i].scratch * size_t(at.n_chunks));
        if (floats > scan_cap_) {
            drop_graphs();
            cuda_check(cudaStreamSynchronize(ops_.stream), "scratch");
            cudaFree(scan_scratch_dev_);
            scan_scratch_dev_ = nullptr;
            scan_cap_ = 0;
            cuda_check(cudaMalloc(&scan_scratch_dev_, floats * 4), "cudaMalloc(scan scratch)");
            scan_cap_ = floats;
        }
        for (const auto& parts : plans) {
            s.plans.emplace_back();
            for (const PlanAt& at : parts) {
                StepCtx::ScanPart p = {s.st, {}};
                p.st.n_tok = std::accumulate(lens_sorted_.begin() + at.seq0, lens_sorted_.begin() + at.seq1, 0);
                p.st.n_seq = at.seq1 - at.seq0;
                p.st.max_len = lens_sorted_[size_t(at.seq1) - 1];
                for (const int32_t** a : {&p.st.row_start, &p.st.len, &p.st.pos0, &p.st.slot}) *a += at.seq0;
                p.plan.n_chunks = at.n_chunks;
                p.plan.max_chunks = at.max_chunks;
                p.plan.chunk_seq = meta_dev_ + at.seq;
                p.plan.chunk_t0 = meta_dev_ + at.t0;
                p.plan.chunk_len = meta_dev_ + at.len;
                p.plan.seq_chunk0 = meta_dev_ + at.first;
                p.plan.scratch_dev = scan_scratch_dev_;
                p.plan.scratch_floats = scan_cap_;
                s.plans.back().push_back(p);
            }
        }
        for (size_t i = 0; i < ops_.caches.size(); i++) {
            ops_.caches[i]->first_page = meta_dev_ + table_at[i].first;
            ops_.caches[i]->tables = meta_dev_ + table_at[i].table;
            ops_.caches[i]->key0 = meta_dev_ + table_at[i].key0;
            ops_.caches[i]->key_pos = meta_dev_ + table_at[i].key_pos;
        }
        s.tc = ops_.ws != nullptr && step.n_tok >= kMinTcTokens;
        s.planes = s.tc && step.n_tok <= kPairTokens ? 2 : 1;
        return s;
    }

    static int keys_seen(const CacheGroup& g, const StepEntry& e) { return e.pos0 + e.n_tokens - g.first_visible(e.pos0); }
    // Which sequences of the step (in ascending order of their portions) run on expanded keys, and how many at a time.
    void plan_expansions(CacheGroup& g, const std::vector<StepEntry>& entries) const {
        const int n = int(entries.size());
        g.first_long = n;
        g.expansions.clear();
        if (g.expand_from <= 0 || !ops_.ws) return;
        while (g.first_long > 0 && entries[size_t(g.first_long) - 1].n_tokens >= g.expand_from) g.first_long--;
        for (int i = g.first_long; i < n; i++) {
            const int keys = keys_seen(g, entries[size_t(i)]);
            if (keys > g.key_rows) {  // more than there is room for: this step stays on the rows
                g.first_long = n;
                g.expansions.clear();
                return;
            }
            if (g.expansions.empty() || g.expansions.back().n_keys + keys > g.key_rows) g.expansions.push_back({i, 0, 0, 0});
            CacheGroup::Expansion& e = g.expansions.back();
            e.n_seq++;
            e.n_keys += keys;
            e.most_keys = std::max(e.most_keys, keys);
        }
    }

    int32_t bigram_row(int64_t prev, int64_t cur) const {
        const int64_t b = bigram_buckets_, r = ((prev * (bigram_prev_ % b)) % b + (cur * (bigram_cur_ % b)) % b) % b;
        return int32_t(r < 0 ? r + b : r);
    }

    void reserve_logits(int rows) {
        if (rows <= logit_rows_) return;
        drop_graphs();
        cuda_check(cudaStreamSynchronize(ops_.stream), "logits");
        cudaFree(logits_dev_);
        cudaFreeHost(logits_);
        logits_dev_ = nullptr;
        logits_ = nullptr;
        logit_rows_ = std::max(rows, max_seqs_);
        cuda_check(cudaMalloc(&logits_dev_, size_t(logit_rows_) * head_.n_out * 4), "cudaMalloc(logits)");
        cuda_check(cudaMallocHost(&logits_, size_t(logit_rows_) * n_vocab_ * 4), "cudaMallocHost(logits)");
    }
    void drop_graphs() {
        if (graphs_.empty()) return;
        cudaStreamSynchronize(ops_.stream);
        for (auto& [n, g] : graphs_) {
            if (g.exec) cudaGraphExecDestroy(g.exec);
            if (g.graph) cudaGraphDestroy(g.graph);
        }
        graphs_.clear();
    }

    // Every launch of a step, from its metadata to the logits of the wanted rows in host memory.
    void encode(const StepCtx& s, const Step& step) {
        cuda_check(ingot_support_fetch(meta_dev_, meta_host_, step.pieces, ops_.stream), "step metadata");
        encode_layers(s, step);
        const bool there = step.n_want > 0 && encode_logits(step);
        cuda_check(ingot_support_deliver(step.logits_at, logits_dev_, head_.n_out, n_vocab_, there || step.n_want > kDeliveredRows ? 0 : step.n_want, status_host_, status_words_.data(),
                                         int(status_words_.size()), ops_.stream), "logits and status");
    }
    void encode_layers(const StepCtx& s, const Step& step) {
        if (bigram_.data || x0_)
            cuda_check(ingot_support_embed_sum_bf16(ops_.x, x0_, embed_.data, n_vocab_, step.tokens, bigram_.data, bigram_buckets_ + 1, step.bigrams, embed_.n_in,
                                                    s.st.n_tok, embed_scale_, embed_status_, ops_.stream), "embedding rows");
        else
            cuda_check(ingot_support_embed_rows_bf16(ops_.x, embed_.data, embed_.n_in, n_vocab_, step.tokens, s.st.n_tok, embed_scale_, embed_status_, ops_.stream), "embedding rows");
        ops_.begin();
        for (size_t i = 0; i < runs_.size(); i++) {
            const Layer& L = layers_[runs_[i].layer];
            // the norm that is read next, unless something else happens to x first
            const bool more = i + 1 < runs_.size() && !runs_[i + 1].entry;
            const Norm following = more ? first_norm(layers_[runs_[i + 1].layer]).of_pass(runs_[i + 1].pass) : Norm();
            const int pass = ops_.pass = runs_[i].pass;
            const Norm norm1 = L.norm1.of_pass(pass), norm2 = L.norm2.of_pass(pass);
            if (runs_[i].entry && loop_step_) ops_.add_vector(s, loop_step_ + size_t(pass) * embed_.n_in, first_norm(L));
            else if (runs_[i].entry) ops_.project_concat(s, loop_in_, x0_);
            if (design_.parallel) {
                if (L.mlp) L.mlp->branch(ops_, s, norm2);
                L.mixer->run(ops_, s, {norm1, L.norm1b, following});
            } else {
                L.mixer->run(ops_, s, {norm1, L.norm1b, L.mlp ? norm2 : following});
                if (L.mlp) L.mlp->run(ops_, s, {norm2, L.norm2b, following});
            }
            if (tap_) tap(s.st.n_tok);
        }
    }
    // Returns whether the rows are in host memory already.
    bool encode_logits(const Step& step) {
        const int ld = embed_.n_in;
        int there = 0;
        if (step.n_want == 1 && LayerOps::streams(head_) && !final_norm_.apart()) {
            cuda_check(ingot_support_gemv_bf16(logits_dev_, head_.data, head_.n_out, head_.n_in, ops_.x + size_t(step.first_want) * ld, final_norm_.w, ops_.eps,
                                               ops_.width, 0, 0, 0, ops_.stream), "logits");
            cap_logits(step);
            return false;
        }
        if (final_norm_.apart()) {
            ingot_residual_norm r = {};
            r.x = ops_.x;
            r.n = ld;
            r.n_mean = ops_.width;
            r.n_rows = step.n_want;
            r.eps = ops_.eps;
            r.rows = step.want_rows;
            r.next = final_norm_;
            r.out = ops_.buf(kNormed);
            cuda_check(ingot_residual_norm_run(&r, ops_.stream), "final norm");
        } else {
            cuda_check(ingot_support_rmsnorm_rows(ops_.buf(kNormed), ops_.x, final_norm_.w, step.want_rows, step.n_want, ld, ops_.width, ops_.eps, ops_.stream), "final norm");
        }
        if (step.n_want == 1 && LayerOps::streams(head_)) {
            cuda_check(ingot_support_gemv_bf16(logits_dev_, head_.data, head_.n_out, head_.n_in, ops_.buf(kNormed), nullptr, 0.f, ld, 0, 0, 0, ops_.stream), "logits");
        } else if (ops_.ws && step.n_want >= kMinTcTokens) {
            cuda_check(ingot_linear_tc_prepare_bf16(ops_.ws, ops_.buf(kNormed), ld, ld, step.n_want, step.n_want <= kPairTokens ? 2 : 1, ops_.stream), "final norm");
            // whole rows as they are: the product may write them where they are wanted
            const bool to_host = softcap_ <= 0 && head_.n_out == n_vocab_ && step.n_want <= kDeliveredRows;
            if (to_host) cuda_check(ingot_linear_tc_run_to(ops_.ws, logits_dev_, step.logits_at, head_.data, head_.n_in, head_.n_out, &there, ops_.stream), "logits");
            else cuda_check(ingot_linear_tc_run(ops_.ws, logits_dev_, head_.data, head_.n_in, head_.n_out, 0, ops_.stream), "logits");
        } else {
            cuda_check(ingot_support_linear_bf16(logits_dev_, head_.data, ops_.buf(kNormed), ld, ld, head_.n_out, 0, step.n_want, 0, ops_.stream), "logits");
        }
        cap_logits(step);
        return there != 0;
    }
    void cap_logits(const Step& step) {
        if (softcap_ > 0) cuda_check(ingot_support_softcap(logits_dev_, size_t(step.n_want) * head_.n_out, softcap_, ops_.stream), "softcap");
    }
    Norm first_norm(const Layer& L) const { return design_.parallel && L.mlp ? L.norm2 : L.norm1; }

    void tap(int n_tok) {
        const int ld = embed_.n_in, w = ops_.width;
        std::vector<float> rows(size_t(n_tok) * ld);
        cuda_check(cudaStreamSynchronize(ops_.stream), "tap");
        cuda_check(cudaMemcpy(rows.data(), ops_.x, rows.size() * 4, cudaMemcpyDeviceToHost), "tap");
        for (int t = 0; t < n_tok; t++) {
            const auto row = rows.begin() + long(size_t(rows_asked_[size_t(t)]) * ld);
            tap_->insert(tap_->end(), row, row + w);
        }
    }

    const Design design_;
    LayerOps ops_;
    int max_seqs_, max_ctx_, num_sms_ = 0, n_vocab_ = 0;
    std::vector<Layer> layers_;
    std::vector<Run> runs_;
    Matrix embed_, head_, bigram_, loop_in_;
    int bigram_buckets_ = 0;
    int64_t bigram_prev_ = 0, bigram_cur_ = 0;
    size_t loop_start_ = 0, loop_stop_ = 0;
    int loop_times_ = 0;
    float* x0_ = nullptr;              // the embedding output, kept for the loop
    float* loop_step_ = nullptr;       // what each pass adds to x before its first layer
    float softcap_ = 0.f, embed_scale_ = 1.f;
    Norm final_norm_;
    int* embed_status_ = nullptr;
    size_t weight_bytes_ = 0;
    float* scan_scratch_dev_ = nullptr;
    size_t scan_cap_ = 0;
    std::vector<int> lens_;            // tokens each sequence has run = position of its next one
    std::vector<int32_t> last_token_;  // of each sequence: part of its state where embeddings look at pairs of tokens
    std::vector<int32_t> meta_;
    std::vector<int32_t> lens_sorted_, rows_asked_;  // of the current step: portions in the order they run; row of each token as asked
    int32_t *meta_dev_ = nullptr, *meta_host_ = nullptr;
    size_t meta_cap_ = 0;
    float *logits_dev_ = nullptr, *logits_ = nullptr, *into_ = nullptr;
    int logit_rows_ = 0;
    std::vector<int*> status_words_;
    int* status_host_ = nullptr;
    std::map<std::pair<int, int>, Graph> graphs_;  // by batch size and reach
    const bool use_graphs_ = !(getenv("INGOT_DECODE_GRAPH") && atoi(getenv("INGOT_DECODE_GRAPH")) == 0);
    const int scan_threads_per_sm_ = getenv("INGOT_SCAN_THREADS") ? std::max(1, atoi(getenv("INGOT_SCAN_THREADS"))) : 1024;
    std::vector<float>* tap_ = nullptr;
    cudaEvent_t ev0_ = nullptr, ev1_ = nullptr;
    float last_ms_ = 0.f;
};

// Selective scans, attention beside a gated recurrent unit; gelu feed-forwards.
Design besudra() { return Design{}; }
// Looped latent attention in parallel with squared-relu experts.
Design banevik() {
    Design d;
    d.norm_offset = 1.f;
    d.parallel = d.tied_head = true;
    return d;
}
// Three kinds of grouped-query attention - windowed, without positions, with sinks - between layer norms before and after each part; silu
// feed-forwards and gated experts.
Design silevik() {
    Design d;
    d.centred = d.sandwich = true;
    d.act = 0;
    d.gated_experts = true;
    d.attention = {{"attention", INGOT_QK_NORM_NONE, false, OutputGate::per_value},
                   {"attention_2", INGOT_QK_NORM_HEAD, false, OutputGate::per_head},
                   {"attention_3", INGOT_QK_NORM_ALL, true, OutputGate::none}};
    return d;
}

// Linear recurrences with matrix states and latent attention without sinks behind input convolutions, norms before and after each part, experts
// by token id, passes of a loop that begin by adding a vector.
Design gatuzen() {
    Design d;
    d.sandwich = d.loop_step = true;
    d.act = 0;
    d.gated_experts = d.table_experts = true;
    d.latent.sink = false;
    d.latent.gate = d.latent.paired = true;
    return d;
}

template <Design (*kDesign)()>
std::unique_ptr<ModelBackend> open_design(const ModelDir& dir, const EngineOptions& opt) {
    return std::make_unique<HybridBackend>(dir, opt, kDesign());
}
const RegisterModel kBesudra("Besudra", open_design<besudra>);
const RegisterModel kBanevik("Banevik", open_design<banevik>);
const RegisterModel kSilevik("Silevik", open_design<silevik>);
const RegisterModel kGatuzen("Gatuzen", open_design<gatuzen>);

}  // namespace
