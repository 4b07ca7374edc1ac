// Recurrent mixers of the model-folder backend: selective scan, attention beside a gated linear recurrent unit, and linear recurrences with
// matrix states (gated linear attention, state-space duality).
#include "layer_ops.h"

namespace {

// Selective scan (Mamba): [x | z] = W_in h; x <- silu(conv(x)); [dt | B | C] = W_x x; dt <- W_dt dt; scan; W_o (y silu(z)).
std::vector<float> pad_rows(const std::vector<float>& v, int rows, int cols, int rows_p, int cols_p) {
    std::vector<float> out(size_t(rows_p) * cols_p, 0.f);
    for (int r = 0; r < rows; r++) std::copy(v.begin() + size_t(r) * cols, v.begin() + size_t(r + 1) * cols, out.begin() + size_t(r) * cols_p);
    return out;
}

class SelectiveScanMixer : public Mixer {
public:
    SelectiveScanMixer(LayerOps& ops, const Json& c, const std::string& p) {
        inner_ = get_int(c, "inner");
        states_ = get_int(c, "state", 1, 256);
        taps_ = get_int(c, "conv", 1, 16);
        const int rank = get_int(c, "dt_rank"), d = ops.width;
        const Groups in = flat(inner_), rk = flat(rank);
        ip_ = in.padded;
        np_ = ingot_scan_state_pad(states_);
        rank_p_ = rk.padded;
        w_in_ = ops.matrix(2 * ip_, flat(d).padded, {Part{p + "in", {2 * inner_, d}, {2, inner_, ip_}, flat(d)}});
        conv_w_ = ops.upload(pad_rows(tensor_f32(ops.dir.tensor(p + "conv", {inner_, taps_})), inner_, taps_, ip_, taps_));
        conv_b_ = ops.vector(p + "conv.b", inner_);
        // rows of W_x: dt, B and C each start on a padded place, so that B and C rows can be fetched 16 bytes at a time
        const std::vector<int64_t> x_shape = {rank + 2 * states_, inner_};
        const Groups st = {1, states_, np_};
        w_x_ = ops.matrix(rank_p_ + 2 * np_, ip_, {Part{p + "x", x_shape, rk, in, 0, 0, 0}, Part{p + "x", x_shape, st, in, rank_p_, 0, rank},
                                                   Part{p + "x", x_shape, st, in, rank_p_ + np_, 0, rank + states_}});
        w_dt_ = ops.matrix(ip_, rank_p_, {Part{p + "dt", {inner_, rank}, in, rk}});
        dt_b_ = ops.vector(p + "dt.b", inner_);
        std::vector<float> a = tensor_f32(ops.dir.tensor(p + "A_log", {inner_, states_}));
        for (float& v : a) v = float(-std::exp(double(v)) * 1.4426950408889634);  // exp(dt A) = 2^(dt A log2 e)
        a2_ = ops.upload(pad_rows(a, inner_, states_, ip_, np_));
        d_ = ops.vector(p + "D", inner_);
        w_o_ = ops.matrix(p + "o", flat(d), in);
        conv_state_ = ops.state(size_t(taps_ - 1) * ip_);
        state_ = ops.state(size_t(ip_) * np_);
        plan_ = ops.scan_plan(ip_ * 2, size_t(ip_) * (np_ + 1), !ops.opt.f32 && states_ <= 32 ? ingot_scan::Kind::selective : ingot_scan::Kind::none, ip_, np_);
        ops.need(kProj, 2 * ip_);
        ops.need(kConv, ip_);
        ops.need(kStateIn, rank_p_ + 2 * np_);
        ops.need(kDt, ip_);
        ops.need(kMix, ip_);
    }
    void run(LayerOps& ops, const StepCtx& s, const Norms& n) override {
        float *xz = ops.buf(kProj), *xc = ops.buf(kConv), *dbc = ops.buf(kStateIn), *dt = ops.buf(kDt);
        const int ld_bc = rank_p_ + 2 * np_;
        ops.norm_project(s, xz, w_in_, n.in);
        const ingot_act_out conv = ops.operand(s, xc, ip_, true);
        ingot_check(ingot_causal_conv(&s.st, xz, 2 * ip_, nullptr, conv_w_, conv_b_, taps_, ip_, ops.opt.f32 ? 1 : 2, ops.at_pass(conv_state_, size_t(taps_ - 1) * ip_), &conv, ops.stream));
        ops.operand_ready(s, ip_);
        ops.project(s, dbc, w_x_, xc, ip_);
        ops.project_rows(s, dt, w_dt_, dbc, ld_bc, 2);
        const ingot_act_out y = ops.operand(s, ops.buf(kMix), ip_, false);
        for (const auto& part : s.plans[plan_])
            ingot_check(ingot_selective_scan(&part.st, &part.plan, xc, ip_, dt, ip_, dt_b_, dbc, ld_bc, rank_p_, rank_p_ + np_, xz + ip_, 2 * ip_, a2_, d_,
                                             ops.at_pass(state_, size_t(ip_) * np_), ip_, states_, ops.opt.f32 ? 1 : 0, &y, ops.stream));
        ops.operand_ready(s, ip_);
        ops.project_residual(s, w_o_, ops.buf(kMix), n);
    }

private:
    size_t plan_;
    int inner_, states_, taps_, ip_, np_, rank_p_;
    Matrix w_in_, w_x_, w_dt_, w_o_;
    float *conv_w_, *conv_b_, *dt_b_, *a2_, *d_, *conv_state_, *state_;
};

// Attention beside a gated linear recurrent unit, both reading the same normalised input:
//   left   chunk-local attention over shared key/value rows (ingot_skv_*)
//   right  y = gelu(W_y h + b), u = conv(W_x h + b), gates from block-diagonal products of u, S; output S * y
// x += W_left (left_scale * attention) + W_right (right_scale * recurrence): one input product for the four input matrices
// and one output product over the two results side by side.
class ParallelMixer : public Mixer {
public:
    ParallelMixer(LayerOps& ops, const Json& c, const std::string& p) {
        const Json &l = c.at("left"), &r = c.at("right");
        const int d = ops.width;
        left_scale_ = get_float(c, "left_scale");
        right_scale_ = get_float(c, "right_scale");
        heads_ = get_int(l, "heads");
        kv_heads_ = get_int(l, "kv_heads");
        dim_ = get_int(l, "dim");
        if (heads_ % kv_heads_ != 0) throw std::runtime_error("model config: \"heads\" is not a multiple of \"kv_heads\"");
        if (l.has("vdim") && get_int(l, "vdim") != dim_) throw std::runtime_error("model config: values that are the keys need \"vdim\" equal to \"dim\"");
        scale_ = get_float(l, "scale");
        const int chunk = l.has("mask") && !l.at("mask").is_null() ? get_int(l.at("mask"), "size") : 0;
        const int row = ops.opt.f32 ? round_up(dim_, 8) : ingot_skv_row_length(dim_);
        if (row < 2 || row > 512) throw std::runtime_error("model config: heads of more than 512 values are not supported");
        row_ = row;
        cache_ = ops.cache_group(kv_heads_, row, chunk, 0, CacheGroup::scaled, &cache_layer_);

        width_ = get_int(r, "width");
        const int blocks = get_int(r, "blocks");
        taps_ = get_int(r, "conv", 1, 16);
        if (width_ % blocks != 0) throw std::runtime_error("model config: \"width\" is not a multiple of \"blocks\"");
        const int m = width_ / blocks, mp = round_up(m, 8);
        const Groups q = {heads_, dim_, row}, k = {kv_heads_, dim_, row}, w = {blocks, m, mp}, in = flat(d);
        wp_ = w.width();
        block_ = mp;
        const std::string L = p + "left.", R = p + "right.";
        k_off_ = q.width();
        y_off_ = k_off_ + k.width();
        x_off_ = y_off_ + wp_;
        proj_ld_ = x_off_ + wp_;
        w_in_ = ops.matrix(proj_ld_, in.padded, {Part{L + "q", {q.count(), d}, q, in, 0}, Part{L + "k", {k.count(), d}, k, in, k_off_},
                                                 Part{R + "y", {width_, d}, w, in, y_off_}, Part{R + "x", {width_, d}, w, in, x_off_}});
        q_norm_ = ops.vector(L + "q.norm", {q.count()}, q);
        k_norm_ = ops.vector(L + "k.norm", {k.count()}, k);
        y_b_ = ops.vector(R + "y.b", {width_}, w);
        x_b_ = ops.vector(R + "x.b", {width_}, w);
        std::vector<float> cw = tensor_f32(ops.dir.tensor(R + "conv", {width_, taps_})), cw_p(size_t(wp_) * taps_, 0.f);
        for (int i = 0; i < width_; i++) std::copy(cw.begin() + size_t(i) * taps_, cw.begin() + size_t(i + 1) * taps_, cw_p.begin() + size_t(i / m * mp + i % m) * taps_);
        conv_w_ = ops.upload(cw_p);
        conv_b_ = ops.vector(R + "conv.b", {width_}, w);
        // block b: m rows of the recurrence gate, then m rows of the input gate
        const Groups gate_rows = {blocks, m, 2 * mp}, gate_cols = {1, m, mp};
        w_gates_ = ops.matrix(2 * wp_, mp, {Part{R + "ra", {blocks, m, m}, gate_rows, gate_cols, 0}, Part{R + "ri", {blocks, m, m}, gate_rows, gate_cols, mp}}, 2 * mp);
        r_b_ = ops.vector(R + "ra.b", {blocks, m}, w);
        i_b_ = ops.vector(R + "ri.b", {blocks, m}, w);
        std::vector<float> lam = ops.host_vector(R + "lam", {width_}, w);
        for (float& v : lam) v = float(double(v) > 30 ? double(v) : std::log1p(std::exp(double(v))));
        softplus_lam_ = ops.upload(lam);
        const Groups heads_out = flat(q.count());
        attn_cols_ = heads_out.padded;
        mix_ld_ = attn_cols_ + wp_;
        w_o_ = ops.matrix(in.padded, mix_ld_, {Part{L + "o", {d, q.count()}, in, heads_out, 0, 0}, Part{R + "o", {d, width_}, in, w, 0, attn_cols_}});
        conv_state_ = ops.state(size_t(taps_ - 1) * wp_);
        state_ = ops.state(size_t(wp_));
        plan_ = ops.scan_plan(wp_, 2 * size_t(wp_), ops.opt.f32 ? ingot_scan::Kind::none : ingot_scan::Kind::gated, wp_, 1);
        ops.need(kProj, proj_ld_);
        ops.need(kConv, wp_);
        ops.need(kGates, 2 * wp_);
        ops.need(kMix, mix_ld_);
        ops.need(kQuery, q.width());
    }
    void run(LayerOps& ops, const StepCtx& s, const Norms& n) override {
        float *proj = ops.buf(kProj), *u = ops.buf(kConv), *gates = ops.buf(kGates), *mix = ops.buf(kMix);
        const CacheGroup& g = *cache_;
        ops.norm_project(s, proj, w_in_, n.in);
        const ingot_act_out conv = ops.operand(s, u, wp_, true, 2);
        ingot_check(ingot_causal_conv(&s.st, proj + x_off_, proj_ld_, x_b_, conv_w_, conv_b_, taps_, wp_, 0, ops.at_pass(conv_state_, size_t(taps_ - 1) * wp_), &conv, ops.stream));
        ops.operand_ready(s, wp_, 2);
        ops.project(s, gates, w_gates_, u, wp_);
        ingot_check(ingot_skv_append(g.kv, cache_layer_ + ops.pass, &s.st, proj, proj_ld_, 0, k_off_, heads_, dim_, q_norm_, k_norm_, ops.eps, ops.buf(kQuery),
                                     g.tables, g.first_page, g.width, ops.stream));
        // the two results side by side are the operand of the output product
        const ingot_act_out left = ops.operand(s, mix, mix_ld_, false);
        ingot_check(ingot_skv_attend(g.kv, cache_layer_ + ops.pass, &s.st, ops.buf(kQuery), heads_, dim_, scale_, left_scale_, &left, g.tables, g.first_page, g.width,
                                     0, ops.stream));
        ingot_act_out right = left;
        if (right.f32) right.f32 += attn_cols_;
        if (right.hi) right.hi = static_cast<char*>(right.hi) + size_t(attn_cols_) * 2;
        if (right.lo) right.lo = static_cast<char*>(right.lo) + size_t(attn_cols_) * 2;
        for (const auto& part : s.plans[plan_])
            ingot_check(ingot_gated_lru(&part.st, &part.plan, u, wp_, gates, 2 * wp_, block_, r_b_, i_b_, softplus_lam_, proj + y_off_, proj_ld_, y_b_, ops.at_pass(state_, size_t(wp_)), wp_,
                                        right_scale_, ops.opt.f32 ? 1 : 0, &right, ops.stream));
        ops.operand_ready(s, mix_ld_);
        ops.project_residual(s, w_o_, mix, n);
    }

private:
    size_t plan_;
    int heads_, kv_heads_, dim_, row_, width_, wp_, block_, taps_, cache_layer_ = 0;
    int k_off_, y_off_, x_off_, proj_ld_, attn_cols_, mix_ld_;
    float scale_, left_scale_, right_scale_;
    CacheGroup* cache_;
    Matrix w_in_, w_gates_, w_o_;
    float *q_norm_, *k_norm_, *y_b_, *x_b_, *conv_w_, *conv_b_, *r_b_, *i_b_, *softplus_lam_, *conv_state_, *state_;
};

// What mixers built on a linear recurrence with a matrix state per head share (kernels: csrc/linear_recurrence.cu): the state, the time
// chunks, and the gated norm of the result as the operand of W_o.
class LinearRecurrence {
public:
    LinearRecurrence(LayerOps& ops, int heads, int states, int values) : heads_(heads), states_(states), values_(values), f32_(ops.opt.f32) {
        state_ = ops.state(floats());
        // as many chunks as give every SM two CTAs of the tensor-core kernel, or four of the other one
        plan_ = ops.scan_plan(heads_ * (f32_ ? round_up(vp(), 32) * 8 : vp() * 4), size_t(heads_) * np() * (vp() + 1));
        ops.need(kMix, width());
        ops.need(kConv, width());
    }
    int np() const { return round_up(states_, 16); }
    int vp() const { return round_up(values_, 16); }
    int width() const { return heads_ * vp(); }
    Groups states(int n) const { return {n, states_, np()}; }
    Groups values() const { return {heads_, values_, vp()}; }
    // in: q .. skip; norm: gate .. gate_first. Leaves the operand of W_o (kConv without tensor cores).
    void run(LayerOps& ops, const StepCtx& s, ingot_linear_scan_in in, ingot_gated_norm norm) const {
        float* y = ops.buf(kMix);
        in.n_head = heads_;
        in.n_state = np();
        in.n_value = vp();
        ingot_check(ingot_linear_scan(&s.st, &s.plans[plan_][0].plan, &in, ops.at_pass(state_, floats()), y, width(), s.lens[0], f32_ ? 1 : 0, ops.stream));
        norm.x = y;
        norm.x_ld = width();
        norm.heads = heads_;
        norm.size = values_;
        norm.padded = vp();
        norm.exact = f32_;
        norm.eps = ops.eps;
        const ingot_act_out out = ops.operand(s, ops.buf(kConv), width(), false);
        ingot_check(ingot_gated_norm_rows(&norm, s.st.n_tok, &out, ops.stream));
        ops.operand_ready(s, width());
    }

private:
    size_t floats() const { return size_t(heads_) * np() * vp(); }
    int heads_, states_, values_;
    bool f32_;
    size_t plan_;
    float* state_;
};

// Gated linear attention: S <- diag(alpha) S + k v^T, o = S^T q dim^(-1/2), alpha = sigmoid(W_a2 W_a1 h + b)^(1 / tau) per key channel;
// W_o (rmsnorm(o) silu(W_g h)), the norm over each head. q, k, v, gate and W_a1 are one product.
class GatedLinearMixer : public Mixer {
public:
    GatedLinearMixer(LayerOps& ops, const Json& c, const std::string& p)
        : heads_(get_int(c, "heads")), dim_(get_int(c, "dim", 1, 512)), rec_(ops, heads_, dim_, get_int(c, "vdim")), power_(float(1.0 / c.at("tau").number())) {
        const int d = ops.width;
        const TensorView& a1 = ops.dir.tensor(p + "a1");
        if (a1.shape.size() != 2 || a1.shape[0] < 1 || a1.shape[0] > 65536) throw std::runtime_error("model: tensor " + p + "a1 is not a matrix");
        const Groups in = flat(d), k = rec_.states(heads_), v = rec_.values(), rank = flat(int(a1.shape[0]));
        k_off_ = k.width();
        v_off_ = k_off_ + k.width();
        g_off_ = v_off_ + v.width();
        a_off_ = g_off_ + v.width();
        proj_ld_ = a_off_ + rank.padded;
        w_in_ = ops.matrix(proj_ld_, in.padded, {Part{p + "q", {k.count(), d}, k, in, 0}, Part{p + "k", {k.count(), d}, k, in, k_off_}, Part{p + "v", {v.count(), d}, v, in, v_off_},
                                                 Part{p + "g", {v.count(), d}, v, in, g_off_}, Part{p + "a1", {rank.count(), d}, rank, in, a_off_}});
        w_a2_ = ops.matrix(p + "a2", k, rank);
        bias_ = ops.vector(p + "a2.b", {k.count()}, k);
        const std::vector<float> norm = ops.host_vector(p + "norm", {v.size}, {1, v.size, v.padded});
        std::vector<float> all;
        for (int h = 0; h < heads_; h++) all.insert(all.end(), norm.begin(), norm.end());
        norm_ = ops.upload(all);
        w_o_ = ops.matrix(p + "o", in, v);
        ops.need(kProj, proj_ld_);
        ops.need(kDt, k.width());
    }
    void run(LayerOps& ops, const StepCtx& s, const Norms& n) override {
        float *proj = ops.buf(kProj), *z = ops.buf(kDt);
        ops.norm_project(s, proj, w_in_, n.in);
        ops.project_rows(s, z, w_a2_, proj + a_off_, proj_ld_, 2);
        ingot_linear_scan_in in = {};
        in.share = 1;
        in.decay = INGOT_DECAY_SIGMOID_POWER;
        in.q_scale = 1.f / std::sqrt(float(dim_));
        in.power = power_;
        in.q = proj;
        in.k = proj + k_off_;
        in.v = proj + v_off_;
        in.z = z;
        in.q_ld = in.k_ld = in.v_ld = proj_ld_;
        in.z_ld = k_off_;
        in.bias = bias_;
        ingot_gated_norm norm = {};
        norm.gate = proj + g_off_;
        norm.gate_ld = proj_ld_;
        norm.weight = norm_;
        norm.parts = heads_;
        norm.act = INGOT_GATE_SILU;
        rec_.run(ops, s, in, norm);
        ops.project_residual(s, w_o_, ops.buf(kConv), n);
    }

private:
    int heads_, dim_;
    LinearRecurrence rec_;
    float power_;
    int k_off_, v_off_, g_off_, a_off_, proj_ld_;
    Matrix w_in_, w_a2_, w_o_;
    float *bias_, *norm_;
};

// Mamba-2: [z | x | B | C | dt] = W_in h; x, B, C <- silu(conv(.)); dt <- softplus(dt + dt_bias); per head S <- exp(-exp(A_log) dt) S + dt B x^T,
// y = S^T C + D x, B and C shared by the heads of a group; W_o (rmsnorm(y silu(z))), the norm in equal parts.
class StateSpaceMixer : public Mixer {
public:
    StateSpaceMixer(LayerOps& ops, const Json& c, const std::string& p)
        : heads_(get_int(c, "heads")), groups_(get_int(c, "groups")), taps_(get_int(c, "conv", 1, 16)), parts_(get_int(c, "norm_groups")),
          rec_(ops, heads_, get_int(c, "state", 1, 512), get_int(c, "vdim")) {
        if (heads_ % groups_ != 0) throw std::runtime_error("model config: \"heads\" is not a multiple of \"groups\"");
        const int d = ops.width;
        const Groups in = flat(d), x = rec_.values(), b = rec_.states(groups_), dt = flat(heads_);
        const int inner = x.count(), n = b.count(), rows = 2 * inner + 2 * n + heads_;
        if (inner % parts_ != 0) throw std::runtime_error("model config: the values do not form \"norm_groups\" equal parts");
        x_off_ = x.width();
        b_off_ = x.width();  // from x_off_
        c_off_ = b_off_ + b.width();
        channels_ = c_off_ + b.width();
        dt_off_ = x_off_ + channels_;
        proj_ld_ = dt_off_ + dt.padded;
        auto part = [&](const Groups& g, int at, int from) { return Part{p + "in", {rows, d}, g, in, at, 0, from}; };
        w_in_ = ops.matrix(proj_ld_, in.padded, {part(x, 0, 0), part(x, x_off_, inner), part(b, x_off_ + b_off_, 2 * inner), part(b, x_off_ + c_off_, 2 * inner + n),
                                                 part(dt, dt_off_, 2 * inner + 2 * n)});
        // the convolution's channels in the same places
        const std::vector<float> cw = tensor_f32(ops.dir.tensor(p + "conv", {inner + 2 * n, taps_})), cb = tensor_f32(ops.dir.tensor(p + "conv.b", {inner + 2 * n}));
        std::vector<float> w(size_t(channels_) * taps_, 0.f), bias(size_t(channels_), 0.f);
        auto place = [&](const Groups& g, int at, int from) {
            for (int i = 0; i < g.count(); i++) {
                const int to = at + i / g.size * g.padded + i % g.size;
                std::copy(cw.begin() + long(from + i) * taps_, cw.begin() + long(from + i + 1) * taps_, w.begin() + long(to) * taps_);
                bias[size_t(to)] = cb[size_t(from + i)];
            }
        };
        place(x, 0, 0);
        place(b, b_off_, inner);
        place(b, c_off_, inner + n);
        conv_w_ = ops.upload(w);
        conv_b_ = ops.upload(bias);
        dt_bias_ = ops.vector(p + "dt_bias", {heads_}, {1, heads_, heads_});
        std::vector<float> rate = ops.host_vector(p + "A_log", {heads_}, {1, heads_, heads_});
        for (float& v : rate) v = float(std::exp(double(v)));
        rate_ = ops.upload(rate);
        skip_ = ops.vector(p + "D", {heads_}, {1, heads_, heads_});
        norm_ = ops.vector(p + "norm", {inner}, x);
        w_o_ = ops.matrix(p + "o", in, x);
        conv_state_ = ops.state(size_t(taps_ - 1) * channels_);
        ops.need(kProj, proj_ld_);
        ops.need(kStateIn, channels_);
    }
    void run(LayerOps& ops, const StepCtx& s, const Norms& n) override {
        float *proj = ops.buf(kProj), *xbc = ops.buf(kStateIn);
        ops.norm_project(s, proj, w_in_, n.in);
        ingot_act_out conv = {};
        conv.f32 = xbc;
        conv.ld = channels_;
        ingot_check(ingot_causal_conv(&s.st, proj + x_off_, proj_ld_, nullptr, conv_w_, conv_b_, taps_, channels_, ops.opt.f32 ? 1 : 2,
                                      ops.at_pass(conv_state_, size_t(taps_ - 1) * channels_), &conv, ops.stream));
        ingot_linear_scan_in in = {};
        in.share = heads_ / groups_;
        in.decay = INGOT_DECAY_STEP;
        in.q_scale = 1.f;
        in.q = xbc + c_off_;
        in.k = xbc + b_off_;
        in.v = xbc;
        in.z = proj + dt_off_;
        in.q_ld = in.k_ld = in.v_ld = channels_;
        in.z_ld = proj_ld_;
        in.bias = dt_bias_;
        in.rate = rate_;
        in.skip = skip_;
        ingot_gated_norm norm = {};
        norm.gate = proj;
        norm.gate_ld = proj_ld_;
        norm.weight = norm_;
        norm.parts = parts_;
        norm.act = INGOT_GATE_SILU;
        norm.gate_first = 1;
        rec_.run(ops, s, in, norm);
        ops.project_residual(s, w_o_, ops.buf(kConv), n);
    }

private:
    int heads_, groups_, taps_, parts_;
    LinearRecurrence rec_;
    int x_off_, b_off_, c_off_, channels_, dt_off_, proj_ld_;
    Matrix w_in_, w_o_;
    float *conv_w_, *conv_b_, *dt_bias_, *rate_, *skip_, *norm_, *conv_state_;
};

}  // namespace

std::unique_ptr<Mixer> make_selective_scan(LayerOps& ops, const Json& config, const std::string& prefix) {
    return std::make_unique<SelectiveScanMixer>(ops, config, prefix);
}
std::unique_ptr<Mixer> make_parallel(LayerOps& ops, const Json& config, const std::string& prefix) {
    return std::make_unique<ParallelMixer>(ops, config, prefix);
}
std::unique_ptr<Mixer> make_gated_linear(LayerOps& ops, const Json& config, const std::string& prefix) {
    return std::make_unique<GatedLinearMixer>(ops, config, prefix);
}
std::unique_ptr<Mixer> make_state_space(LayerOps& ops, const Json& config, const std::string& prefix) {
    return std::make_unique<StateSpaceMixer>(ops, config, prefix);
}
