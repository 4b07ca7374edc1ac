"""The recurrent / latent-attention / table-routed design's own mechanisms in whole models (the tests shared with the other designs are in
test_gpu_hybrid_model.py): the residual stream run by run, memory over tiles and portions, strong decays, passes of a loop, every constant."""
import json

import numpy as np
import pytest

import gatuzen_models as G
import hybrid_models as H
from ingot_b200 import models as M

pytestmark = pytest.mark.gpu
TOL = {True: 3e-5, False: 0.12}


def open_model(tmp, cfg, w, **kw):
    return M.Model(H.write(tmp, cfg, w), **kw)


def three_kinds(**kw):
    return G.config([G.mamba2(4, 2, 12, 14, conv=3, norm_groups=2, mlp=G.moe(3, 1, 20)), G.latent(3, 12, 12, 20, 10, scaling=(4.0, 128, 8.0, 1.0), mlp=G.moe(5, 2, 24)),
                     G.gla(2, 16, 20, tau=6.0, mlp=G.moe(4, 4, 16))], vocab=70, width=52, loop=(1, 3, 2), **kw)


def feed(m, seq, tokens, cuts):
    out, at, k = [], 0, 0
    while at < len(tokens):
        n = min(cuts[k % len(cuts)], len(tokens) - at)
        out.append(m.step([(seq, at, tokens[at:at + n], list(range(n)))]))
        at += n
        k += 1
    return np.concatenate(out)


@pytest.mark.parametrize("f32", [True, False])
def test_residual_stream_after_every_layer_run(tmp_path, f32):
    """Taken before what the next pass adds."""
    cfg = three_kinds()
    w = G.random_weights(cfg, 4)
    t = np.random.default_rng(0).integers(0, 70, 90).tolist()
    want = []
    G.reference_logits(cfg, w, t, want)
    with open_model(tmp_path, cfg, w, f32=f32, max_tokens=128) as m:
        m.tap()
        m.step([(0, 0, t[:80], [79])])
        whole = m.residuals().reshape(5, 80, 52)
        for p in range(80, 90):
            m.step([(0, p, t[p:p + 1], [0])])
        single = m.residuals().reshape(10, 5, 52).transpose(1, 0, 2)
    for g, x in zip(np.concatenate([whole, single], axis=1), want):
        assert np.abs(g - x).max() < (1e-5 if f32 else 4e-2) * np.abs(x).max()


def far_token(kind):
    """A layer, and a sequence in which token 5, the only one of its kind, stands out in every key; decays are next to none."""
    layer = {"gla": G.gla(2, 16, 16, tau=64.0), "mamba2": G.mamba2(2, 1, 16, 16), "latent": G.latent(2, 16, 4, 24, 16, base=1e6, scale=0.8)}[kind]
    cfg = G.config([layer], vocab=40, width=32, groups=1, taps=2, residual_mult=1.0)
    w = G.random_weights(cfg, 3)
    t = np.random.default_rng(2).integers(2, 40, 700).tolist()
    t[5] = 1
    w["embed"][1] = 0
    w["embed"][1, 0] = 8.0
    w["embed"][2:, 0] = 0
    if kind == "gla":
        w["l0.mix.a2.b"][:] = 5.0
        w["l0.mix.k"][:, 0] = 4.0
        w["l0.mix.q"][:, 1:] += 0.25
    elif kind == "mamba2":
        w["l0.mix.A_log"][:] = -8.0
        w["l0.mix.in"][32:80, 0] = 6.0  # its x and B
        w["l0.mix.D"][:] = 0.1
    else:
        w["l0.mix.dkv"][:24, 0] = 4.0
        w["embed"][2:, 1] = 3.0         # all other tokens have in common what asks for it
        key = w["l0.mix.uk"] @ w["l0.mix.dkv.norm"]
        for h in range(2):
            w["l0.mix.q"][h * 20:h * 20 + 16, 1] = 0.5 * np.sign(key[h * 16:h * 16 + 16])
    return cfg, G.rounded(w), t


@pytest.mark.parametrize("kind", ["gla", "mamba2", "latent"])
@pytest.mark.parametrize("f32", [True, False])
def test_a_far_token_decides(tmp_path, f32, kind):
    """Taking it away shows hundreds of tokens later, at the end of the prompt and in decoded tokens, whatever the portions."""
    cfg, w, t = far_token(kind)
    want = G.reference_logits(cfg, w, t)
    other = list(t)
    other[5] = 2
    assert H.error(G.reference_logits(cfg, w, other), want)[650:].max() > 3 * TOL[f32]
    with open_model(tmp_path, cfg, w, f32=f32, max_tokens=768) as m:
        for cuts in ([700], [300, 390] + [1] * 10, [100, 2, 17, 64]):
            assert H.error(feed(m, 0, t, cuts), want).max() < TOL[f32], cuts
            m.release(0)


@pytest.mark.parametrize("taps", [1, 2, 4, 9])
@pytest.mark.parametrize("f32", [True, False])
def test_reach_of_the_input_convolutions(tmp_path, taps, f32):
    """A layer whose mixer is silenced: a token is seen by its feed-forward up to taps - 1 tokens later and not beyond, across portions."""
    cfg = G.config([G.gla(1, 8, 8, mlp=G.moe(2, 1, 24))], vocab=60, width=32, taps=taps)
    w = G.random_weights(cfg, taps)
    w["l0.norm1b"][:] = 0
    w["l0.mlp.table"][:] = 0
    t = np.random.default_rng(1).integers(0, 60, 60).tolist()
    with open_model(tmp_path, cfg, w, f32=f32, max_tokens=64) as m:
        for cuts in ([60], [16, 2, 1, 1, 3, 1], [20] + [1] * 40):
            def logits(tokens):
                out = feed(m, 0, tokens, cuts)
                m.release(0)
                return out
            base = logits(t)
            for j in (0, 15, 17, 30):
                other = list(t)
                other[j] = (t[j] + 7) % 60
                moved = np.abs(logits(other) - base).max(axis=1)
                assert not moved[:j].any() and not moved[j + taps:].any()
                assert (moved[j:j + taps] > 1e-6).all()


@pytest.mark.parametrize("f32", [True, False])
def test_experts_that_a_table_names_more_than_once(tmp_path, f32):
    """Token ids whose rows name an expert twice or three times: it counts as often, for steps of few tokens and of many."""
    cfg = G.config([G.gla(2, 24, 16, mlp=G.moe(4, 3, 32)), G.mamba2(3, 1, 16, 16)], vocab=50, width=40)
    w = G.random_weights(cfg, 6)
    w["l0.mlp.table"][::2] = 1
    w["l0.mlp.table"][1::4, 2] = w["l0.mlp.table"][1::4, 0]
    t = np.random.default_rng(3).integers(0, 50, 330).tolist()
    want = H.reference_logits(cfg, w, t)
    with open_model(tmp_path, cfg, w, f32=f32, max_tokens=384) as m:
        for cuts in ([330], [20, 22, 60, 64, 100, 61, 1, 1, 1]):
            assert H.error(feed(m, 0, t, cuts), want).max() < TOL[f32], cuts
            m.release(0)


@pytest.mark.parametrize("f32", [True, False])
def test_strong_decays(tmp_path, f32):
    """Powers of the sigmoid that lose a state within a few tokens, or one token, beside rows that keep it."""
    cfg = G.config([G.gla(2, 24, 16, tau=0.5, mlp=G.moe(2, 1, 16)), G.mamba2(3, 1, 16, 16)], vocab=50, width=40)
    w = G.random_weights(cfg, 5)
    b = w["l0.mix.a2.b"]
    b[::3], b[1::3], b[2::3] = 12.0, -3.0, -30.0
    w["l1.mix.A_log"][:] = [4.0, 1.0, -6.0]
    w["l1.mix.dt_bias"][:] = [3.0, 0.0, -2.0]
    t = np.random.default_rng(3).integers(0, 50, 230).tolist()
    want = G.reference_logits(cfg, w, t)
    with open_model(tmp_path, cfg, w, f32=f32, max_tokens=256) as m:
        for cuts in ([230], [9, 33, 64, 2], [150] + [1] * 80):
            assert H.error(feed(m, 0, t, cuts), want).max() < TOL[f32]
            m.release(0)


@pytest.mark.parametrize("expand", ["0", "2", "40", "1000000"])
def test_the_kernels_a_portion_takes_do_not_show(tmp_path, monkeypatch, expand):
    """Portions of all sizes of several sequences beside single tokens: latent attention on the rows or on expanded keys, recurrences token by
    token or in tiles, against the plain implementation."""
    monkeypatch.setenv("INGOT_LATENT_EXPAND", expand)
    cfg = G.config([G.latent(6, 40, 24, 70, 40, scale=0.15, mlp=G.moe(4, 2, 32)), G.gla(3, 24, 40, mlp=None), G.mamba2(4, 2, 20, 24, mlp=G.moe(2, 2, 40)),
                    G.latent(4, 16, 8, 48, 72)], vocab=40, width=48)
    w = G.random_weights(cfg, 4)
    rng = np.random.default_rng(0)
    tokens = [rng.integers(0, 40, n).tolist() for n in (600, 330, 150)]
    want = [G.reference_logits(cfg, w, t) for t in tokens]
    with open_model(tmp_path, cfg, w, max_tokens=1152, max_seqs=3, max_step_tokens=320) as m:
        at, got = [0, 0, 0], [[], [], []]
        cuts = [[150, 2, 100, 1, 180, 3, 64], [40, 1, 39, 130, 120], [1, 2, 41, 100, 6]]
        for k in range(40):
            step = []
            for s in range(3):
                n = min(cuts[s][k % len(cuts[s])], len(tokens[s]) - at[s])
                if n > 0:
                    step.append((s, at[s], tokens[s][at[s]:at[s] + n], list(range(n))))
            if not step:
                break
            rows, r = m.step(step), 0
            for s, p, t, _ in step:
                got[s].append(rows[r:r + len(t)])
                r += len(t)
                at[s] += len(t)
        assert at == [600, 330, 150]
        for s in range(3):
            assert H.error(np.concatenate(got[s]), want[s]).max() < TOL[False], s


def test_passes_and_sequences_have_states_of_their_own(tmp_path):
    """Two sequences whose tokens alternate, in slots that change hands; a pass of the loop never sees another's state."""
    cfg = G.config([G.gla(2, 8, 8, mlp=G.moe(2, 1, 8)), G.mamba2(2, 1, 8, 8)], vocab=50, width=32, loop=(0, 2, 3))
    w = G.random_weights(cfg, 2)
    rng = np.random.default_rng(3)
    a, b, c = (rng.integers(0, 50, n).tolist() for n in (60, 33, 21))
    wa, wb, wc = (G.reference_logits(cfg, w, x) for x in (a, b, c))
    one = dict(cfg, loop={"start": 0, "stop": 2, "times": 1})
    w1 = dict(w, **{"loop.step": w["loop.step"][:1]})
    assert H.error(G.reference_logits(one, w1, a), wa).max() > 0.1
    with open_model(tmp_path, cfg, w, f32=True, max_tokens=192, max_seqs=2) as m:
        got_a, got_b = [], []
        for at_a, n_a, at_b, n_b in ((0, 7, 0, 2), (7, 2, 2, 20), (9, 30, 22, 1), (39, 1, 23, 10)):
            rows = m.step([(1, at_b, b[at_b:at_b + n_b], list(range(n_b))), (0, at_a, a[at_a:at_a + n_a], list(range(n_a)))])
            got_b.append(rows[:n_b])
            got_a.append(rows[n_b:])
        m.release(1)
        got_c = []
        for k in range(20):  # c takes b's slot while a goes on
            rows = m.step([(0, 40 + k, a[40 + k:41 + k], [0]), (1, k, c[k:k + 1], [0])])
            got_a.append(rows[:1])
            got_c.append(rows[1:])
        assert H.error(np.concatenate(got_a), wa).max() < 3e-5 and H.error(np.concatenate(got_b), wb).max() < 3e-5
        assert H.error(np.concatenate(got_c), wc[:20]).max() < 3e-5


@pytest.mark.parametrize("f32", [True, False])
def test_single_tokens_on_the_streaming_kernels(tmp_path, f32):
    """Widths the weight-streaming products of single tokens take, experts included."""
    cfg = G.config([G.mamba2(8, 2, 32, 64, norm_groups=2, mlp=G.moe(3, 2, 256)), G.latent(4, 32, 32, 64, 64, scale=0.1, mlp=G.moe(4, 1, 256)), G.gla(4, 64, 64, mlp=G.moe(2, 2, 512))],
                   vocab=300, width=256)
    w = G.random_weights(cfg, 9)
    t = np.random.default_rng(5).integers(0, 300, 70).tolist()
    want = G.reference_logits(cfg, w, t)
    with open_model(tmp_path, cfg, w, f32=f32, max_tokens=128, max_seqs=2) as m:
        got = np.concatenate([m.step([(0, 0, t[:3], [0, 1, 2])])] + [m.step([(0, p, t[p:p + 1], [0])]) for p in range(3, 70)])
    assert H.error(got, want).max() < TOL[f32]


def changes():
    mixer = lambda i, *k: ("layers", i, "mixer") + k
    return [(("logit_scale",), 1.25), (("embedding", "scale"), 0.2), (("norm", "eps"), 0.3), (("norm", "groups"), 4), (("norm", "groups"), 1), (("residual_mult",), 1.0),
            (("residual_mult",), 0.3), (mixer(1, "scale"), 0.6), (mixer(1, "rot", "base"), 50.0), (mixer(1, "rot", "scaling", "factor"), 9.0),
            (mixer(1, "rot", "scaling", "original"), 2000), (mixer(1, "rot", "scaling", "fast"), 1.5), (mixer(1, "rot", "scaling", "slow"), 0.02), (mixer(2, "tau"), 1.0),
            (mixer(0, "norm_groups"), 4), (mixer(0, "norm_groups"), 1), (("loop", "stop"), 2)]


def changed(cfg, path, value):
    c = json.loads(json.dumps(cfg))
    at = c
    for k in path[:-1]:
        at = at[k]
    at[path[-1]] = value
    return c


def test_constants_come_from_the_configuration(tmp_path):
    cfg = three_kinds()
    w = G.random_weights(cfg, 1)
    t = np.random.default_rng(4).integers(0, 70, 60).tolist()
    base = G.reference_logits(cfg, w, t)
    for i, (path, value) in enumerate(changes()):
        c = changed(cfg, path, value)
        want = G.reference_logits(c, w, t)
        assert H.error(want, base).max() > 1e-4, path
        with open_model(tmp_path / str(i), c, w, f32=True, max_tokens=64) as m:
            assert H.error(m.step([(0, 0, t, list(range(60)))]), want).max() < 5e-5, path


def test_what_a_configuration_may_leave_out(tmp_path):
    """No loop, no input convolutions, one group of the norms, no scaled rotation."""
    cfg = G.config([G.gla(2, 8, 12, mlp=G.moe(2, 1, 16)), G.latent(2, 8, 6, 16, 12), G.mamba2(2, 1, 8, 8)], vocab=50, width=32, taps=1)
    w = G.random_weights(cfg, 8)
    for n in [n for n in w if ".canon" in n]:
        w[n][:] = 0
    t = np.random.default_rng(6).integers(0, 50, 50).tolist()
    bare = json.loads(json.dumps(cfg))
    bare["norm"]["groups"] = 1
    bare["residual_mult"] = 1.0
    del bare["layers"][1]["mixer"]["rot"]["scaling"]
    want = G.reference_logits(bare, w, t)
    del bare["canon"], bare["norm"]["groups"], bare["residual_mult"]
    bare["loop"] = None
    bare["layers"][2].pop("mlp")
    w = {k: v for k, v in w.items() if ".canon" not in k}
    for f32 in (True, False):
        with open_model(tmp_path / str(f32), bare, w, f32=f32, max_tokens=64) as m:
            assert H.error(feed(m, 0, t, [30, 2, 1]), want).max() < TOL[f32]


def test_refusals(tmp_path):
    cfg = three_kinds()
    w = G.random_weights(cfg)

    def refused(change, text, name, weights=w):
        c = json.loads(json.dumps(cfg))
        change(c)
        with pytest.raises(M.ModelError, match=text):
            open_model(tmp_path / name, c, weights)
    mixer = lambda c, i: c["layers"][i]["mixer"]
    refused(lambda c: c["norm"].update(groups=3), "norm.groups", "a")
    refused(lambda c: mixer(c, 0).update(groups=3), "multiple", "b")
    refused(lambda c: mixer(c, 0).update(norm_groups=5), "equal parts", "c")
    refused(lambda c: mixer(c, 1)["rot"].update(dims=7), "even", "d")
    refused(lambda c: mixer(c, 1)["rot"].update(dims=14), "at most", "e")
    refused(lambda c: c["canon"].update(taps=3), "shape", "f")
    refused(lambda c: c["loop"].update(times=3), "shape", "g")
    refused(lambda c: c["layers"][2].update(type="mamba3"), "unknown layer type", "h")
    refused(lambda c: c["canon"].update(taps=17), "taps", "i")
    nothing = lambda c: None
    high = dict(w, **{"l0.mlp.table": w["l0.mlp.table"] + 1})
    refused(nothing, "does not exist", "j", high)
    refused(nothing, "expected I32", "k", dict(w, **{"l0.mlp.table": w["l0.mlp.table"].astype(np.float32)}))
    refused(nothing, "a1 is missing", "l", {k: v for k, v in w.items() if k != "l2.mix.a1"})
