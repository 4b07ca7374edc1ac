"""Recurrences over channels in steps that hold single tokens beside prompts: every form (csrc/scan_routes.h), in one call for all sequences and in one for
the short and one for the long ones, with the states that are left; and whole models."""
import ctypes as C

import numpy as np
import pytest

import hybrid_models as H
import hybrid_reference as R
from hybrid_step import Step, act_out, dev, lib, plan
from ingot_b200 import models as M

pytestmark = pytest.mark.gpu
# The last sequence is the long one. 70 tokens after 63 single ones are the tile kernel's in one call, 300 after three the stream's. A sequence without a token stays as it is.
LENS = [[1, 1, 1, 300], [1] * 63 + [70], [1, 64, 65, 130], [0, 3, 200]]


def calls(lens, apart, chunk, floats):
    """[pos0 -> (step, plan, what keeps them alive)] over the sequences; apart: those of at most 64 tokens first, then the others."""
    def part(a, b):
        def of(pos0):
            st, pl = Step(lens, pos0, list(range(len(lens)))), plan(lens[a:b], chunk, floats)
            step = type(st.c).from_buffer_copy(st.c)
            step.n_tok, step.max_len, step.n_seq = sum(lens[a:b]), max(lens[a:b]), b - a
            for f in ("row_start", "len", "pos0", "slot"):
                setattr(step, f, getattr(step, f) + 4 * a)
            return step, pl.c, (st, pl)
        return of
    small = sum(n <= 64 for n in lens)
    return [part(0, small), part(small, len(lens))] if apart else [part(0, len(lens))]


@pytest.mark.parametrize("apart,chunk", [(False, 10 ** 9), (False, 48), (True, 48), (True, 32)])
@pytest.mark.parametrize("inner,n_state", [(36, 5), (100, 16), (6148, 20)])
@pytest.mark.parametrize("lens", LENS, ids=str)
def test_selective_scan(lens, inner, n_state, apart, chunk):
    import torch
    rng = np.random.default_rng(inner)
    pad, n = lib().ingot_scan_state_pad(n_state), len(lens)
    A = -np.exp(rng.uniform(-3, 2, (inner, n_state)))
    D, bias = rng.standard_normal(inner), rng.uniform(-4, -1, inner)
    a2 = np.zeros((inner, pad))
    a2[:, :n_state] = A * np.log2(np.e)
    a2d, dd, bd = dev(a2), dev(D), dev(bias)
    state = torch.full((n, inner, pad), float("nan"), device="cuda")
    left = np.zeros((n, inner, n_state))
    for begin in (0, 1):
        x, raw, z = ([rng.standard_normal((m, inner)) for m in lens] for _ in range(3))
        B, Cm = ([rng.standard_normal((m, n_state)) for m in lens] for _ in range(2))
        want = []
        for i, m in enumerate(lens):
            dt = R.softplus(raw[i] + bias)
            want.append(R.selective_scan(x[i], dt, A, B[i], Cm[i], D, left[i]) * R.silu(z[i]))
            for t in range(m):
                left[i] = np.exp(dt[t][:, None] * A) * left[i] + (dt[t] * x[i][t])[:, None] * B[i][t]
        want = np.concatenate(want)
        bc = np.zeros((sum(lens), 2 * pad))
        bc[:, :n_state], bc[:, pad:pad + n_state] = np.concatenate(B), np.concatenate(Cm)
        xd, td, zd, bcd = dev(np.concatenate(x)), dev(np.concatenate(raw)), dev(np.concatenate(z)), dev(bc)
        out = torch.full((sum(lens), inner), float("nan"), device="cuda")
        o = act_out(out)
        for call in calls(lens, apart, chunk, inner * (pad + 1)):
            step, p, keep = call([begin * m for m in lens])
            lib(lib().ingot_selective_scan(C.byref(step), C.byref(p), xd.data_ptr(), inner, td.data_ptr(), inner, bd.data_ptr(), bcd.data_ptr(), 2 * pad, 0, pad, zd.data_ptr(),
                                           inner, a2d.data_ptr(), dd.data_ptr(), state.data_ptr(), inner, n_state, 0, C.byref(o), None))
            torch.cuda.synchronize()
        assert np.abs(out.cpu().numpy() - want).max() < 3e-5 * max(1.0, np.abs(want).max())
        some = np.array(lens) > 0
        assert np.abs(state.cpu().numpy()[some, :, :n_state] - left[some]).max() < 3e-5 * max(1.0, np.abs(left).max()) and torch.isnan(state[torch.from_numpy(~some)]).all()


@pytest.mark.parametrize("apart,chunk", [(False, 10 ** 9), (False, 48), (True, 48), (True, 32)])
@pytest.mark.parametrize("width,block", [(40, 8), (257, 257), (4100, 100)])
@pytest.mark.parametrize("lens", LENS, ids=str)
def test_gated_lru(lens, width, block, apart, chunk):
    import torch
    rng = np.random.default_rng(width)
    n = len(lens)
    br, bi, yb = (rng.standard_normal(width) for _ in range(3))
    lam = rng.uniform(-6, 1, width)
    dv = [dev(v) for v in (br, bi, R.softplus(lam), yb)]
    state, left = torch.full((n, width), float("nan"), device="cuda"), np.zeros((n, width))
    for begin in (0, 1):
        u, gr, gi, y = ([rng.standard_normal((m, width)) for m in lens] for _ in range(4))
        want = []
        for i in range(n):
            s = R.gated_lru_scan(u[i], R.sigmoid(gr[i] + br), R.sigmoid(gi[i] + bi), lam, left[i])
            want.append(0.75 * s * R.gelu_tanh(y[i] + yb))
            left[i] = s[-1] if len(s) else left[i]
        want = np.concatenate(want)
        g = np.stack([np.concatenate(gr).reshape(len(want), -1, block), np.concatenate(gi).reshape(len(want), -1, block)], axis=2).reshape(len(want), 2 * width)
        ud, gd, yd = dev(np.concatenate(u)), dev(g), dev(np.concatenate(y))
        out = torch.full((len(want), width), float("nan"), device="cuda")
        o = act_out(out)
        for call in calls(lens, apart, chunk, 2 * width):
            step, p, keep = call([begin * m for m in lens])
            lib(lib().ingot_gated_lru(C.byref(step), C.byref(p), ud.data_ptr(), width, gd.data_ptr(), 2 * width, block, dv[0].data_ptr(), dv[1].data_ptr(), dv[2].data_ptr(),
                                      yd.data_ptr(), width, dv[3].data_ptr(), state.data_ptr(), width, 0.75, 0, C.byref(o), None))
            torch.cuda.synchronize()
        assert np.abs(out.cpu().numpy() - want).max() < 2e-5
        some = np.array(lens) > 0
        assert np.abs(state.cpu().numpy()[some] - left[some]).max() < 2e-5 and torch.isnan(state[torch.from_numpy(~some)]).all()


def test_models_decode_beside_a_prompt(tmp_path):
    """Four sequences decode while another reads its prompt, twice; wide enough that the short ones run apart. Bound as in test_gpu_hybrid_model.py."""
    cfg = H.config([H.mamba(4096, 8, 4, 4), H.parallel(2, 1, 16, 32, 4096, 16, 4)], vocab=96, width=64)
    w = H.random_weights(cfg, 5)
    rng = np.random.default_rng(7)
    tokens = [rng.integers(0, 96, n).tolist() for n in (22, 9, 31, 80, 100, 70)]
    want = [H.reference_logits(cfg, w, t) for t in tokens]
    with M.Model(H.write(tmp_path / "m", cfg, w), max_tokens=1024, max_seqs=6) as m:
        m.step([(i, 0, tokens[i][:-2], []) for i in range(4)])
        for k, prompt in ((2, 4), (1, 5)):
            short = [(i, len(tokens[i]) - k, tokens[i][-k:][:1], [0]) for i in range(4)]
            rows = m.step(short + [(prompt, 0, tokens[prompt], list(range(len(tokens[prompt]))))])
            for i in range(4):
                assert H.off(rows[i:i + 1], want[i][len(tokens[i]) - k:][:1], None) < 4e-2
            assert H.off(rows[4:], want[prompt], None) < 4e-2
