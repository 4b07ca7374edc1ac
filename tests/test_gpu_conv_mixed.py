"""The input convolution of steps in which one portion is much longer than the others, and of more tokens than runs of 4 or 8 have a grid for."""
import ctypes as C

import numpy as np
import pytest

import hybrid_reference as R
from hybrid_step import Step, act_out, dev, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps", [2, 4])
@pytest.mark.parametrize("channels", [24, 2052])
@pytest.mark.parametrize("lens", [[1] * 63 + [300], [1, 2, 3, 4, 5, 9, 700], [400] + [1] * 31 + [7], [1] * 70 + [17, 200], [0] * 40 + [150, 1]], ids=lambda v: f"{len(v)}-{max(v)}")
def test_one_long_portion(lens, channels, taps):
    """Two portions of every sequence, so that slots are read as well as written. Four f32 products and sums per value."""
    import torch
    rng = np.random.default_rng(channels + taps)
    n, w = len(lens), rng.standard_normal((channels, taps))
    xs = [rng.standard_normal((2 * m, channels)) for m in lens]
    want = [R.causal_conv(x, w, np.zeros(channels)) for x in xs]
    wd, state = dev(w), torch.full((n, taps - 1, channels), float("nan"), device="cuda")
    for begin in (0, 1):
        st = Step(lens, [begin * m for m in lens], list(range(n)))
        x = dev(np.concatenate([v[begin * m:(begin + 1) * m] for v, m in zip(xs, lens)]))
        out = torch.full((st.n_tok, channels), float("nan"), device="cuda")
        o = act_out(out)
        lib(lib().ingot_causal_conv(C.byref(st.c), x.data_ptr(), channels, None, wd.data_ptr(), None, taps, channels, 0, state.data_ptr(), C.byref(o), None))
        assert np.abs(out.cpu().numpy() - np.concatenate([v[begin * m:(begin + 1) * m] for v, m in zip(want, lens)])).max() < 2e-5
    got = state.cpu().numpy()
    for i, m in enumerate(lens):
        assert np.isnan(got[i]).all() if m == 0 else np.array_equal(got[i], np.concatenate([np.zeros((taps, channels)), xs[i]])[-(taps - 1):].astype(np.float32))


@pytest.mark.parametrize("lens", [[262200], [524400], [1] * 1100 + [600]], ids=["runs of 8", "runs of 16", "many sequences"])
def test_grids_at_their_limits(lens):
    import torch
    channels, taps = 4, 4
    rng = np.random.default_rng(0)
    w, xs = rng.standard_normal((channels, taps)), [rng.standard_normal((m, channels)).astype(np.float32) for m in lens]
    st, x, wd = Step(lens, [0] * len(lens), list(range(len(lens)))), dev(np.concatenate(xs)), dev(w)
    state, out = torch.full((len(lens), taps - 1, channels), float("nan"), device="cuda"), torch.full((sum(lens), channels), float("nan"), device="cuda")
    o = act_out(out)
    lib(lib().ingot_causal_conv(C.byref(st.c), x.data_ptr(), channels, None, wd.data_ptr(), None, taps, channels, 0, state.data_ptr(), C.byref(o), None))
    padded = [np.concatenate([np.zeros((taps - 1, channels)), v]) for v in xs]
    want = np.concatenate([sum(w[:, j] * v[j:len(v) - (taps - 1 - j)] for j in range(taps)) for v in padded])
    assert np.abs(out.cpu().numpy() - want).max() < 2e-5
    assert np.array_equal(state.cpu().numpy(), np.stack([v[-(taps - 1):] for v in padded]).astype(np.float32))
