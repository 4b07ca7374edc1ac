"""Streams of recurrences over channels (csrc/recurrent.cu) do the arithmetic of the passes over chunks in their order: a sequence that is alone in its step
(chunks: too few channels for a stream) and many times the same (streams) leave the same bits, outputs and states, over two portions; a sequence that is one
chunk has those of its tokens one after the other. test_scan_routes.py checks that the two take different launches."""
import ctypes as C

import numpy as np
import pytest

from hybrid_step import Step, act_out, dev, lib, plan

pytestmark = pytest.mark.gpu
# (tokens, tokens of a chunk): more chunks than lanes, chunks of whole tiles and of others, of single tokens, two
CUTS = [(1111, 32), (600, 48), (523, 41), (450, 16), (441, 1), (700, 129), (500, 260)]
SCANS = [(128, 3, 36), (124, 16, 36), (120, 20, 36), (128, 32, 36), (192, 3, 49), (192, 16, 49), (188, 24, 49), (192, 31, 49)]  # channels, states, copies: 32 and 64 channels per CTA
UNITS = [(128, 32, 36), (99, 33, 36)]  # channels, block, copies


def token_by_token(run, n):
    """A sequence as one chunk has the bits of its tokens one after the other: in portions too short for a stream."""
    parts, state = [], None
    for a in range(0, n, 64):
        out, state = run(1, 0, state, slice(a, min(n, a + 64)), 10 ** 9)
        parts.append(out[0])
    out, left = run(1, 0, None, slice(None), 10 ** 9)
    assert np.array_equal(out[0].view(np.int32), np.concatenate(parts).view(np.int32)) and np.array_equal(left.view(np.int32), state.view(np.int32))


def both(run, copies):
    """run(copies, portion, state or None) -> (outputs [copies, n, channels], state [copies, ...])."""
    one = many = None
    for portion in (0, 1):
        a, one = run(1, portion, one)
        b, many = run(copies, portion, many)
        for x, y in ((a, b), (one, many)):
            assert np.isfinite(x).all()
            assert all(np.array_equal(x[0].view(np.int32), v.view(np.int32)) for v in y)


@pytest.mark.parametrize("inner,n_state,copies", SCANS)
@pytest.mark.parametrize("n,chunk", CUTS)
def test_selective_scan(n, chunk, inner, n_state, copies):
    """Both widths of a CTA and every number of states per lane; decays from nearly none to fast ones."""
    import torch
    rng = np.random.default_rng(n + inner)
    pad = lib().ingot_scan_state_pad(n_state)
    a2 = np.zeros((inner, pad))
    a2[:, :n_state] = -np.exp(rng.uniform(-6, 2, (inner, n_state)))
    a2d, dd, bd = dev(a2), dev(rng.standard_normal(inner)), dev(rng.uniform(-4, -1, inner))
    x = [[rng.standard_normal((n, w)).astype(np.float32) for w in (inner, inner, inner, 2 * pad)] for _ in range(2)]

    def run(copies, portion, state, rows=slice(None), chunk=chunk):
        x_p = [v[rows] for v in x[portion]]
        m, at = len(x_p[0]), portion * n + (rows.start or 0)
        st, pl = Step([m] * copies, [at] * copies, list(range(copies))), plan([m] * copies, chunk, inner * (pad + 1))
        xd, td, zd, bcd = (dev(np.tile(v, (copies, 1))) for v in x_p)
        state = torch.full((copies, inner, pad), float("nan"), device="cuda") if state is None else dev(state)
        out = torch.full((copies * m, inner), float("nan"), device="cuda")
        o = act_out(out)
        lib(lib().ingot_selective_scan(C.byref(st.c), C.byref(pl.c), xd.data_ptr(), inner, td.data_ptr(), inner, bd.data_ptr(), bcd.data_ptr(), 2 * pad, 0, pad, zd.data_ptr(), inner,
                                       a2d.data_ptr(), dd.data_ptr(), state.data_ptr(), inner, n_state, 0, C.byref(o), None))
        torch.cuda.synchronize()
        return out.cpu().numpy().reshape(copies, m, inner), state.cpu().numpy()

    both(run, copies)
    token_by_token(run, n)


@pytest.mark.parametrize("width,block,copies", UNITS)
@pytest.mark.parametrize("n,chunk", CUTS)
def test_gated_lru(n, chunk, width, block, copies):
    import torch
    rng = np.random.default_rng(n + width)
    dv = [dev(v) for v in (rng.standard_normal(width), rng.standard_normal(width), np.log1p(np.exp(rng.uniform(-6, 1, width))), rng.standard_normal(width))]
    x = [[rng.standard_normal((n, w)).astype(np.float32) for w in (width, 2 * width, width)] for _ in range(2)]

    def run(copies, portion, state, rows=slice(None), chunk=chunk):
        x_p = [v[rows] for v in x[portion]]
        m, at = len(x_p[0]), portion * n + (rows.start or 0)
        st, pl = Step([m] * copies, [at] * copies, list(range(copies))), plan([m] * copies, chunk, 2 * width)
        ud, gd, yd = (dev(np.tile(v, (copies, 1))) for v in x_p)
        state = torch.full((copies, width), float("nan"), device="cuda") if state is None else dev(state)
        out = torch.full((copies * m, width), float("nan"), device="cuda")
        o = act_out(out)
        lib(lib().ingot_gated_lru(C.byref(st.c), C.byref(pl.c), ud.data_ptr(), width, gd.data_ptr(), 2 * width, block, dv[0].data_ptr(), dv[1].data_ptr(), dv[2].data_ptr(),
                                  yd.data_ptr(), width, dv[3].data_ptr(), state.data_ptr(), width, 0.75, 0, C.byref(o), None))
        torch.cuda.synchronize()
        return out.cpu().numpy().reshape(copies, m, width), state.cpu().numpy()

    both(run, copies)
    token_by_token(run, n)
