"""Rows of 128-wide heads are the same bits whichever kernel appends them (csrc/attn_gqa.cu): a prompt at once, and in portions of few tokens."""
import ctypes as C

import numpy as np
import pytest

import silevik_reference as R
from hybrid_step import Step, act_out, dev, lib
from test_gpu_grouped_attention import EPS, F16, Shape, Weights, pad, sequence

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv", [(4, 1), (5, 5), (24, 8)])
@pytest.mark.parametrize("norm,rot,mix", [(None, 128, None), ("head", 0, 0.4), ("whole", 90, 0.7), ("head", 34, None), ("head", 128, None)])
def test_prompt_and_portions(heads, kv, norm, rot, mix):
    """Queries as stored, and the result of one more query over all cached rows."""
    import torch
    s, n = Shape(heads, kv, 128, 128, norm=norm, rot=rot, mix=mix), 97
    x, w = sequence(s, n, np.random.default_rng(heads)), Weights(s, 2)
    p = lambda t: None if t is None else t.data_ptr()
    f, gain = R.frequencies(rot, s.base, None) if rot else (np.zeros(1), 1.0)
    turns, td, fd = dev(f / (2 * np.pi), np.float64), dev([[3, 1, 0, 5, 2, 6, 4]], np.int32), dev([0], np.int32)
    qn, kn = (None if norm is None else dev(a) for a in (w.q, w.k))
    off = np.cumsum([0] + [h * d for h, _, d in s.parts()]).tolist()
    got = []
    for portion in (n, 48):
        h = C.c_void_p()
        lib(lib().ingot_skv_create_joined(C.byref(h), 1, kv, 256, F16, 0, 7))
        try:
            queries = []
            for a in range(0, n, portion):
                m = min(portion, n - a)
                st, q = Step([m], [a], [0]), torch.zeros(m, heads, 128, device="cuda", dtype=torch.float16)
                proj = dev(np.concatenate([pad(v[a:a + m], d) for v, (_, _, d) in zip(x, s.parts())], axis=1))
                first = dev(pad(x[-1][a:a + m], 128))
                lib(lib().ingot_gqa_append(h, 0, C.byref(st.c), p(proj), proj.shape[1], off[0], off[1], off[2], C.byref(s.c), p(qn), p(kn), EPS, p(turns), gain,
                                           p(first) if mix is not None else None, 0, mix or 0.0, p(q), p(td), p(fd), 7, None))
                torch.cuda.synchronize()
                queries.append(q.cpu().numpy())
            st, out = Step([1], [n - 1], [0]), torch.zeros(1, heads * 128, device="cuda")
            q, o = dev(queries[-1][-1:], np.float16), act_out(out)
            lib(lib().ingot_gqa_attend(h, 0, C.byref(st.c), p(q), C.byref(s.c), s.scale, None, None, 0, 0, C.byref(o), p(td), p(fd), 7, 2, None))
            torch.cuda.synchronize()
            got.append((np.concatenate(queries).view(np.int16), out.cpu().numpy().view(np.int32)))
        finally:
            lib().ingot_skv_destroy(h)
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
