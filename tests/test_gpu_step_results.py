"""Where the logits of a step go (ingot_model_step): into the caller's memory by the device, or by way of the backend's own."""
import ctypes as C
import mmap

import numpy as np
import pytest

import hybrid_models as H
from ingot_b200 import models as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def folder(tmp_path_factory):
    cfg = H.config([H.mamba(44, 10, 6, 3), H.parallel(6, 2, 20, 37, 36, 3, 4, ff=52)], vocab=101, width=42)
    return H.write(tmp_path_factory.mktemp("results"), cfg, H.random_weights(cfg, 1))


def room(kind, count):
    """[count] floats of the caller's, and what has to stay alive (or be called) for them."""
    import torch
    if kind == "pageable":
        out = np.full(count, np.nan, np.float32)
        return out, None
    if kind in ("pinned", "unaligned"):  # "unaligned": 4 bytes past an address that 16-byte stores want
        t = torch.full((count + 1,), float("nan"), pin_memory=True)
        return t.numpy()[kind == "unaligned":][:count], t
    area, rt = mmap.mmap(-1, (count * 4 + mmap.PAGESIZE - 1) // mmap.PAGESIZE * mmap.PAGESIZE), torch.cuda.cudart()
    at = C.addressof(C.c_char.from_buffer(area))
    assert int(rt.cudaHostRegister(at, mmap.PAGESIZE, 0)) == 0  # "begun": only the first page is pinned
    out = np.frombuffer(area, np.float32)[:count]
    out[:] = np.nan
    return out, lambda: rt.cudaHostUnregister(at)


@pytest.mark.parametrize("wanted", [1, 7, 64, 65, 130])
@pytest.mark.parametrize("kind", ["pinned", "unaligned", "pageable", "begun"])
def test_logits_reach_any_memory(folder, kind, wanted):
    """Up to 64 rows are written by a kernel where all of them are pinned, more by the copy engine; other memory is copied to on the host. The
    same bits everywhere, and in the arrays that Model.step returns; the next step finds nothing of it."""
    t = np.random.default_rng(2).integers(0, 101, 140).tolist()
    want = sorted(np.random.default_rng(wanted).permutation(140)[:wanted].tolist())
    with M.Model(folder, max_tokens=256) as m:
        first, after = m.step([(0, 0, t, want)]).copy(), m.step([(0, 140, t[:1], [0])]).copy()
        m.release(0)
        out, held = room(kind, wanted * 101)
        i32 = lambda x: np.array(x, np.int32)
        args = [i32([0]), i32([0]), i32([140]), i32(t), i32([wanted]), i32(want)]
        assert M.lib().ingot_model_step(m.handle, 1, *[a.ctypes.data for a in args], out.ctypes.data) == 0
        kept = out.reshape(wanted, 101).copy()
        got = m.step([(0, 140, t[:1], [0])])
        assert np.array_equal(kept, first) and np.array_equal(got, after)
        assert np.array_equal(out.reshape(wanted, 101), kept)
        if callable(held):
            held()
