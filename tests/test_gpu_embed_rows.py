"""Embedding rows (ingot_support_embed_rows_bf16): the table's values in f32, whatever the length and place of a row; ids outside it give zeros and a status."""
import ctypes as C

import numpy as np
import pytest

from ingot_b200 import models as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 62, 1024, 1028, 4096, 4100, 9000])
@pytest.mark.parametrize("rows,shift", [(1, 0), (7, 0), (7, 1), (300, 0)])
def test_rows(rows, shift, n):
    """shift: the table begins so many values past an aligned address."""
    import torch
    rng = np.random.default_rng(n + rows)
    flat = torch.from_numpy(rng.standard_normal(50 * n + 8).astype(np.float32)).bfloat16().cuda()
    table, ids = flat[shift:shift + 50 * n].view(50, n), rng.integers(0, 50, rows).astype(np.int32)
    if rows > 1:
        ids[1], ids[3] = -1, 50
    out, status = torch.full((rows + 1, n), float("nan"), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    p, idd = C.c_void_p, torch.from_numpy(ids).cuda()
    assert M.lib().ingot_support_embed_rows_bf16(p(out.data_ptr()), p(flat.data_ptr() + 2 * shift), n, 50, p(idd.data_ptr()), rows, C.c_float(0.75), p(status.data_ptr()), None) == 0
    torch.cuda.synchronize()
    held = torch.from_numpy((ids >= 0) & (ids < 50)).cuda()
    want = table[idd.clamp(0, 49).long()].float() * 0.75 * held[:, None]
    assert torch.equal(out[:rows], want) and torch.isnan(out[rows]).all() and status.item() == int(rows > 1)
