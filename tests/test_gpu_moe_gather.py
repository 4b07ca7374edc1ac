"""Rows of experts are copies of their tokens' rows (csrc/moe.cu, ingot_moe_gather), on both sides of the line between a CTA and a warp per row."""
import numpy as np
import pytest

from hybrid_step import dev, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 72, 2048, 4104])
@pytest.mark.parametrize("rows,there", [(1, None), (592, None), (593, None), (1000, 700), (40, 13), (700, 0)])
@pytest.mark.parametrize("planes", [1, 2])
def test_rows_are_copied(planes, rows, there, n):
    import torch
    rng, top = np.random.default_rng(rows + n), 3
    tokens = -(-rows // top)
    src = [torch.randint(-2 ** 15, 2 ** 15, (tokens, n), dtype=torch.int16, device="cuda") for _ in range(planes)]
    out = [torch.full((rows, n), 77, dtype=torch.int16, device="cuda") for _ in range(planes)]
    pair = rng.permutation(tokens * top)[:rows]
    pd, held = dev(pair, np.int32), None if there is None else dev([there], np.int32)
    p = lambda t: None if t is None else t.data_ptr()
    two = lambda v: (p(v[0]), p(v[1]) if planes == 2 else None)
    lib(lib().ingot_moe_gather(*two(out), *two(src), p(pd), rows, p(held), top, n, None))
    torch.cuda.synchronize()
    m, at = rows if there is None else there, torch.from_numpy(pair // top).cuda()
    for s, o in zip(src, out):
        assert torch.equal(o[:m], s[at[:m]]) and (o[m:] == 77).all()
