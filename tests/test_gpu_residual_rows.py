"""Rows of prompts (backend/residual_norm.cu): which norms a launch has is a matter of their weights."""
import numpy as np
import pytest

import residual_norm as N
import silevik_reference as R
from hybrid_step import dev

pytestmark = pytest.mark.gpu
EPS = 1e-5


@pytest.mark.parametrize("rows", [64, 65])
@pytest.mark.parametrize("n", [2048, 4096])
def test_a_bias_without_a_weight_is_no_norm(n, rows):
    import torch
    rng = np.random.default_rng(n)
    x, product, w, b = rng.standard_normal((rows, n)), rng.standard_normal((1, rows, n)), rng.standard_normal(n) + 1, rng.standard_normal(n)
    want = x + product[0]
    xd, out = dev(x), torch.full((rows, n), float("nan"), device="cuda")
    N.run(xd, EPS, product=dev(product), post=(None, b), next_norm=(w, None), out=out)
    assert np.abs(xd.cpu().numpy() - want).max() < 1e-6 * np.abs(want).max()
    read = R.rms_norm(want, w, EPS)
    assert np.abs(out.cpu().numpy() - read).max() < 2e-5 * np.abs(read).max()
    want = x + R.rms_norm(product[0], w, EPS)
    xd = dev(x)
    N.run(xd, EPS, product=dev(product), post=(w, None), next_norm=(None, b))
    assert np.abs(xd.cpu().numpy() - want).max() < 2e-5 * np.abs(want).max()
