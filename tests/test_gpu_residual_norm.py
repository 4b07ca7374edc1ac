"""The residual sum with norms before and after it (backend/residual_norm.cu) against the plain statement, at lengths on both sides of every
launch shape, padded or not."""
import numpy as np
import pytest

import gatuzen_reference as G
import residual_norm as N
import silevik_reference as R
from hybrid_step import dev

pytestmark = pytest.mark.gpu
EPS = 1e-5
SIZES = [(8, 5), (48, 48), (1024, 1021), (1032, 1030), (4096, 4096), (4104, 4100), (8192, 8191), (9000, 8999)]


def plain(x, pair):
    return R.rms_norm(x, pair[0], EPS) if pair[1] is None else R.layer_norm(x, *pair, EPS)


@pytest.mark.parametrize("centred", [True, False])
@pytest.mark.parametrize("n,count", SIZES)
def test_every_term(n, count, centred):
    import torch
    rng = np.random.default_rng(n)
    rows, slices, top = 5, 3, 2
    pad = lambda a: np.pad(a, [(0, 0)] * (a.ndim - 1) + [(0, n - count)])
    x, product, branch = 40 + rng.standard_normal((rows, count)), rng.standard_normal((slices, rows, count)), rng.standard_normal((7, count))
    pairs = [(rng.standard_normal(count) + 1, rng.standard_normal(count) if centred else None) for _ in range(3)]
    gain, self_gain = rng.random(rows), rng.standard_normal(rows)
    self_gain[2] = 0.0
    row_of = np.array([[0, 6], [-1, 3], [2, -1], [-1, -1], [5, 1]])
    y = product.sum(axis=0) * gain[:, None] + self_gain[:, None] * plain(x, pairs[0])
    for r, t in zip(range(rows), row_of):
        y[r] += sum(branch[i] for i in t if i >= 0)
    want = x + plain(y, pairs[1])
    read = plain(want, pairs[2])
    xd = dev(pad(x))
    out = torch.full((rows, n), float("nan"), device="cuda")
    hi, lo = (torch.full((rows, n), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    N.run(xd, EPS, count, product=dev(pad(product)), gain=dev(gain), branch=dev(pad(branch)), row_of=dev(row_of, np.int32), top=top, self_gain=dev(self_gain), self_norm=pairs[0],
          post=pairs[1], next_norm=pairs[2], out=out, hi=hi, lo=lo)
    assert np.abs(xd.cpu().numpy()[:, :count] - want).max() < 2e-4 and not xd.cpu().numpy()[:, count:].any()
    got = out.cpu().numpy()
    assert np.abs(got[:, :count] - read).max() < (3e-4 if centred else 2e-5) * np.abs(read).max() and not got[:, count:].any()
    assert ((hi.float() + lo.float() - out).abs().max() <= 1e-4 * out.abs().max()).item()


@pytest.mark.parametrize("rows", [64, 65, 593, 1200])
@pytest.mark.parametrize("n", [2048, 4096])
@pytest.mark.parametrize("kind", ["rms", "centred", "groups"])
def test_many_rows(n, rows, kind):
    """Rows of a prompt, on both sides of the line to the launch that keeps the weights, one or several rows per CTA; slices, gains, branch rows, and
    without each of the norms. Bounds as in test_every_term."""
    import torch
    rng = np.random.default_rng(n + rows)
    top, groups = 3, 4 if kind == "groups" else 1
    x, product, branch = 4 + rng.standard_normal((rows, n)), rng.standard_normal((2, rows, n)), rng.standard_normal((40, n))
    pairs = [(rng.standard_normal(n) + 1, rng.standard_normal(n) if kind == "centred" else None) for _ in range(2)]
    gain, row_of = rng.random(rows), rng.integers(-1, 40, (rows, top))
    norm = (lambda v, p: G.grouped_rms_norm(v, p[0], groups, EPS)) if groups > 1 else plain
    y = product.sum(axis=0) * gain[:, None] + (branch[row_of] * (row_of >= 0)[:, :, None]).sum(axis=1)
    for post, following, terms in ((True, True, True), (False, True, True), (True, False, True), (False, True, False)):
        want = x + ((norm(y, pairs[0]) if post else y) if terms else 0)
        xd, out = dev(x), torch.full((rows, n), float("nan"), device="cuda")
        hi, lo = (torch.full((rows, n), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
        given = dict(product=dev(product), gain=dev(gain), branch=dev(branch), row_of=dev(row_of, np.int32), top=top) if terms else {}
        N.run(xd, EPS, n, post=pairs[0] if post else None, next_norm=pairs[1] if following else None, out=out, hi=hi, lo=lo, groups=groups, **given)
        assert np.abs(xd.cpu().numpy() - want).max() < 2e-4
        if following:
            read = norm(want, pairs[1])
            assert np.abs(out.cpu().numpy() - read).max() < 3e-4 * np.abs(read).max()
            assert ((hi.float() + lo.float() - out).abs().max() <= 1e-4 * out.abs().max()).item()


def test_a_norm_alone_of_chosen_rows():
    import torch
    rng = np.random.default_rng(0)
    x, pair = rng.standard_normal((9, 64)), (rng.standard_normal(64), rng.standard_normal(64))
    xd, out = dev(x), torch.zeros(3, 64, device="cuda")
    N.run(xd, EPS, rows=dev([7, 0, 7], np.int32), next_norm=pair, out=out)
    assert np.abs(out.cpu().numpy() - R.layer_norm(x[[7, 0, 7]], *pair, EPS)).max() < 1e-5
    assert np.array_equal(xd.cpu().numpy(), x.astype(np.float32))  # x is only read


def test_the_variance_is_taken_around_the_mean():
    """Values with a mean a thousand times their spread: squares would lose it."""
    import torch
    x = 3000.0 + np.arange(256.0)[None] % 7
    xd, out = dev(x), torch.zeros(1, 256, device="cuda")
    N.run(xd, EPS, next_norm=(np.ones(256), np.zeros(256)), out=out)
    assert np.abs(out.cpu().numpy() - R.layer_norm(x, 1.0, 0.0, EPS)).max() < 1e-3


@pytest.mark.parametrize("n,count,groups", [(8, 6, 2), (48, 46, 2), (192, 192, 4), (256, 256, 2), (1024, 1024, 8), (2048, 2048, 4), (4096, 4096, 2), (4096, 4096, 32), (4104, 4100, 5),
                                             (8192, 8192, 2), (9216, 9216, 3), (16, 16, 16)])
def test_norms_in_groups_and_a_vector_for_all_rows(n, count, groups):
    import torch
    rng = np.random.default_rng(n + groups)
    rows = 4
    pad = lambda a: np.pad(a, [(0, 0)] * (a.ndim - 1) + [(0, n - count)])
    size = np.repeat(10.0 ** rng.uniform(-2, 2, groups), count // groups)  # groups of very different size: a value in the wrong one shows
    x, product, shift = rng.standard_normal((rows, count)) * size, rng.standard_normal((2, rows, count)) * size[::-1], rng.standard_normal(count)
    w = [rng.standard_normal(count) + 1 for _ in range(2)]
    for post, add in ((True, True), (True, False), (False, True)):
        want = x + (G.grouped_rms_norm(product.sum(axis=0), w[0], groups, EPS) if post else 0) + (shift if add else 0)
        read = G.grouped_rms_norm(want, w[1], groups, EPS)
        xd, out = dev(pad(x)), torch.full((rows, n), float("nan"), device="cuda")
        N.run(xd, EPS, count, product=dev(pad(product)) if post else None, post=(w[0], None) if post else None, next_norm=(w[1], None), out=out, groups=groups,
              shift=dev(pad(shift[None])) if add else None)
        assert np.abs(xd.cpu().numpy()[:, :count] - want).max() < 2e-6 * np.abs(want).max() and not xd.cpu().numpy()[:, count:].any()
        assert np.abs(out.cpu().numpy()[:, :count] - read).max() < 2e-5 * np.abs(read).max() and not out.cpu().numpy()[:, count:].any()


def test_a_vector_alone():
    x, v = np.ones((3, 8)), np.arange(8.0)
    xd = dev(x)
    N.run(xd, EPS, shift=dev(v[None]))
    assert np.array_equal(xd.cpu().numpy(), x + v)


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("n,count,groups", [(48, 46, 2), (1024, 1024, 1), (2048, 2048, 4), (4096, 4095, 1), (8192, 8192, 2), (9216, 9216, 3)])
def test_convolution_of_single_tokens(n, count, groups, taps):
    """Token by token, three sequences in slots that hold what earlier ones left: the norm's results convolved over each sequence."""
    import torch
    rng = np.random.default_rng(n + taps)
    pad = lambda a: np.pad(a, [(0, 0)] * (a.ndim - 1) + [(0, n - count)])
    steps, slots, began = 6, [2, 0, 3], [0, 0, 2]  # the third sequence begins later
    w, taps_w = rng.standard_normal(count) + 1, rng.standard_normal((count, taps))
    cw = dev(np.pad(taps_w, [(0, n - count), (0, 0)]))
    state = torch.full((4, max(taps - 1, 1), n), float("nan"), device="cuda")
    xs = rng.standard_normal((steps, 3, count))
    want = [G.causal_conv(G.grouped_rms_norm(xs[b:, s], w, groups, EPS), taps_w) for s, b in enumerate(began)]
    for t in range(steps):
        who = [s for s in range(3) if t >= began[s]]
        xd = dev(pad(xs[t, who]))
        out = torch.full((len(who), n), float("nan"), device="cuda")
        hi, lo = (torch.full((len(who), n), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(2))
        N.run(xd, EPS, count, next_norm=(w, None), out=out, hi=hi, lo=lo, groups=groups,
              conv=(cw, state, dev([slots[s] for s in who], np.int32), dev([t - began[s] for s in who], np.int32)))
        got = out.cpu().numpy()
        for r, s in enumerate(who):
            assert np.abs(got[r, :count] - want[s][t - began[s]]).max() < 3e-5 and not got[r, count:].any()
        assert ((hi.float() + lo.float() - out).abs().max() <= 1e-4 * out.abs().max()).item()
