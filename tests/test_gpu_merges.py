"""Merges of key splits (csrc/attn_decode.cu, csrc/attn_prefill_sm100.cu, csrc/attn_gqa.cu): numbers that are not finite reach the results that see them, and no others;
clusters of key shares at every width of the kernel."""
import numpy as np
import pytest

from helpers import D, H, HKV
from test_gpu_grouped_attention import F16, Shape, Weights, reference, run, sequence

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["decode", "layers", "portion"])
@pytest.mark.parametrize("keys", [300, 1000, 4096, 9000])  # one split, a cluster, few splits, many
def test_numbers_that_are_not_finite(keys, call):
    """One key or value of KV head 2: its three query heads. NaN for a key that is; of a value its own column alone, an infinity as such."""
    import torch

    import ingot_b200 as ib
    g = torch.Generator("cuda").manual_seed(keys)
    k, v = (torch.randn(HKV, keys, D, device="cuda", generator=g).half() for _ in range(2))
    n = 200 if call == "portion" else 1
    q = torch.randn(n, H, D, device="cuda", generator=g)

    def result(k, v):
        layers = 4 if call == "layers" else 1
        kv = ib.KVCache(ib.KV_CONTIGUOUS, layers, HKV, keys)
        for l in range(layers):
            kv.layer_view(l, "k").copy_(k)
            kv.layer_view(l, "v").copy_(v)
        if call == "layers":
            out = torch.empty(layers, 1, H, D, device="cuda")
            ib.attn_decode_layers(kv, 0, q.half()[None].repeat(layers, 1, 1, 1).contiguous(), out, max_seq_len=keys)
        else:
            out = ib.attn_prefill(kv, 0, q.bfloat16(), keys - n) if call == "portion" else ib.attn_decode(kv, 0, q.half(), max_seq_len=keys)
        torch.cuda.synchronize()
        assert kv.status() == 0
        return out.reshape(-1, H, D)

    want, at = result(k, v), keys // 3 if call != "portion" else (keys - n) // 3
    others = [h for h in range(H) if h // (H // HKV) != 2]
    for kind, x in (("key", float("nan")), ("value", float("nan")), ("value", float("inf"))):
        k2, v2 = k.clone(), v.clone()
        (k2 if kind == "key" else v2)[2, at, 5] = x
        got = result(k2, v2)
        assert torch.equal(got[:, others], want[:, others])
        mine = got[:, 6:9]
        if kind == "key":
            assert torch.isnan(mine).all()
        else:
            assert (torch.isnan(mine[..., 5]) if x != x else torch.isposinf(mine[..., 5])).all()
            rest = [d for d in range(D) if d != 5]
            assert torch.equal(mine[..., rest], want[:, 6:9][..., rest])


@pytest.mark.parametrize("keys", [129, 700, 1500])
@pytest.mark.parametrize("dim,vdim", [(64, 64), (80, 48), (128, 128), (144, 200), (256, 256)])
def test_clusters_of_every_width(dim, vdim, keys):
    """Two to eight shares of the keys of heads below, at and above 64, 128 and 256 columns. Bound as in test_gpu_grouped_attention.py."""
    s = Shape(6, 2, dim, vdim, gate="element", sink=True)
    rng = np.random.default_rng(keys + dim)
    w, seqs = Weights(s, 4), [sequence(s, n, rng) for n in (keys + 2, 20)]
    got = run(s, seqs, [[keys, 1, 1], [18, 1, 1]], w, F16, 2)
    for x, y in zip(seqs, got):
        want = reference(s, x, w)
        assert np.abs(y - want).max() < 6e-3 * max(1.0, np.abs(want).max())
