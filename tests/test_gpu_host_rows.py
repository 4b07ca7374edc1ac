"""Single-token calls on host rows (ingot_attn_layers_host) whose results lie where their inputs do: the inputs are read before the results are written."""
import pytest

import helpers
from helpers import D

pytestmark = pytest.mark.gpu
H, HKV = 24, 8


@pytest.mark.parametrize("L,keys", [(28, 60), (28, 250), (320, 40)])  # 320 layers: more CTAs than the GPU holds at a time
@pytest.mark.parametrize("at", ["queries", "one head on", "keys", "values", "all"])
def test_results_over_the_inputs(at, L, keys):
    """The same bits as into memory of their own."""
    import torch

    import ingot_b200 as ib
    g = torch.Generator().manual_seed(keys)
    q_n, kv_n = L * H * D, L * HKV * D
    rows = torch.randn(q_n + 2 * kv_n, generator=g)
    k, v = (torch.randn(L, HKV, keys - 1, D, generator=g).half().cuda() for _ in range(2))
    inv = helpers.to_dev(helpers.inv_freq())

    def run(begin):
        """Results from `begin` floats into a block that starts with the inputs."""
        kv = ib.KVCache(ib.KV_CONTIGUOUS, L, HKV, keys)
        for l in range(L):
            kv.layer_view(l, "k")[:, :keys - 1].copy_(k[l])
            kv.layer_view(l, "v")[:, :keys - 1].copy_(v[l])
        block = torch.zeros(2 * q_n + 2 * kv_n).pin_memory()
        block[:len(rows)] = rows
        out = block[begin:begin + q_n].view(L, 1, H, D)
        ib.attn_layers_host(kv, 0, block[:q_n].view(L, 1, H, D), block[q_n:q_n + kv_n].view(L, 1, HKV, D), block[q_n + kv_n:q_n + 2 * kv_n].view(L, 1, HKV, D), out, inv, keys - 1)
        torch.cuda.synchronize()
        assert kv.status() == 0
        return out.clone(), torch.stack([kv.layer_view(l, w)[:, keys - 1].clone() for l in range(L) for w in "kv"]).cpu()

    want = run(q_n + 2 * kv_n)
    got = run({"queries": 0, "one head on": D, "keys": q_n, "values": q_n + kv_n, "all": q_n - 64 * D}[at])
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
