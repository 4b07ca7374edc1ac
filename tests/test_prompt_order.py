"""The order of the CTAs of a prompt's attention (csrc/prompt_order.h): which it is, and results on the side that small caches never reach."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# heads, KV heads, tokens, side by side; each measured at least as fast that way (B200)
MEASURED = [(32, 8, 4096, True), (24, 8, 8192, True), (16, 16, 24000, True), (32, 32, 16384, True), (24, 8, 32768, False), (32, 32, 40000, False), (32, 32, 72000, False),
            (64, 64, 32768, False)]


def test_orders_that_were_measured(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    source, exe = tmp_path / "order.cpp", str(tmp_path / "order")
    rows = ", ".join(f"{{{(n * h // kv + 255) // 256}u, {n * kv * 512}ull}}" for h, kv, n, _ in MEASURED)
    source.write_text(f'''#include <cstdio>
#include "prompt_order.h"
int main() {{
    const struct {{ unsigned tiles; unsigned long long bytes; }} cases[] = {{{rows}}};
    for (const auto& c : cases) std::printf("%d", heads_side_by_side(c.tiles, 148, c.bytes));
}}''')
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "inference-agent_b200", "csrc"), str(source), "-o", exe], check=True, timeout=120)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout == "".join(str(int(m[3])) for m in MEASURED)


@pytest.mark.gpu
def test_few_tiles_over_many_keys():
    """700 tokens behind 24900 of 32 heads: 400 MB of keys and values, head after head. Bound: f16 rows, queries and weights."""
    import torch

    import ingot_b200 as ib
    heads, before, n = 32, 24900, 700
    g = torch.Generator("cuda").manual_seed(0)
    kv = ib.KVCache(ib.KV_CONTIGUOUS, 1, heads, before + n)
    k, v = (torch.randn(heads, before + n, 128, device="cuda", generator=g).half() for _ in range(2))
    kv.layer_view(0, "k").copy_(k)
    kv.layer_view(0, "v").copy_(v)
    q = torch.randn(n, heads, 128, device="cuda", generator=g).bfloat16()
    out = ib.attn_prefill(kv, 0, q, before)
    torch.cuda.synchronize()
    assert kv.status() == 0
    seen = torch.arange(before + n, device="cuda")[None, :] <= before + torch.arange(n, device="cuda")[:, None]
    for h in range(heads):
        s = (q[:, h].double() @ k[h].double().T / 128 ** 0.5).masked_fill(~seen, -np.inf)
        want = torch.softmax(s, dim=1) @ v[h].double()
        assert (out[:, h].double() - want).abs().max().item() < 2e-3 * max(1.0, want.abs().max().item())
