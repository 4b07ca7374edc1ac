"""The framework's work as its users have it done: attention over a KV cache through the library's entry points, and model folders
through the step function.

Attention calls have the shape of Llama-3.2-3B (24 query and 8 KV heads of 128, f16 cache, 28 layers where all layers are meant). Models
are four layers at the widths of the benchmarks, random weights, 32768-row output matrix: selective scans with a parallel layer
("besudra"), grouped-query attention with dense feed-forwards ("silevik"), matrix-state recurrences and latent attention with experts by
token id ("gatuzen"). A model is opened once per process, as a serving program does; every pass starts its sequences again at position 0.
"""
import copy
import json
import math
import os
import shutil
import sys
import tempfile
import zlib

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inference-agent_b200"))
import ingot_b200 as ib  # noqa: E402
from ingot_b200 import grouped_bench, hybrid_bench, matrix_bench  # noqa: E402
from ingot_b200 import models as M  # noqa: E402

H, HKV, D, LAYERS, BLOCK, VOCAB = 24, 8, 128, 28, 16, 32768


def listed():
    return [
        # One token's attention in all layers at once over full caches: what the reference's own benchmark of its decode attention runs.
        {"name": "decode, 28 layers at once", "kind": "layers", "keys": 4096},
        # A generated token of a chat: append and attention layer after layer, replayed as the graph a decoding loop keeps.
        {"name": "decode, layer by layer", "kind": "token", "keys": 1000},
        # The smallest call: one token whose rows are in host memory, early in a conversation.
        {"name": "decode from host rows", "kind": "host", "keys": 300},
        # A serving step: one new token for each of 64 sequences of mixed length on a paged cache.
        {"name": "decode, 64 paged sequences", "kind": "paged", "seqs": 64, "shortest": 256, "longest": 8192, "pick": 3},
        # The next portion of a long prompt.
        {"name": "prompt portion of 512", "kind": "portion", "tokens": 512, "before": 3584},
        # A whole long document.
        {"name": "prompt of 32768", "kind": "prompt", "tokens": 32768},
        # A short question and its answer, one user.
        {"name": "besudra, one request", "kind": "requests", "model": "besudra", "size": "w2048", "seqs": 1, "prompt": 45, "new": 16},
        # Reading a prompt; ordinary and large.
        {"name": "besudra, prompt of 2048", "kind": "requests", "model": "besudra", "size": "w4096", "seqs": 1, "prompt": 2048, "new": 0},
        {"name": "silevik, prompt of 4096", "kind": "requests", "model": "silevik", "size": "w4096", "seqs": 1, "prompt": 4096, "new": 0},
        # Several users at a time: ragged prompts in one step, then their answers together.
        {"name": "silevik, 8 requests", "kind": "requests", "model": "silevik", "size": "w2048", "seqs": 8, "prompt": 250, "new": 16},
        {"name": "gatuzen, prompt of 1000", "kind": "requests", "model": "gatuzen", "size": "w2048", "seqs": 1, "prompt": 1000, "new": 0},
        {"name": "gatuzen, 4 requests", "kind": "requests", "model": "gatuzen", "size": "w2048", "seqs": 4, "prompt": 30, "new": 16},
    ]


def draw(rng):
    def log(lo, hi):
        return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))
    kind = rng.choice(["layers", "token", "host", "paged", "portion", "prompt", "requests", "requests", "requests", "requests", "requests", "requests"])
    if kind == "layers":
        return {"kind": kind, "keys": log(300, 8192)}
    if kind == "token":
        return {"kind": kind, "keys": log(40, 4096)}
    if kind == "host":
        return {"kind": kind, "keys": log(20, 4096)}
    if kind == "paged":
        return {"kind": kind, "seqs": log(2, 64), "shortest": log(20, 256), "longest": log(512, 8192), "pick": rng.randrange(1000)}
    if kind == "portion":
        return {"kind": kind, "tokens": log(65, 1024), "before": rng.randrange(7000)}
    if kind == "prompt":
        return {"kind": kind, "tokens": log(1024, 32768)}
    model, size = rng.choice([("besudra", "w2048"), ("besudra", "w4096"), ("silevik", "w2048"), ("silevik", "w4096"), ("gatuzen", "w2048")])
    if rng.random() < 0.5:
        return {"kind": kind, "model": model, "size": size, "seqs": 1, "prompt": log(200, 1500 if model == "gatuzen" else 4096), "new": 0}
    seqs = log(1, 16)
    return {"kind": kind, "model": model, "size": size, "seqs": seqs, "prompt": log(8, 300), "new": rng.randint(6, 16)}


# ---- attention ------------------------------------------------------------------------------------------------------

def generator(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed) & 0x7FFFFFFF)


def normal(g, *shape, dtype=torch.float32):
    return torch.randn(shape, generator=g, device=g.device, dtype=torch.float32).to(dtype)


def inv_freq():
    return (500000.0 ** (-torch.arange(0, D, 2, dtype=torch.float64) / D)).float().cuda()


def lengths(case):
    """Keys of each sequence, the new token's included."""
    rng = np.random.default_rng([case["pick"], 1])
    return rng.integers(case["shortest"], case["longest"] + 1, size=case["seqs"]).astype(np.int32)


def attention_inputs(case, seed):
    """What the calls of the case are given, drawn in a fixed order. k, v: the cache's rows, [layer][head][position][128]."""
    g, kind = generator(seed), case["kind"]
    x = {}
    if kind in ("layers", "token", "host"):
        n = case["keys"]
        x["k"], x["v"] = (normal(g, LAYERS, HKV, n, D, dtype=torch.float16) for _ in range(2))
        if kind == "layers":
            x["q"] = normal(g, LAYERS, 1, H, D, dtype=torch.float16)
        else:
            x["new_q"], x["new_k"], x["new_v"] = normal(g, LAYERS, 1, H, D), normal(g, LAYERS, 1, HKV, D), normal(g, LAYERS, 1, HKV, D)
    elif kind == "paged":
        blocks = int(((lengths(case) + BLOCK - 1) // BLOCK).sum())
        x["k"], x["v"] = (normal(g, blocks, HKV, BLOCK, D, dtype=torch.float16) for _ in range(2))
        x["order"] = torch.randperm(blocks, generator=g, device="cuda")
        x["new_q"], x["new_k"], x["new_v"] = normal(g, case["seqs"], H, D), normal(g, case["seqs"], HKV, D), normal(g, case["seqs"], HKV, D)
    elif kind == "portion":
        n = case["tokens"]
        x["k"], x["v"] = (normal(g, 1, HKV, case["before"] + n, D, dtype=torch.float16) for _ in range(2))
        x["new_q"], x["new_k"], x["new_v"] = normal(g, n, H, D), normal(g, n, HKV, D), normal(g, n, HKV, D)
    else:
        x["k"], x["v"] = (normal(g, 1, HKV, case["tokens"], D, dtype=torch.float16) for _ in range(2))
        x["q"] = normal(g, case["tokens"], H, D, dtype=torch.bfloat16)
    return x


def block_tables(case, order):
    """[sequences][most blocks]: the sequences' blocks follow one another in `order`."""
    nb = (lengths(case) + BLOCK - 1) // BLOCK
    table, at = np.full((len(nb), int(nb.max())), -1, dtype=np.int32), 0
    order = order.cpu().numpy()
    for i, n in enumerate(nb):
        table[i, :n] = order[at:at + n]
        at += n
    return table


class Layers:
    """What torch sees of all layers of a contiguous cache, [layer][head][position][128]; the cache lives as long as its views."""

    def __init__(self, kv, which):
        self.kv = kv
        fn = ib.lib().ingot_kv_k_dev if which == "k" else ib.lib().ingot_kv_v_dev
        self.__cuda_array_interface__ = {"shape": (kv.n_layer, kv.n_head_kv, kv.capacity, D), "typestr": "<f2", "data": (fn(kv.handle, 0), False), "version": 2}


def prepare_attention(case, seed):
    x, kind = attention_inputs(case, seed), case["kind"]
    s = {"kind": kind, "inv": inv_freq()}
    if kind == "paged":
        lens = lengths(case)
        kv = ib.KVCache(ib.KV_PAGED, 1, HKV, x["k"].shape[0], max_seqs=case["seqs"])
        kv.layer_view(0, "k").copy_(x["k"])
        kv.layer_view(0, "v").copy_(x["v"])
        s.update(lens=torch.from_numpy(lens).cuda(), longest=int(lens.max()), positions=torch.from_numpy(lens - 1).cuda(),
                 ids=torch.arange(case["seqs"], dtype=torch.int32, device="cuda"), tables=torch.from_numpy(block_tables(case, x["order"])).cuda())
    else:
        kv = ib.KVCache(ib.KV_CONTIGUOUS, x["k"].shape[0], HKV, x["k"].shape[2])
        s["ks"], s["vs"] = (torch.as_tensor(Layers(kv, w), device=torch.device("cuda", torch.cuda.current_device())) for w in "kv")
        s["ks"].copy_(x["k"])
        s["vs"].copy_(x["v"])
    s["kv"] = kv
    if kind in ("layers", "prompt"):
        s["q"], s["out"] = x["q"], torch.empty(x["q"].shape, device="cuda")
        return s
    s["new"] = tuple(x[n] for n in ("new_q", "new_k", "new_v"))
    if kind == "portion":
        s["pos"] = case["before"]
        s["rows"] = [c[0, :, s["pos"]:] for c in (s["ks"], s["vs"])]
    elif kind in ("token", "host"):
        s["pos"] = case["keys"] - 1
        s["rows"] = [c[:, :, s["pos"]] for c in (s["ks"], s["vs"])]
    if kind == "host":
        # one pinned block, so that the rows of all layers travel in one copy
        block = torch.empty(sum(t.numel() for t in s["new"]), pin_memory=True)
        parts, at = [], 0
        for t in s["new"]:
            parts.append(block[at:at + t.numel()].view(t.shape).copy_(t))
            at += t.numel()
        s["new"], s["out"] = tuple(parts), torch.empty((LAYERS, 1, H, D), pin_memory=True)
    if kind == "token":
        s["out"] = torch.empty((LAYERS, 1, H, D), device="cuda")
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            one_token(s)  # sizes the handle's scratch
            side.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"], stream=side):
                one_token(s)
        torch.cuda.current_stream().wait_stream(side)
    return s


def one_token(s):
    q, k, v = s["new"]
    for l in range(LAYERS):
        rotated = ib.rope_kv_append(s["kv"], l, q[l], k[l], v[l], s["inv"], s["pos"])
        ib.attn_decode(s["kv"], l, rotated, out=s["out"][l], max_seq_len=s["pos"] + 1)


def run_attention(s):
    kind, kv = s["kind"], s["kv"]
    if kind == "layers":
        return ib.attn_decode_layers(kv, 0, s["q"], s["out"], max_seq_len=kv.capacity)
    if kind == "token":
        s["graph"].replay()
        return [s["out"], *s["rows"]]
    if kind == "host":
        ib.attn_layers_host(kv, 0, *s["new"], s["out"], s["inv"], s["pos"])
        torch.cuda.current_stream().synchronize()  # the caller reads the host rows
        return [s["out"], *s["rows"]]
    if kind == "prompt":
        return ib.attn_prefill(kv, 0, s["q"], 0, out=s["out"])
    q, k, v = s["new"]
    if kind == "paged":
        rotated = ib.rope_kv_append(kv, 0, q, k, v, s["inv"], positions=s["positions"], seq_ids=s["ids"], block_tables=s["tables"])
        return ib.attn_decode(kv, 0, rotated, seq_lens=s["lens"], max_seq_len=s["longest"], block_tables=s["tables"])
    rotated = ib.rope_kv_append(kv, 0, q, k, v, s["inv"], s["pos"])
    return [ib.attn_prefill(kv, 0, rotated, s["pos"]), *s["rows"]]


def turned(x, positions):
    """Neighbouring pairs of the last axis turned by position times frequency (f32 angles, as the models define them). x [token][head][128]."""
    angle = (positions.float()[:, None] * inv_freq()).double()[:, None, :]
    c, s = angle.cos(), angle.sin()
    u, v = x.double()[..., 0::2], x.double()[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2)


def causal(q, k, v, pos0):
    """q [token][24][128] at positions pos0 + i, k, v [8][key][128], all 64 bits."""
    n, keys = q.shape[0], k.shape[1]
    out = torch.empty(n, H, D, dtype=torch.float64, device=q.device)
    for h in range(H):
        kk, vv = k[h // (H // HKV)], v[h // (H // HKV)]
        for a in range(0, n, 4096):
            b = min(n, a + 4096)
            end = min(keys, pos0 + b)
            s = q[a:b, h] @ kk[:end].T / D ** 0.5
            s.masked_fill_(torch.arange(end, device=q.device)[None, :] > pos0 + torch.arange(a, b, device=q.device)[:, None], -math.inf)
            out[a:b, h] = torch.softmax(s, dim=1) @ vv[:end]
    return out


def exact_attention(case, seed):
    x, kind = attention_inputs(case, seed), case["kind"]
    if kind == "layers":
        return torch.stack([causal(x["q"][l].double(), x["k"][l].double(), x["v"][l].double(), case["keys"] - 1) for l in range(LAYERS)])
    if kind == "prompt":
        return causal(x["q"].double(), x["k"][0].double(), x["v"][0].double(), 0)
    if kind == "paged":
        outs, table = [], block_tables(case, x["order"])
        for i, n in enumerate(lengths(case).tolist()):
            at = torch.from_numpy(table[i, :(n + BLOCK - 1) // BLOCK].astype(np.int64)).cuda()
            k, v = (x[c][at].double().transpose(0, 1).reshape(HKV, -1, D)[:, :n].clone() for c in "kv")
            p = torch.tensor([n - 1], device="cuda")
            k[:, n - 1], v[:, n - 1] = turned(x["new_k"][i:i + 1], p)[0], x["new_v"][i].double()
            outs.append(causal(turned(x["new_q"][i:i + 1], p), k, v, n - 1))
        return torch.cat(outs)
    if kind == "portion":
        pos = torch.arange(case["before"], case["before"] + case["tokens"], device="cuda")
        k, v = x["k"][0].double(), x["v"][0].double()
        k[:, case["before"]:], v[:, case["before"]:] = turned(x["new_k"], pos).transpose(0, 1), x["new_v"].double().transpose(0, 1)
        return [causal(turned(x["new_q"], pos), k, v, case["before"]), k[:, case["before"]:], v[:, case["before"]:]]
    pos, outs, rows = torch.tensor([case["keys"] - 1], device="cuda"), [], ([], [])
    for l in range(LAYERS):
        k, v = x["k"][l].double(), x["v"][l].double()
        k[:, -1], v[:, -1] = turned(x["new_k"][l], pos)[0], x["new_v"][l, 0].double()
        outs.append(causal(turned(x["new_q"][l], pos), k, v, case["keys"] - 1))
        rows[0].append(k[:, -1])
        rows[1].append(v[:, -1])
    return [torch.stack(outs), torch.stack(rows[0]), torch.stack(rows[1])]


def attention_work(case):
    """Cached rows read once, queries in and results out; both products over the keys that are seen."""
    kind, row = case["kind"], HKV * D * 2 * 2
    if kind in ("layers", "token", "host"):
        new = 0 if kind == "layers" else LAYERS * ((H + 2 * HKV) * D * 4 + row)
        q = LAYERS * H * D * (2 + 4) if kind == "layers" else LAYERS * H * D * 4
        return {"bytes": LAYERS * case["keys"] * row + new + q, "flops": 4 * LAYERS * H * D * case["keys"]}
    if kind == "paged":
        keys = int(lengths(case).sum())
        return {"bytes": keys * row + case["seqs"] * ((2 * H + 2 * HKV) * D * 4 + row), "flops": 4 * H * D * keys}
    n, before = case["tokens"], case.get("before", 0)
    flops = 4 * H * D * (n * before + n * (n + 1) // 2)
    if kind == "portion":
        return {"bytes": (before + n) * row + n * (2 * H + 2 * HKV) * D * 4 + n * row, "flops": flops}
    return {"bytes": n * row + n * H * D * (2 + 4), "flops": flops}


# ---- models ---------------------------------------------------------------------------------------------------------

BENCH = {"besudra": hybrid_bench, "silevik": grouped_bench, "gatuzen": matrix_bench}


def model_config(case):
    cfg = copy.deepcopy(BENCH[case["model"]].config(case["size"]))
    if case["model"] == "silevik":  # dense feed-forwards in every layer: close choices of a router have no tolerance
        for layer in cfg["layers"]:
            layer["mlp"] = copy.deepcopy(cfg["layers"][0]["mlp"])
    return cfg


def weight(model, cfg, name, shape):
    """A tensor of the model, the same for every seed: bf16, or int32 for a table of experts."""
    g = generator(zlib.crc32(name.encode()))
    if name.endswith("table"):
        experts = cfg["layers"][int(name[1:name.index(".")])]["mlp"]["router"]["experts"]
        return torch.rand(shape[0], experts, generator=g, device="cuda").argsort(dim=1)[:, :shape[1]].int()
    x = torch.randn(shape, generator=g, device="cuda")
    if "norm" in name:
        x = 0.1 * x + (0 if name.endswith(".b") and model == "silevik" else 1)
    elif name.endswith("vmix"):
        x = 0.5 + 0.1 * x
    elif name.endswith(("dt.b", "dt_bias")):
        x = x - 3
    elif name.endswith("a2.b"):
        x = x + 2
    elif len(shape) > 1 and not (name == "embed" or model == "besudra" and name.endswith(("conv", "A_log"))):
        x = x / shape[-1] ** 0.5
    return x.bfloat16()


_open = {}


def opened(case):
    """The model of the case, opened once per process. Its folder is gone again by then: the weights are on the device."""
    key = (case["model"], case["size"])
    if key not in _open:
        cfg, tensors = model_config(case), {}
        for name, shape in BENCH[case["model"]].weight_shapes(cfg).items():
            w = weight(case["model"], cfg, name, shape)
            tensors[name] = ("I32", w.cpu().numpy()) if w.dtype == torch.int32 else ("BF16", w.view(torch.int16).cpu().numpy().view(np.uint16))
        folder = tempfile.mkdtemp(prefix="ingot_cases_")
        try:
            with open(os.path.join(folder, "config.json"), "w") as f:
                json.dump(cfg, f)
            M.write_safetensors(os.path.join(folder, "model.safetensors"), tensors)
            _open[key] = M.Model(folder, max_tokens=8192, max_seqs=16, max_step_tokens=4800)
        finally:
            shutil.rmtree(folder, ignore_errors=True)
    return _open[key]


def prompts(case):
    """Lengths of the prompts: one as long as asked, the others down to about half of it."""
    return [case["prompt"] - i * case["prompt"] // (2 * case["seqs"]) for i in range(case["seqs"])]


def tokens(case, seed):
    """One array per sequence: the prompt and what is generated after it."""
    rng = np.random.default_rng(seed)
    return [rng.integers(0, VOCAB, n + case["new"]).astype(np.int32) for n in prompts(case)]


def run_model(s):
    model, ids, lens = s["model"], s["ids"], s["lens"]
    out = [model.step([(i, 0, t[:n], [n - 1]) for i, (t, n) in enumerate(zip(ids, lens))])]
    for j in range(s["new"]):
        out.append(model.step([(i, n + j, t[n + j:n + j + 1], [0]) for i, (t, n) in enumerate(zip(ids, lens))]))
    return out


def model_work(case):
    """Weights read once per step (of experts, those that the step's tokens can need), the logits out; products of every token, attention over
    what is seen and the recurrences as they are stated."""
    cfg = model_config(case)
    shapes, lens, new, seqs = BENCH[case["model"]].weight_shapes(cfg), prompts(case), case["new"], case["seqs"]
    n_all, d = sum(lens) + seqs * new, cfg["width"]
    shared = expert = flops = 0
    for name, shape in shapes.items():
        if len(shape) < 2 or name in ("embed", "head") or name.endswith(("table", "conv", "canon1", "canon2", "A_log")):
            continue
        size = math.prod(shape)
        if ".mlp.e" in name:
            expert += size
        else:
            shared += size
            per = shape[0] * shape[2] if len(shape) == 3 else 1
            flops += 2 * n_all * size if per else 0
    r = cfg["layers"][0]["mlp"]["router"] if case["model"] == "gatuzen" else None
    part = (lambda n: min(1.0, n * r["top"] / r["experts"])) if r else (lambda n: 0.0)
    if r:
        flops += 2 * n_all * expert * r["top"] / r["experts"]
    head = VOCAB * d
    bytes_ = 2 * (shared + head) * (1 + new) + 2 * expert * (part(sum(lens)) + new * part(seqs)) + (1 + new) * seqs * VOCAB * 4 + n_all * d * 2
    flops += 2 * (1 + new) * seqs * head
    for layer in cfg["layers"]:
        m, t = layer["mixer"], layer["type"]
        for n in lens:
            if t in ("gla", "mamba2"):
                flops += 4 * (n + new) * m["heads"] * m["vdim"] * (m["dim"] if t == "gla" else m["state"])
                continue
            if t == "mamba1":
                flops += 6 * (n + new) * m["inner"] * m["state"]
                continue
            a = m["left"] if t == "parallel" else m
            width = a["heads"] * (a["dim"] + a.get("rot_dim", 0) + a["vdim"])
            flops += width * (n + new) * (n + new + 1)  # windows and chunks are at most half of a quarter less at the largest size
    return {"bytes": bytes_, "flops": flops}


# The models once more in 64 bits, a sequence at a time. W(name): the tensor in 64 bits.

def rms(x, w, eps, groups=1):
    p = x.reshape(*x.shape[:-1], groups, -1)
    return (p / (p.square().mean(-1, keepdim=True) + eps).sqrt()).reshape(x.shape) * w


def layer_norm(x, w, b, eps):
    c = x - x.mean(-1, keepdim=True)
    return c / (c.square().mean(-1, keepdim=True) + eps).sqrt() * w + b


def softplus(z):
    return torch.logaddexp(z, torch.zeros_like(z))


def conv(x, w, b=None):
    y = torch.zeros_like(x) if b is None else b.expand_as(x).clone()
    for j in range(w.shape[1]):
        back = w.shape[1] - 1 - j
        if back < len(x):
            y[back:] += w[:, j] * x[:len(x) - back]
    return y


def attend(q, k, v, scale, seen, sink=None):
    """q [n][heads][d], k, v [n][kv heads][d]; seen [n][n]."""
    out = []
    for h in range(q.shape[1]):
        g = h // (q.shape[1] // k.shape[1])
        s = (q[:, h] @ k[:, g].T * scale).masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(len(s), 1)], dim=1)
        out.append(torch.softmax(s, dim=1)[:, :len(k)] @ v[:, g])
    return torch.stack(out, dim=1)


def positions(n, rot):
    f = [float(rot["base"]) ** (-2.0 * i / rot["dims"]) for i in range(rot["dims"] // 2)]
    gain, c = 1.0, rot.get("scaling")
    if c:
        def turning(t):
            return rot["dims"] * math.log(c["original"] / (2 * math.pi * t)) / (2 * math.log(float(rot["base"])))
        lo, hi = max(math.floor(turning(c["fast"])), 0), min(math.ceil(turning(c["slow"])), rot["dims"] - 1)
        part = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(len(f))]
        f, gain = [v / c["factor"] * p + v * (1 - p) for v, p in zip(f, part)], 0.1 * math.log(c["factor"]) + 1.0
    return torch.arange(n, dtype=torch.float64, device="cuda")[:, None, None] * torch.tensor(f, dtype=torch.float64, device="cuda"), gain


def rotate(x, rot):
    angle, gain = positions(len(x), rot)
    u, v, rest = x[..., 0:rot["dims"]:2], x[..., 1:rot["dims"]:2], x[..., rot["dims"]:]
    c, s = gain * angle.cos(), gain * angle.sin()
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2), rest], dim=-1)


def visible(n, window=0, chunk=0):
    i, j = torch.arange(n, device="cuda")[:, None], torch.arange(n, device="cuda")[None, :]
    seen = j <= i
    if window:
        seen &= i - j < window
    if chunk:
        seen &= i // chunk == j // chunk
    return seen


def gated(h, W, p, act):
    g = h @ W(p + "gate").T
    return ((torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * (h @ W(p + "up").T)) @ W(p + "down").T


def scan_mixer(h, W, p, m):
    n, rank = m["state"], m["dt_rank"]
    x, z = (h @ W(p + "in").T).split(m["inner"], dim=1)
    x = torch.nn.functional.silu(conv(x, W(p + "conv"), W(p + "conv.b")))
    dt, b, c = (x @ W(p + "x").T).split([rank, n, n], dim=1)
    dt = softplus(dt @ W(p + "dt").T + W(p + "dt.b"))
    a, s, y = -W(p + "A_log").exp(), torch.zeros(m["inner"], n, dtype=torch.float64, device="cuda"), []
    for t in range(len(x)):
        s = torch.exp(dt[t][:, None] * a) * s + (dt[t] * x[t])[:, None] * b[t]
        y.append(s @ c[t])
    return ((torch.stack(y) + W(p + "D") * x) * torch.nn.functional.silu(z)) @ W(p + "o").T


def parallel_mixer(h, W, p, m, eps):
    a, b, n = m["left"], m["right"], len(h)
    q, k = h @ W(p + "left.q").T, h @ W(p + "left.k").T
    heads = [rms(q, W(p + "left.q.norm"), eps).reshape(n, a["heads"], -1), rms(k, W(p + "left.k.norm"), eps).reshape(n, a["kv_heads"], -1), k.reshape(n, a["kv_heads"], -1)]
    left = attend(*heads, a["scale"], visible(n, chunk=a["mask"]["size"])).reshape(n, -1) @ W(p + "left.o").T
    y = torch.nn.functional.gelu(h @ W(p + "right.y").T + W(p + "right.y.b"), approximate="tanh")
    u = conv(h @ W(p + "right.x").T + W(p + "right.x.b"), W(p + "right.conv"), W(p + "right.conv.b"))
    gate = lambda w: torch.sigmoid((torch.einsum("nbi,boi->nbo", u.reshape(n, b["blocks"], -1), W(p + w)) + W(p + w + ".b")).reshape(n, -1))  # noqa: E731
    log_a = -8.0 * gate("right.ra") * softplus(W(p + "right.lam"))
    a_t, x, s, out = log_a.exp(), torch.sqrt(-torch.expm1(2 * log_a)) * gate("right.ri") * u, torch.zeros_like(u[0]), []
    for t in range(n):
        s = a_t[t] * s + x[t]
        out.append(s)
    return m["left_scale"] * left + m["right_scale"] * ((torch.stack(out) * y) @ W(p + "right.o").T)


def besudra(ids, W, cfg):
    eps, x = cfg["norm"]["eps"], W("embed")[ids]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        h = rms(x, W(p + "norm1"), eps)
        x = x + (scan_mixer(h, W, p + "mix.", m) if layer["type"] == "mamba1" else parallel_mixer(h, W, p + "mix.", m, eps))
        if layer["mlp"]:
            x = x + gated(rms(x, W(p + "norm2"), eps), W, p + "mlp.", "gelu")
    return rms(x, W("final.norm"), eps)


def silevik(ids, W, cfg):
    eps, first, n = cfg["norm"]["eps"], None, len(ids)
    x = W("embed")[ids] * cfg["embedding"]["scale"]
    norm = lambda v, name: layer_norm(v, W(name), W(name + ".b"), eps)  # noqa: E731
    for i, layer in enumerate(cfg["layers"]):
        p, m, kind = f"l{i}.", layer["mixer"], layer["type"]
        h, q = norm(x, p + "norm1"), p + "mix."
        queries, keys = h @ W(q + "q").T, h @ W(q + "k").T
        if kind == "attention_3":
            queries, keys = rms(queries, W(q + "q.norm"), eps), rms(keys, W(q + "k.norm"), eps)
        queries, keys = queries.reshape(n, m["heads"], -1), keys.reshape(n, m["kv_heads"], -1)
        if kind == "attention_2":
            queries, keys = rms(queries, W(q + "q.norm"), eps), rms(keys, W(q + "k.norm"), eps)
        else:
            queries, keys = rotate(queries, m["rot"]), rotate(keys, m["rot"])
        v = (h @ W(q + "v").T).reshape(n, m["kv_heads"], -1)
        if first is None:
            first = v
        else:
            v = (1 - W(q + "vmix")) * v + W(q + "vmix") * first
        y = attend(queries, keys, v, m["scale"], visible(n, window=m["mask"]["size"] if m.get("mask") else 0), W(q + "sink") if kind == "attention_3" else None)
        if kind == "attention_2":
            y = y * torch.sigmoid(h @ W(q + "g").T)[:, :, None]
        y = y.reshape(n, -1)
        if kind == "attention":
            y = y * torch.sigmoid(h @ W(q + "g").T)
        x = x + norm(y @ W(q + "o").T, p + "norm1b")
        x = x + norm(gated(norm(x, p + "norm2"), W, p + "mlp.", "silu"), p + "norm2b")
    return norm(x, "final.norm") * cfg["logit_scale"]


def recurrence(q, k, v, decay):
    """q, k, decay [n][heads][states], v [n][heads][values]."""
    s, out = torch.zeros(*k.shape[1:], v.shape[2], dtype=torch.float64, device="cuda"), []
    for t in range(len(q)):
        s = decay[t][:, :, None] * s + k[t][:, :, None] * v[t][:, None, :]
        out.append(torch.einsum("hnv,hn->hv", s, q[t]))
    return torch.stack(out)


def gatuzen_mixer(h, W, p, m, kind, eps):
    n, heads = len(h), m["heads"]
    split = lambda x: x.reshape(n, heads, -1)  # noqa: E731
    if kind == "gla":
        z = split((h @ W(p + "a1").T) @ W(p + "a2").T + W(p + "a2.b"))
        y = recurrence(split(h @ W(p + "q").T) * m["dim"] ** -0.5, split(h @ W(p + "k").T), split(h @ W(p + "v").T), torch.exp(-softplus(-z) / m["tau"]))
        y = rms(y, W(p + "norm"), eps).reshape(n, -1) * torch.nn.functional.silu(h @ W(p + "g").T)
    elif kind == "mamba2":
        inner, states = heads * m["vdim"], m["groups"] * m["state"]
        z, x, dt = (h @ W(p + "in").T).split([inner, inner + 2 * states, heads], dim=1)
        x, b, c = torch.nn.functional.silu(conv(x, W(p + "conv"), W(p + "conv.b"))).split([inner, states, states], dim=1)
        dt = softplus(dt + W(p + "dt_bias"))
        b, c = (t.reshape(n, m["groups"], -1).repeat_interleave(heads // m["groups"], dim=1) for t in (b, c))
        decay = torch.exp(-W(p + "A_log").exp() * dt)[:, :, None].expand_as(b)
        y = recurrence(c, b * dt[:, :, None], split(x), decay) + W(p + "D")[:, None] * split(x)
        y = rms(y.reshape(n, -1) * torch.nn.functional.silu(z), W(p + "norm"), eps, m["norm_groups"])
    else:
        row, d = h @ W(p + "dkv").T, m["dim"]
        q, latent = split(h @ W(p + "q").T), rms(row[:, :m["kv_rank"]], W(p + "dkv.norm"), eps)
        k_rot = rotate(row[:, None, m["kv_rank"]:], m["rot"]).expand(n, heads, m["rot_dim"])
        q = torch.cat([q[..., :d], rotate(q[..., d:], m["rot"])], dim=-1)
        k = torch.cat([split(latent @ W(p + "uk").T), k_rot], dim=-1)
        y = attend(q, k, split(latent @ W(p + "uv").T), m["scale"], visible(n)).reshape(n, -1) * torch.sigmoid(h @ W(p + "g").T)
    return y @ W(p + "o").T


def gatuzen(ids, W, cfg):
    eps, groups, gain = cfg["norm"]["eps"], cfg["norm"]["groups"], cfg["residual_mult"]
    x = W("embed")[ids] * cfg["embedding"]["scale"]
    norm = lambda v, name: rms(v, W(name), eps, groups)  # noqa: E731

    def read(name, taps):
        h = norm(x, name)
        return h + conv(h, W(taps))
    for i, layer in enumerate(cfg["layers"]):
        p, r = f"l{i}.", layer["mlp"]["router"]
        x = x + gain * norm(gatuzen_mixer(read(p + "norm1", p + "canon1"), W, p + "mix.", layer["mixer"], layer["type"], eps), p + "norm1b")
        h, table = read(p + "norm2", p + "canon2"), W(p + "mlp.table")[ids]
        y = torch.zeros_like(h)
        for e in range(r["experts"]):
            at = (table == e).any(dim=1)
            if at.any():
                y[at] += gated(h[at], W, f"{p}mlp.e{e}.", "silu") / r["top"]
        x = x + gain * norm(y, p + "norm2b")
    return norm(x, "final.norm") * cfg["logit_scale"]


def exact_model(case, seed):
    cfg, rows = model_config(case), []
    shapes = BENCH[case["model"]].weight_shapes(cfg)

    def W(name):
        w = weight(case["model"], cfg, name, shapes[name])
        return w if w.dtype == torch.int32 else w.double()
    forward = {"besudra": besudra, "silevik": silevik, "gatuzen": gatuzen}[case["model"]]
    for ids, n in zip(tokens(case, seed), prompts(case)):
        rows.append((forward(torch.from_numpy(ids).long().cuda(), W, cfg)[n - 1:] @ W("head").T).cpu().numpy())
    return [np.stack([r[j] for r in rows]) for j in range(1 + case["new"])]


# ---- what is measured -----------------------------------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] != "requests":
        return prepare_attention(case, seed)
    return {"kind": "requests", "model": opened(case), "ids": tokens(case, seed), "lens": prompts(case), "new": case["new"]}


def run(state):
    return run_model(state) if state["kind"] == "requests" else run_attention(state)


def work(case):
    return model_work(case) if case["kind"] == "requests" else attention_work(case)


def tolerance(case):
    # attention: f16 caches, queries and softmax weights, 3e-4 off 64 bits; models: bf16 weights and activations through four layers, 1e-2 off
    # (2e-4 where a scaled embedding outweighs what the layers add)
    if case["kind"] != "requests":
        return {"rel": 0.0015, "max": 0.03}
    return {"besudra": {"rel": 0.03, "max": 0.3}, "silevik": {"rel": 0.001, "max": 0.02}, "gatuzen": {"rel": 0.025, "max": 0.25}}[case["model"]]


def exact(case, seed):
    return exact_model(case, seed) if case["kind"] == "requests" else exact_attention(case, seed)
