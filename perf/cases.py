"""The attention calls whose speed matters to a user of this framework, as cases that a harness can time.

Every case goes through the public entry points of `flash_attn_legacy` the way a user's program calls
them: `flash_attention` (alone for inference, with its autograd backward for training),
`flash_attn_varlen_func` for packed batches and `flash_attn_with_kvcache` for decode steps and prompt
chunks behind a cache.  Run with the repository's root as the working folder.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs on the GPU, made from the seed
    run(state)           one pass, and everything it computes
    work(case)           bytes and floating-point operations a pass cannot do without
    tolerance(case)      how far two correct implementations may be apart
    exact(case, seed)    the results in 64 bits, by plain torch
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "flash-attention-legacy_b200"))

from flash_attn_legacy import flash_attention, flash_attn_varlen_func, flash_attn_with_kvcache  # noqa: E402

DEVICE = "cuda"


def listed():
    return [
        # One chat session being answered: one new token against a short cache, where launches and host
        # work are what a step costs.
        {"name": "decode_single", "kind": "decode", "batch": 1, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "capacity": 4096, "min_len": 1999, "max_len": 1999, "layout": "bshd", "append": True},
        # A small batch generated through the HuggingFace hook: [B,H,S,d] caches that are exactly as long
        # as the text so far (an odd length), the new token already in them.
        {"name": "decode_hook_b8", "kind": "decode", "batch": 8, "heads": 32, "kv_heads": 4, "head_dim": 64,
         "capacity": 2049, "min_len": 2049, "max_len": 2049, "layout": "bhsd", "append": False},
        # A serving step: 64 sequences of 1024 to 32512 cached tokens, one new token each.
        {"name": "decode_serving_b64", "kind": "decode", "batch": 64, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "capacity": 32768, "min_len": 1024, "max_len": 32512, "layout": "bshd", "append": True},
        # The smallest forward of the reference's benchmark: a short prompt, two entries.
        {"name": "forward_tiny", "kind": "forward", "batch": 2, "heads": 8, "kv_heads": 8, "head_dim": 64,
         "seqlen": 128, "causal": True, "layout": "bhnd"},
        # The reference's standard forward shape.
        {"name": "forward_small", "kind": "forward", "batch": 2, "heads": 8, "kv_heads": 8, "head_dim": 64,
         "seqlen": 1024, "causal": True, "layout": "bhnd"},
        # Prefill of one prompt of no particular length in a transformer block: q, k, v are views of the
        # projections' [B,N,H,d] memory and the result goes back as such.
        {"name": "prefill_ragged", "kind": "forward", "batch": 1, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "seqlen": 2987, "causal": True, "layout": "bnhd"},
        # A prompt chunk behind caches filled to different lengths (chunked prefill of a serving loop).
        {"name": "chunk_prefill", "kind": "chunk", "batch": 4, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "capacity": 8192, "min_len": 512, "max_len": 7000, "new": 1024, "layout": "bshd"},
        # Training step of an encoder: many short sequences of an odd length, no mask.
        {"name": "train_encoder", "kind": "train", "batch": 32, "heads": 16, "kv_heads": 16, "head_dim": 64,
         "seqlen": 577, "causal": False, "layout": "bnhd"},
        # Training step of a decoder layer: grouped-query attention, causal (the headline benchmark).
        {"name": "train_gqa", "kind": "train", "batch": 4, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "seqlen": 4096, "causal": True, "layout": "bhnd"},
        # Training step with the widest heads the framework takes.
        {"name": "train_wide_heads", "kind": "train", "batch": 2, "heads": 16, "kv_heads": 16, "head_dim": 256,
         "seqlen": 2048, "causal": True, "layout": "bhnd"},
        # Training step on packed documents of 64 to 4096 tokens.
        {"name": "train_packed", "kind": "packed", "sequences": 16, "min_len": 64, "max_len": 4096, "len_seed": 3,
         "heads": 16, "kv_heads": 16, "head_dim": 128, "causal": True},
        # Training step on one very long document.
        {"name": "train_long", "kind": "train", "batch": 1, "heads": 32, "kv_heads": 8, "head_dim": 128,
         "seqlen": 131072, "causal": True, "layout": "bhnd"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _heads(rng):
    """(query heads, KV heads): multi-head, grouped-query and multi-query attention."""
    return rng.choice([(8, 8), (16, 16), (32, 32), (32, 8), (32, 8), (32, 4), (16, 2), (40, 8), (8, 1)])


def draw(rng):
    kind = rng.choice(["decode", "decode", "forward", "forward", "chunk", "train", "train", "train", "packed"])
    heads, kv_heads = _heads(rng)
    head_dim = rng.choice([64, 64, 64, 128, 128, 128, 128, 32, 96, 256])
    while True:
        if kind == "decode":
            capacity = _log_int(rng, 300, 33000)
            append = rng.random() < 0.7
            low = rng.randint(min(100, capacity // 2), capacity - 1)
            case = {"kind": kind, "batch": _log_int(rng, 1, 96), "heads": heads, "kv_heads": kv_heads,
                    "head_dim": head_dim, "capacity": capacity, "min_len": low,
                    "max_len": rng.randint(low, capacity - 1), "layout": rng.choice(["bshd", "bhsd"]),
                    "append": append}
            fits = case["batch"] * capacity * kv_heads * head_dim <= 64 * 32768 * 8 * 128
        elif kind == "chunk":
            new = _log_int(rng, 2, 2048)
            cached = _log_int(rng, 128, 16384)
            case = {"kind": kind, "batch": _log_int(rng, 1, 16), "heads": heads, "kv_heads": kv_heads,
                    "head_dim": head_dim, "capacity": new + cached + rng.randint(0, 999),
                    "min_len": rng.randint(0, cached), "max_len": cached, "new": new,
                    "layout": rng.choice(["bshd", "bhsd"])}
            fits = case["batch"] * case["capacity"] * kv_heads * head_dim <= 1 << 30
        elif kind == "packed":
            high = _log_int(rng, 100, 8192)
            case = {"kind": kind, "sequences": _log_int(rng, 2, 64), "min_len": rng.randint(1, high),
                    "max_len": high, "len_seed": rng.randint(0, 999), "heads": heads, "kv_heads": kv_heads,
                    "head_dim": head_dim, "causal": rng.random() < 0.8}
            fits = sum(_packed_lengths(case)) * heads * head_dim <= 1 << 28
        else:
            seqlen = _log_int(rng, 65, 20000)
            case = {"kind": kind, "batch": _log_int(rng, 1, 48), "heads": heads, "kv_heads": kv_heads,
                    "head_dim": head_dim, "seqlen": seqlen, "causal": rng.random() < 0.7,
                    "layout": rng.choice(["bhnd", "bnhd"])}
            fits = case["batch"] * seqlen * heads * head_dim <= 1 << 28
        if fits and work(case)["flops"] <= 2e14:
            return case


def _cache_lengths(case):
    """Cached positions per entry, spread evenly over the case's range (prepare() shuffles them)."""
    n, lo, hi = case["batch"], case["min_len"], case["max_len"]
    return [lo + (hi - lo) * i // max(n - 1, 1) for i in range(n)]


def _packed_lengths(case):
    rng = random.Random(case["len_seed"])
    return [rng.randint(case["min_len"], case["max_len"]) for _ in range(case["sequences"])]


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEVICE, dtype=torch.float16)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    order = random.Random(seed)
    kind, h, hk, d = case["kind"], case["heads"], case["kv_heads"], case["head_dim"]
    s = dict(case)
    if kind in ("forward", "train"):
        b, n = case["batch"], case["seqlen"]

        def tensor(heads):
            if case["layout"] == "bnhd":
                return _randn(gen, b, n, heads, d).transpose(1, 2)
            return _randn(gen, b, heads, n, d)

        s["q"], s["k"], s["v"] = tensor(h), tensor(hk), tensor(hk)
        if kind == "train":
            s["d_out"] = tensor(h)
            for name in ("q", "k", "v"):
                s[name].requires_grad_(True)
    elif kind == "packed":
        lens = _packed_lengths(case)
        order.shuffle(lens)
        total = sum(lens)
        s["q"], s["k"], s["v"] = _randn(gen, total, h, d), _randn(gen, total, hk, d), _randn(gen, total, hk, d)
        s["d_out"] = _randn(gen, total, h, d)
        for name in ("q", "k", "v"):
            s[name].requires_grad_(True)
        cu = [0]
        for x in lens:
            cu.append(cu[-1] + x)
        s["cu"] = torch.tensor(cu, dtype=torch.int32, device=DEVICE)
        s["longest"] = max(lens)
    else:
        b, cap = case["batch"], case["capacity"]
        new = case.get("new", 1)
        shape = (b, cap, hk, d) if case["layout"] == "bshd" else (b, hk, cap, d)
        s["k_cache"], s["v_cache"] = _randn(gen, *shape), _randn(gen, *shape)
        s["q"] = _randn(gen, b, new, h, d)
        if kind == "chunk" or case["append"]:
            s["k"], s["v"] = _randn(gen, b, new, hk, d), _randn(gen, b, new, hk, d)
        lens = _cache_lengths(case)
        order.shuffle(lens)
        s["lens"] = torch.tensor(lens, dtype=torch.int32, device=DEVICE)
    return s


def run(s):
    kind = s["kind"]
    if kind == "forward":
        with torch.no_grad():
            return flash_attention(s["q"], s["k"], s["v"], is_causal=s["causal"], out_layout=s["layout"])
    if kind == "train":
        out = flash_attention(s["q"], s["k"], s["v"], is_causal=s["causal"], out_layout=s["layout"])
        return (out.detach(), *torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["d_out"]))
    if kind == "packed":
        out = flash_attn_varlen_func(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["longest"], s["longest"],
                                     causal=s["causal"])
        return (out.detach(), *torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["d_out"]))
    # A pass writes the same new rows at the same positions each time: the cache a pass leaves behind is
    # the one it would leave the first time.
    out = flash_attn_with_kvcache(s["q"], s["k_cache"], s["v_cache"], k=s.get("k"), v=s.get("v"),
                                  cache_seqlens=s["lens"], cache_layout=s["layout"])
    return (out, s["k_cache"], s["v_cache"]) if "k" in s else out


def work(case):
    """Each input read once, each output written once (2 bytes a value); matrix products over the visible
    (query, key) pairs: 2 in a forward, 5 more in a backward, 2 * head_dim operations a pair each."""
    kind, h, hk, d = case["kind"], case["heads"], case["kv_heads"], case["head_dim"]
    if kind in ("forward", "train", "packed"):
        lens = _packed_lengths(case) if kind == "packed" else [case["seqlen"]] * case["batch"]
        pairs = h * sum(n * (n + 1) // 2 if case["causal"] else n * n for n in lens)
        q_values, kv_values = sum(lens) * h * d, sum(lens) * hk * d
        if kind == "forward":
            return {"bytes": 2 * (2 * q_values + 2 * kv_values), "flops": 4 * d * pairs}
        return {"bytes": 2 * (4 * q_values + 4 * kv_values), "flops": 14 * d * pairs}
    b, new = case["batch"], case.get("new", 1)
    lens = _cache_lengths(case)
    appended = new if kind == "chunk" or case["append"] else 0
    keys = sum(lens) + b * appended
    values = 2 * b * new * h * d + 2 * keys * hk * d + 2 * b * appended * hk * d
    pairs = h * sum(new * n + new * (new + 1) // 2 if appended else new * n for n in lens)
    return {"bytes": 2 * values, "flops": 4 * d * pairs}


def tolerance(case):
    """fp16 results, with the probabilities and the score gradients rounded to fp16 before the products
    that consume them.  About four times the distance from the same arithmetic in 64 bits: outputs 2.4e-4
    to 2.9e-4 (2-norm) and up to 3.6e-3 (largest), gradients 2.8e-4 to 4.3e-4 and up to 1.5e-2."""
    if case["kind"] in ("train", "packed"):
        return {"rel": 1.7e-3, "max": 6e-2}
    return {"rel": 1.2e-3, "max": 1.5e-2}


def _attention64(q, k, v, scale, causal, d_out=None):
    """softmax(q k^T * scale) v of one sequence in 64 bits, q [H,n,d], k and v [H_kv,m,d], the causal mask
    aligned to the end of the keys; with d_out also the gradients.  One head at a time, in blocks of rows."""
    group = q.shape[0] // k.shape[0]
    n, m = q.shape[1], k.shape[1]
    out = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    grads = None if d_out is None else [torch.zeros(x.shape, dtype=torch.float64, device=q.device) for x in (q, k, v)]
    rows = max(1, (1 << 27) // m)
    columns = torch.arange(m, device=q.device)
    for h in range(q.shape[0]):
        kh, vh = k[h // group].double(), v[h // group].double()
        for i in range(0, n, rows):
            qh = q[h, i:i + rows].double()
            p = qh @ kh.T * scale
            if causal:
                last = torch.arange(i, i + qh.shape[0], device=q.device) + (m - n)
                p.masked_fill_(columns[None, :] > last[:, None], -math.inf)
            p = torch.softmax(p, dim=-1)
            out[h, i:i + rows] = p @ vh
            if d_out is not None:
                g = d_out[h, i:i + rows].double()
                ds = p * (g @ vh.T - (g * out[h, i:i + rows]).sum(-1, keepdim=True)) * scale
                grads[0][h, i:i + rows] = ds @ kh
                grads[1][h // group] += ds.T @ qh
                grads[2][h // group] += p.T @ g
    return out, grads


def exact(case, seed):
    """What run() returns for the inputs of this seed, in 64 bits; None where that takes too long, and in
    the place of the caches, whose rows are copied and not computed."""
    if work(case)["flops"] > 1e13 or work(case)["bytes"] > 2e10:
        return None
    s = prepare(case, seed)
    kind, d = case["kind"], case["head_dim"]
    scale = 1.0 / math.sqrt(d)
    with torch.no_grad():
        if kind in ("forward", "train"):
            parts = [_attention64(s["q"][b], s["k"][b], s["v"][b], scale, case["causal"],
                                  s["d_out"][b] if kind == "train" else None) for b in range(case["batch"])]
            out = torch.stack([o for o, _ in parts])
            return out if kind == "forward" else (out, *(torch.stack([g[i] for _, g in parts]) for i in range(3)))
        if kind == "packed":
            cu = s["cu"].tolist()
            parts = []
            for a, b in zip(cu, cu[1:]):
                o, grads = _attention64(*(s[name][a:b].transpose(0, 1) for name in ("q", "k", "v")), scale,
                                        case["causal"], s["d_out"][a:b].transpose(0, 1))
                parts.append([x.transpose(0, 1) for x in (o, *grads)])
            return tuple(torch.cat([part[i] for part in parts]) for i in range(4))
        axis = 0 if case["layout"] == "bshd" else 1
        outs = []
        for b, filled in enumerate(s["lens"].tolist()):
            kv = []
            for name in ("k", "v"):
                old = s[name + "_cache"][b].narrow(axis, 0, filled)
                old = old.transpose(0, 1) if axis == 0 else old
                kv.append(torch.cat([old, s[name][b].transpose(0, 1)], dim=1) if name in s else old)
            o, _ = _attention64(s["q"][b].transpose(0, 1), *kv, scale, kind == "chunk")
            outs.append(o.transpose(0, 1))
        out = torch.stack(outs)
        return (out, None, None) if "k" in s else out
