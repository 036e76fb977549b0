"""Timed cases of the certified decode path: what a serving program has it do.

    step     one layer's decode step of one sequence: `append_token`, then `certified_attention_layer`
             (what the adapter calls per layer and token)
    stats    the same with `collect_stats=True`: the certificate is read back every step (quality runs)
    batch    one layer's step of several sequences through `certified_attention_batch` (append included)
    token    one token of a model whose activations are in host memory, all layers through
             `certified_decode_token_host`
    prefill  the caches of several layers built from a prefill's keys and values by
             `create_tiered_cache_int4v_from_model`

Keys and values are N(0,1) with four outlier key channels per KV head (scaled by 8).  "planted" blocks of keys are similar
to the query, which concentrates the attention as retrieval prompts do; without them it is diffuse, as in a random-init
model.  Each pass of a decode case decodes the next of 64 seeded tokens; after the last one the sequence goes back to the
last complete block of its prompt and decodes them again.
"""
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("certified-quantised-attention_b200"))  # run from the root of a checkout

from dotcache.kernels import certified_attention as ca  # noqa: E402
from dotcache.kernels import tiered_kv_cache as tc  # noqa: E402

BLOCK, D, TOKENS = 16, 128, 64
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def _case(kind, tokens, **more):
    c = dict(kind=kind, tokens=tokens, count=1, kv_heads=8, group=4, dtype="bf16", planted=0, v_tolerance=0.05,
             explore="none", consistency=False, values="int4", scratch_blocks=0, ragged=False)
    c.update(more)
    return c


def listed():
    return [
        # the first tokens after a short prompt, a tensor-parallel share of the heads: launches and host work
        dict(_case("step", 600, kv_heads=4, group=2, dtype="fp16", planted=4), name="step_600_fp16_g2"),
        # 8K in float32 with the entry point's default checks (score consistency on)
        dict(_case("step", 8192, dtype="fp32", consistency=True), name="step_8k_fp32"),
        # 32K retrieval-shaped prompt at the paper's knobs, exploration drawn from the caller's generator
        dict(_case("step", 32773, planted=64, explore="generator"), name="step_32k"),
        # 128K at the paper's knobs, exploration drawn in the kernel: the long-context headline
        dict(_case("step", 131072, planted=64, explore="kernel"), name="step_128k"),
        # long, diffuse, the tighter value tolerance, eight query heads per KV head, an odd length
        dict(_case("step", 100003, group=8, v_tolerance=0.02), name="step_100k_diffuse_g8"),
        # FP16 originals held in host memory behind a scratch of 2048 blocks
        dict(_case("step", 32768, planted=64, explore="kernel", scratch_blocks=2048), name="step_32k_scratch"),
        # certificate and telemetry of every step on the host
        dict(_case("stats", 8192, planted=64, explore="generator"), name="stats_8k"),
        # four long sequences of a decoder, diffuse
        dict(_case("batch", 65536, count=4), name="batch_4x64k"),
        # many short requests of different lengths
        dict(_case("batch", 8192, count=32, planted=16, ragged=True), name="batch_32x8k"),
        # one token through eight layers, activations in pinned host memory
        dict(_case("token", 32768, count=8, planted=64, explore="kernel"), name="token_8x32k"),
        # a short prompt with a ragged end
        dict(_case("prefill", 5003, count=2, dtype="fp16"), name="prefill_2x5k_fp16"),
        # a long prompt
        dict(_case("prefill", 65536, count=4), name="prefill_4x64k"),
    ]


def _size(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "stats", "batch", "batch", "token", "prefill", "prefill"))
    kv, g = rng.choice(((8, 4), (8, 4), (8, 4), (8, 8), (8, 2), (8, 1), (4, 4), (4, 2), (2, 4)))
    planted = rng.choice((0, 8, 64))
    more = dict(kv_heads=kv, group=g, dtype=rng.choice(("bf16", "bf16", "fp16", "fp32")), planted=planted,
                v_tolerance=rng.choice((0.05, 0.02)))
    if kind == "prefill":
        count = rng.choice((1, 2, 4))
        more["dtype"] = rng.choice(("bf16", "bf16", "fp16"))
        return _case(kind, _size(rng, 200, 65536), count=count, **dict(more, planted=0))
    if kind == "batch":
        count = _size(rng, 2, 48)
        return _case(kind, _size(rng, 512, 262144 // max(count, 4)), count=count, ragged=rng.random() < 0.5,
                     **dict(more, dtype=rng.choice(("bf16", "fp16"))))
    if kind == "token":
        count = _size(rng, 2, 16)
        return _case(kind, _size(rng, 512, 65536 // count), count=count,
                     **dict(more, dtype=rng.choice(("bf16", "fp16")), explore=rng.choice(("none", "kernel"))))
    more["explore"] = rng.choice(("none", "kernel", "generator"))
    more["consistency"] = rng.random() < 0.3
    more["values"] = "model" if rng.random() < 0.15 else "int4"
    if more["values"] == "int4" and rng.random() < 0.1:
        tokens = _size(rng, 8192, 32768)
        return _case(kind, tokens, scratch_blocks=max(64, tokens // BLOCK), **more)
    top = 131072 if kind == "step" and more["dtype"] != "fp32" else 32768
    return _case(kind, _size(rng, 300, top), **more)


def _lengths(case):
    n, count = case["tokens"], case["count"]
    if not case["ragged"]:
        return [n] * count
    return [max(64, n - (n * 37 * i // (53 * count)) - 5 * i) for i in range(count)]


def _knobs(case):
    return dict(v_tolerance=case["v_tolerance"], top_k_fp16_keys=4, ranking_fallback=True, ranking_r=1, tau_cov=0.995,
                k_min=2, k_max=128, score_consistency_check=case["consistency"],
                exploration_rate=0.0 if case["explore"] == "none" else 0.02)


def _prompt(case, n, gen):
    """(q, k, v, outlier channels): one query per decoded token, and a prompt of n tokens."""
    kv, g, dt = case["kv_heads"], case["group"], DTYPES[case["dtype"]]
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    outlier = torch.rand(kv, D, device="cuda", generator=gen).argsort(dim=1)[:, :4]
    k, v = randn(kv, n, D), randn(kv, n, D)
    k.scatter_(2, outlier[:, None, :].expand(kv, n, 4), 8.0 * randn(kv, n, 4))
    q0 = randn(kv * g, D)
    nb = n // BLOCK
    m = min(case["planted"], nb // 2)
    if m:
        # cosine 0.9 to one query head of the group, norms kept
        at = torch.rand(nb, device="cuda", generator=gen).argsort()[:m]
        head = torch.randint(0, g, (kv, m), device="cuda", generator=gen) + torch.arange(kv, device="cuda")[:, None] * g
        qh = torch.nn.functional.normalize(q0[head], dim=-1)[:, :, None, :]
        blk = k[:, : nb * BLOCK].view(kv, nb, BLOCK, D)[:, at]
        perp = torch.nn.functional.normalize(blk - (blk * qh).sum(-1, keepdim=True) * qh, dim=-1)
        k[:, : nb * BLOCK].view(kv, nb, BLOCK, D)[:, at] = blk.norm(dim=-1, keepdim=True) * (0.9 * qh + 0.19 ** 0.5 * perp)
    q = q0 + 0.1 * randn(TOKENS, kv * g, D)
    q = (q * (q0.norm(dim=-1, keepdim=True) / q.norm(dim=-1, keepdim=True))).to(dt)
    return q, k.to(dt), v.to(dt), outlier


def _new_tokens(case, outlier, gen):
    kv, dt = case["kv_heads"], DTYPES[case["dtype"]]
    k = torch.randn(TOKENS, kv, D, device="cuda", generator=gen)
    v = torch.randn(TOKENS, kv, D, device="cuda", generator=gen)
    k.scatter_(2, outlier.expand(TOKENS, kv, 4), 8.0 * torch.randn(TOKENS, kv, 4, device="cuda", generator=gen))
    return k.to(dt), v.to(dt)


def _cache(case, k, v):
    past = [(k[None], v[None])]
    if case["values"] == "model":
        return tc.create_tiered_cache_from_model(past, [0])[0]
    cap = case["scratch_blocks"] or None
    return tc.create_tiered_cache_int4v_from_model(past, [0], fp16_key_cache_capacity=cap, fp16_value_cache_capacity=cap)[0]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "prefill":
        past = []
        for _ in range(case["count"]):
            _, k, v, _ = _prompt(case, case["tokens"], gen)
            past.append((k[None], v[None]))
        return {"case": case, "past": past}
    caches, q, nk, nv = [], [], [], []
    for n in _lengths(case):
        qs, k, v, outlier = _prompt(case, n, gen)
        caches.append(_cache(case, k, v))
        del k, v
        a, b = _new_tokens(case, outlier, gen)
        q.append(qs), nk.append(a), nv.append(b)
    s = {"case": case, "caches": caches, "knobs": _knobs(case), "i": 0, "start": [c.num_tokens // BLOCK * BLOCK for c in caches]}
    if case["kind"] == "batch":
        s.update(q=torch.stack(q, 1), k=torch.stack(nk, 1), v=torch.stack(nv, 1))  # [TOKENS, B, heads, 128]
    elif case["kind"] == "token":
        rows = [torch.cat((a.flatten(1), b.flatten(1), c.flatten(1)), 1) for a, b, c in zip(q, nk, nv)]
        s["qkv"] = torch.stack(rows, 1).cpu().pin_memory()  # [TOKENS, layers, (heads + 2 KV heads) * 128]
        s["out"] = torch.empty(len(caches), case["kv_heads"] * case["group"], D).pin_memory()
    else:
        s.update(q=q[0], k=nk[0][:, :, None, :], v=nv[0][:, :, None, :])
        if case["explore"] == "generator":
            s["knobs"]["exploration_generator"] = torch.Generator(device="cuda").manual_seed(seed + 1)
    return s


def _next(s):
    """Index of the token to decode; back to the prompt's last complete block after the last one."""
    i = s["i"]
    if i == TOKENS:
        i = 0
        for c, n in zip(s["caches"], s["start"]):
            c.num_tokens, c.num_blocks, c.num_quantized_blocks = n, n // BLOCK, n // BLOCK
    s["i"] = i + 1
    return i


def _cache_tensors(c):
    return [t for t in (c.keys_int8, c.keys_scale, c.keys_zero_points, c.correction, c.values_int4_packed,
                        c.values_int4_scales, c.values_int4_zeros, c.values_int4_errors, c.values_norm_max_per_block,
                        c.keys_scale_max, c.keys_fp16_gpu, c.values_fp16_gpu, c.values_fp16) if t is not None]


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "prefill":
        made = tc.create_tiered_cache_int4v_from_model(s["past"], list(range(case["count"])))
        return [_cache_tensors(c) for c in made.values()]
    i = _next(s)
    if kind == "batch":
        out = ca.certified_attention_batch(s["caches"], s["q"][i], case["group"], new_keys=s["k"][i], new_values=s["v"][i],
                                           **s["knobs"])
        return [out, [c.keys_fp16_gpu for c in s["caches"]]]
    if kind == "token":
        out = ca.certified_decode_token_host(s["caches"], s["qkv"][i], case["group"], s["out"], **s["knobs"])
        return [out, [c.keys_fp16_gpu for c in s["caches"]]]
    cache = s["caches"][0]
    cache.append_token(s["k"][i], s["v"][i])
    out, stats = ca.certified_attention_layer(cache, s["q"][i], case["group"], collect_stats=kind == "stats", **s["knobs"])
    if kind == "stats":
        return [out, {k: v for k, v in stats.items() if not isinstance(v, str)}]
    if case["scratch_blocks"]:
        return out
    return [out, _cache_tensors(cache)]


def work(case):
    kv, g, count, n = case["kv_heads"], case["group"], case["count"], sum(_lengths(case))
    size = 4 if case["dtype"] == "fp32" else 2
    keys, int4 = 128 + 64, 64 + 32      # bytes per token and KV head: INT8 keys and scales, INT4 values and scales
    if case["kind"] == "prefill":
        # both originals in, INT8 keys, INT4 values and the Tier-2 copies out
        return {"bytes": n * kv * (2 * D * size + keys + int4 + 2 * D * size), "flops": 0}
    values = int4 if case["values"] == "int4" else D * size
    rows = count * (2 * kv * g + 4 * kv) * D * size  # q, output, new key and value in, their Tier-2 rows out
    return {"bytes": n * kv * (keys + values) + rows, "flops": 4 * n * kv * g * D}


def tolerance(case):
    # the caches are integer codes and elementwise float32 arithmetic in a fixed order; attention rows are float32 sums
    return "exact" if case["kind"] == "prefill" else {"rel": 1e-5}
