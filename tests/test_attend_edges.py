"""Phase 2 against a float64 evaluation of the same masks on the same cache: every group size and Tier-2 type, a single
block, odd block counts (pairs), one-token trailing blocks, more than 32 pairs per warp, promoted keys and values,
densely recomputed heads.

Tolerance 1e-5 of a row's norm: logits are float32 sums of 128 products with |logit| below 30, so they carry up to
30 * 2^-24 * 2 = 3.6e-6, which the softmax turns into as much of a weight; sums add a few 2^-24."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from dotcache.kernels import certified_attention as ca
    from dotcache.kernels.tiered_kv_cache import create_tiered_cache_from_model, create_tiered_cache_int4v_from_model

DT = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def _reference(c, ws, q, g, scale):
    kv, n, nq, nact = c.kv_heads, c.num_tokens, c.num_quantized_blocks, c.active_blocks
    H = kv * g
    pad = nact * 16
    k2 = torch.zeros(kv, pad, 128, dtype=torch.float64, device="cuda")
    v2 = torch.zeros_like(k2)
    vt = c.values_fp16 if c.values_fp16 is not None else c.values_fp16_gpu
    k2[:, :n], v2[:, :n] = c.keys_fp16_gpu[:, :n].double(), vt[:, :n].double()
    s16 = torch.einsum("kgd,knd->kgn", q.double().view(kv, g, 128), k2).view(H, nact, 16) * scale
    s8 = s16.clone()
    tok = ws.token_scores[: kv * nq * g * 16].view(kv, nq, g, 16).permute(0, 2, 1, 3).reshape(H, nq, 16)
    s8[:, :nq] = tok.double()
    cert, flags = ws.read_cert()
    dense = torch.tensor([bool(d) or bool(flags[2]) for d in cert["dense"]], device="cuda")
    km = ws.topk_mask[:, :nact].bool() | dense[:, None]
    vm = ws.value_mask[:, :nact].bool() | dense[:, None]
    s = torch.where(km[:, :, None], s16, s8).reshape(H, pad)
    s[:, n:] = float("-inf")
    w = torch.softmax(s, -1).view(H, nact, 16)
    v4 = v2.clone()
    if c.values_int4_packed is not None and nq:
        t = nq * 16
        p = c.values_int4_packed[:, :t]
        codes = torch.stack([p & 15, p >> 4], -1).reshape(kv, t, 128).double()
        v4[:, :t] = (codes * c.values_int4_scales[:, :t].double().repeat_interleave(16, -1)
                     + c.values_int4_zeros[:, :t].double().repeat_interleave(16, -1))
    f = vm[:, :, None].double()
    out = (torch.einsum("kgn,knd->kgd", (w * f).reshape(kv, g, pad), v2)
           + torch.einsum("kgn,knd->kgd", (w * (1 - f)).reshape(kv, g, pad), v4)).reshape(H, 128)
    return out, int(dense.sum())


@pytest.mark.parametrize("tokens,kv,g,dtype,splits,over", [
    (16, 2, 4, "bf16", 0, {}),
    (17, 1, 8, "fp16", 0, {}),
    (16 * 7 + 1, 3, 1, "fp32", 0, {}),
    (16 * 33 + 9, 2, 2, "bf16", 3, dict(exploration_rate=0.3)),
    (16 * 47, 2, 4, "fp16", 5, dict(exploration_rate=0.5, v_tolerance=0.0)),
    (16 * 1100 + 3, 1, 4, "bf16", 1, dict(exploration_rate=0.05)),
    (16 * 1100 + 3, 1, 8, "fp16", 1, dict(exploration_rate=0.05, v_tolerance=0.02)),
    (16 * 600 + 15, 2, 8, "bf16", 4, dict(exploration_rate=0.1, ranking_r=4)),
    (16 * 520, 2, 2, "fp32", 1, dict(exploration_rate=0.2, ranking_r=4)),
    (16 * 300 + 5, 2, 4, "fp16", 0, dict(score_consistency_check=True, eps_guard=-100.0)),
    (16 * 300 + 5, 2, 4, "model", 2, dict(exploration_rate=0.2)),
])
def test_attend_matches_float64(tokens, kv, g, dtype, splits, over):
    gen = torch.Generator(device="cuda").manual_seed(tokens + g)
    dt = DT.get(dtype, torch.bfloat16)
    k = torch.randn(1, kv, tokens, 128, device="cuda", generator=gen)
    k[..., 5] *= 8
    v = torch.randn(1, kv, tokens, 128, device="cuda", generator=gen)
    q = torch.randn(kv * g, 128, device="cuda", generator=gen).to(dt)
    make = create_tiered_cache_from_model if dtype == "model" else create_tiered_cache_int4v_from_model
    c = make([(k.to(dt), v.to(dt))], [0], max_new_tokens=16)[0]
    knobs = dict(v_tolerance=0.05, top_k_fp16_keys=4, ranking_fallback=True, tau_cov=0.995, k_min=2, k_max=128,
                 score_consistency_check=False)
    knobs.update(over)
    if splits:
        ca._workspace(c, kv * g, g, q.device).num_splits = splits
    out, _ = ca.certified_attention_layer(c, q, g, None, False, **knobs)
    ref, n_dense = _reference(c, c._certified_workspace["cqa_ws"], q, g, 128 ** -0.5)
    assert n_dense or not ("ranking_r" in over or "eps_guard" in over)
    err = (out.double() - ref).norm(dim=1) / ref.norm(dim=1)
    assert err.max().item() < 1e-5, err
