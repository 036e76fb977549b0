"""The summary of a step against torch reductions of the same masks, rows and certificates: one block, part of a warp's
share of the blocks, more than one round per thread, one head, more heads than a warp has lanes, caches without INT4
values.

Counts are exact, and so are float32 extremes; sums of certificate fields are float64 here and there (1e-12).  The sum of
a row of n mass fractions is float32 in both, at most n * 2^-24 of the sum apart: 7e-5 at 1100 blocks."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from dotcache.kernels import certified_attention as ca
    from dotcache.kernels.tiered_kv_cache import create_tiered_cache_from_model, create_tiered_cache_int4v_from_model


@pytest.mark.parametrize("tokens,kv,g,int4", [(16, 1, 1, True), (16 * 9 + 5, 2, 4, False), (16 * 1100 + 1, 2, 2, True),
                                              (16 * 70, 5, 8, True)])
def test_summary_matches_torch(tokens, kv, g, int4):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    k, v = (torch.randn(1, kv, tokens, 128, device="cuda", generator=gen).bfloat16() for _ in range(2))
    q = torch.randn(kv * g, 128, device="cuda", generator=gen).bfloat16()
    make = create_tiered_cache_int4v_from_model if int4 else create_tiered_cache_from_model
    c = make([(k, v)], [0], max_new_tokens=48)[0]
    H, nq, nact = kv * g, c.num_quantized_blocks, c.active_blocks
    for _ in range(2):       # the ticket of the last CTA is back at zero after a call
        ca.certified_attention_layer(c, q, g, None, True, v_tolerance=0.05, top_k_fp16_keys=4, tau_cov=0.995, k_min=2,
                                     k_max=128, exploration_rate=0.1)
    ws = c._certified_workspace["cqa_ws"]
    got = ws.summary[1].tolist()
    cert, flags = ws.read_cert()
    col = lambda name: torch.tensor([float(x) for x in cert[name]], dtype=torch.float64)  # noqa: E731
    gap = (col("fp16_top1").float() - col("fp16_top2").float()).double()
    e = torch.exp(2 * col("delta"))
    e_key = 2 * e * col("tail_mass") * (e - 1)
    exact = {0: float(flags[2]), 10: col("k_star").min(), 11: col("k_star").max(), 14: col("e_val").max(), 16: col("e_pre").max(),
             19: col("tail_mass").max(), 23: gap.min(),
             26: (ws.topk_mask[:, :nact] == 0).sum(), 31: ws.value_mask[:, :nq].bool().any(0).sum()}
    for i, name in enumerate(("consistency_violation", "boundary_triggered", "rung1_triggered", "value_promoted_blocks", "dense",
                              "exploration_blocks", "ranking_disagree_r1", "ranking_disagree_r3", "k_star")):
        exact[1 + i] = col(name).sum()
    if int4:
        exact[29] = c.values_int4_errors.max()
    exact[30] = c.values_norm_max_per_block[:, :nact].max()
    for i, want in exact.items():
        assert got[i] == float(want), (i, got[i], float(want))
    close = {12: col("delta").sum(), 13: col("e_val").sum(), 15: col("e_pre").sum(), 17: col("tau_actual").sum(),
             18: col("tail_mass").sum(), 20: col("int8_top1").sum(), 21: col("fp16_top1").sum(), 22: gap.sum(),
             24: e_key.sum(), 25: e_key.max()}
    for i, want in close.items():
        assert abs(got[i] - float(want)) <= 1e-12 * max(1.0, abs(float(want)), H), (i, got[i], float(want))
    rho = ws.mass_frac[:, :nq].double().sum(1)
    assert abs(got[27] - float(rho.sum())) < 1e-4 * H and abs(got[28] - float(rho.max())) < 1e-4
