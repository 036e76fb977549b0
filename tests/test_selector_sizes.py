"""The selector at the sizes where its paths change: one block, a warp of blocks, the ordered list's limit and one more,
one and two rounds of a CTA's threads, heavy ties beyond the list; and every CTA width (a batch uses narrower ones) against
single calls.  Bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import golden_cases as gc
from cqa_b200 import synth

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import cuda_harness as hz
    from oracle import cqa_oracle as orc
    from dotcache.kernels import certified_attention as ca


@pytest.mark.parametrize("blocks,repeat,over", [
    (1, 0, {}), (31, 0, {}), (256, 0, {}), (257, 0, {}), (384, 0, {}), (385, 0, {}), (1024, 0, dict(v_tolerance=0.01)),
    (1025, 0, dict(k_max=None)), (2100, 0, dict(v_tolerance=0.0)),
    (400, 400, {}), (900, 3, {}), (1300, 450, dict(ranking_r=6)),
])
def test_selector_matches_oracle(blocks, repeat, over):
    """`repeat`: the first 16 tokens fill that many blocks, whose masses and value errors then tie exactly."""
    dtype, tail = "bfloat16", 5
    base = synth.make_layer_inputs(900 + blocks, blocks * 16 + tail, kv_heads=2, gqa_group=2, dtype=dtype)
    k, v = base.k.copy(), base.v.copy()
    for b in range(1, repeat):
        at = (b * 7) % blocks if repeat < blocks // 2 else b
        k[:, at * 16:(at + 1) * 16], v[:, at * 16:(at + 1) * 16] = k[:, :16], v[:, :16]
    n = blocks * 16
    cc, oc = hz.make_cuda_cache(k[:, :n], v[:, :n], dtype, 64), hz.make_oracle_cache(k[:, :n], v[:, :n], dtype, 64)
    for t in range(n, n + tail):
        cc.append_token(hz.to_dev(k[:, t:t + 1], dtype), hz.to_dev(v[:, t:t + 1], dtype))
        oc.append_token(k[:, t:t + 1], v[:, t:t + 1])
    knobs = dict(gc.PAPER_KNOBS)
    knobs.update(over)
    u = np.random.default_rng(blocks).random((4, blocks), dtype=np.float32)
    R = orc.layer_step(oc, base.q, 2, **dict(knobs, exploration_u=u))
    out, _ = hz.cuda_step(cc, base.q, dtype, 2, knobs, u)
    hz.compare_step(cc, R, out, f"{blocks} blocks")


@pytest.mark.parametrize("count,top", [(40, 700), (24, 1500), (6, 4200)])
def test_batch_widths_match_single_calls(count, top):
    """40 x 700 blocks run with 256 threads per CTA, 24 x 1500 with 256, 6 x 4200 with 512; one sequence with 1024."""
    kv, g = 4, 4
    gen = torch.Generator(device="cuda").manual_seed(count)
    caches, singles = [], []
    for i in range(count):
        n = 16 * max(1, top - (top * i * 3) // (4 * count)) + i % 16
        k = torch.randn(kv, n, 128, device="cuda", generator=gen).bfloat16()
        v = torch.randn(kv, n, 128, device="cuda", generator=gen).bfloat16()
        for to in (caches, singles):
            to.append(ca_cache(k, v))
    q = torch.randn(count, kv * g, 128, device="cuda", generator=gen).bfloat16()
    knobs = dict(v_tolerance=0.05, top_k_fp16_keys=4, ranking_fallback=True, tau_cov=0.995, k_min=2, k_max=128)
    out = ca.certified_attention_batch(caches, q, g, **knobs)
    for i in range(0, count, max(1, count // 6)):
        ref, _ = ca.certified_attention_layer(singles[i], q[i], g, None, False, score_consistency_check=False, **knobs)
        a, b = (c[i]._certified_workspace["cqa_ws"] for c in (caches, singles))
        nact = caches[i].active_blocks
        for name in ("m_b", "s_b", "mass_frac", "topk_mask", "explore_mask", "value_mask"):
            cols = caches[i].num_quantized_blocks if name in ("m_b", "s_b", "mass_frac") else nact
            assert torch.equal(getattr(a, name)[:, :cols], getattr(b, name)[:, :cols]), (i, name)
        ca_, fa = a.read_cert()
        cb_, fb = b.read_cert()
        assert fa[:4] == fb[:4]
        for name in ca_:
            assert np.array_equal(ca_[name], cb_[name]), (i, name)
        # float32 sums in another order (other split counts): 1e-5 of the row
        assert ((out[i] - ref).norm(dim=1) <= 1e-5 * ref.norm(dim=1)).all()


def ca_cache(k, v):
    from dotcache.kernels.tiered_kv_cache import create_tiered_cache_int4v_from_model

    return create_tiered_cache_int4v_from_model([(k[None], v[None])], [0], max_new_tokens=16)[0]
