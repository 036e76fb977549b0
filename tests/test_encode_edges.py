"""Block encoder of the prefill at the places where it can go wrong, bit for bit against the CPU oracle: blocks per warp
and per CTA (1, 4, 5, a ragged tail), quotients on and beside half-integers, constant rows, scales beyond the range of
an approximate reciprocal, a source off the 16-byte boundary, and the reserve behind the prompt."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import cuda_harness as hz
    from cqa_b200 import synth
    from dotcache.kernels.tiered_kv_cache import create_tiered_cache_int4v_from_model


def _rows(kind, n, dtype, seed):
    rng = np.random.default_rng(seed)
    k, v = (rng.standard_normal((3, n, 128), dtype=np.float32) for _ in range(2))
    if kind == "grid":          # few-bit values: exact half-integer quotients everywhere
        k, v = np.round(k * 8) / 8, np.round(v * 8) / 8
    elif kind == "constant":    # the 1e-8 floor of the range; signed zeros
        k[:, ::2] = 0.375
        k[1] = -2.5
        v[:] = 0.25
        v[2, : n // 2] = 0.0
    elif kind == "huge":
        k *= np.float32(3e33)
        v *= np.float32(3e3)
    return synth.round_to_dtype(k, dtype), synth.round_to_dtype(v, dtype)


@pytest.mark.parametrize("kind,tokens,dtype", [
    ("normal", 16, "bfloat16"), ("normal", 16 * 4, "float16"), ("normal", 16 * 5 + 15, "float32"),
    ("grid", 16 * 9 + 1, "bfloat16"), ("grid", 16 * 9, "float16"), ("grid", 16 * 3, "float32"),
    ("constant", 16 * 6 + 7, "bfloat16"), ("huge", 16 * 5, "bfloat16"), ("normal", 16 * 700 + 3, "bfloat16"), ("normal", 7, "float16"),
])
def test_encode_matches_oracle(kind, tokens, dtype):
    k, v = _rows(kind, tokens, dtype, tokens)
    al = tokens // 16 * 16
    past = [(hz.to_dev(k, dtype)[None], hz.to_dev(v, dtype)[None])]
    torch.empty(1 << 26, dtype=torch.uint8, device="cuda").fill_(0xA5)     # stale bytes in the allocator's next blocks
    cc = create_tiered_cache_int4v_from_model(past, [0], max_new_tokens=40)[0]
    oc = hz.make_oracle_cache(k[:, :al], v[:, :al], dtype, 40 + tokens - al, defer=cc._defer_int4_flag())
    for t in range(al, tokens):
        oc.append_token(k[:, t:t + 1], v[:, t:t + 1])
    hz.compare_caches(cc, oc, f"{kind} {tokens}")
    top, blk = (tokens + 15) // 16 * 16, (tokens + 15) // 16
    for name in ("keys_int8", "values_int4_packed", "values_int4_scales", "values_int4_zeros", "keys_fp16_gpu", "values_fp16_gpu"):
        assert not getattr(cc, name)[:, top:].any(), name
    for name in ("keys_scale", "keys_zero_points", "values_int4_errors", "values_int4_error_sums", "values_int4_error_counts",
                 "values_norm_max_per_block"):
        assert not getattr(cc, name)[:, blk:].any(), name
    assert (cc.correction[:, blk:] == 1).all()


def test_encode_from_an_unaligned_source():
    k, v = _rows("normal", 69, "bfloat16", 5)
    flat = torch.zeros(2, k.size + 1, dtype=torch.bfloat16, device="cuda")
    flat[:, 1:] = torch.stack((hz.to_dev(k, "bfloat16").flatten(), hz.to_dev(v, "bfloat16").flatten()))
    off = [t[1:].view(1, 3, 69, 128) for t in flat]      # two bytes past a 16-byte boundary
    assert off[0].data_ptr() % 16 == 2
    cc = create_tiered_cache_int4v_from_model([tuple(off)], [0], max_new_tokens=16)[0]
    oc = hz.make_oracle_cache(k[:, :64], v[:, :64], "bfloat16", 16, defer=True)
    for t in range(64, 69):
        oc.append_token(k[:, t:t + 1], v[:, t:t + 1])
    hz.compare_caches(cc, oc, "unaligned")
