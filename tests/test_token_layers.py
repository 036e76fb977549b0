"""One call for a token of all layers against a step per layer with the same kernels: the scores of blocks that the
append does not touch are taken while it runs (one block, none when the token completes one, several), one and
two kernels for the rows, layers that share their output rows.  The rows are the same sums in the same order, so they
are equal."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from dotcache.kernels import certified_attention as ca
    from dotcache.kernels.tiered_kv_cache import create_tiered_cache_int4v_from_model

KNOBS = dict(v_tolerance=0.05, top_k_fp16_keys=4, ranking_fallback=True, ranking_r=1, tau_cov=0.995, k_min=2, k_max=128)


def _setup(layers, tokens, kv, g, dt):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    past = [tuple(torch.randn(1, kv, tokens, 128, device="cuda", generator=gen).to(dt) for _ in range(2)) for _ in range(layers)]
    make = lambda: list(create_tiered_cache_int4v_from_model(past, list(range(layers)), max_new_tokens=32).values())
    qkv = torch.randn(3, layers, (kv * g + 2 * kv) * 128, device="cuda", generator=gen).to(dt)
    return make, qkv


def _step_rows(cache, row, kv, g):
    q, k, v = row.split([kv * g * 128, kv * 128, kv * 128])
    cache.append_token(k.view(kv, 1, 128), v.view(kv, 1, 128))
    return ca.certified_attention_layer(cache, q.view(kv * g, 128), g, collect_stats=False, **KNOBS)[0].cpu()


@pytest.mark.parametrize("layers,tokens,kv,g,dt", [
    (2, 16, 2, 4, torch.bfloat16), (2, 30, 2, 1, torch.float16), (66, 46, 1, 2, torch.bfloat16),
    (3, 16 * 600 + 13, 2, 8, torch.bfloat16)])
def test_rows_of_a_token(layers, tokens, kv, g, dt):
    make, qkv = _setup(layers, tokens, kv, g, dt)
    one, each = make(), make()
    host, out = qkv.cpu().pin_memory(), torch.empty(layers, kv * g, 128).pin_memory()
    for t in range(3):
        out.fill_(float("nan"))
        ca.certified_decode_token_host(one, host[t], g, out, **KNOBS)
        for l in range(layers):
            assert torch.equal(out[l], _step_rows(each[l], qkv[t, l], kv, g).view(kv * g, 128)), (t, l)


def test_layers_with_common_rows():
    kv, g, layers = 2, 4, 3
    make, qkv = _setup(layers, 200, kv, g, torch.bfloat16)
    one, each = make(), make()
    host, out = qkv.cpu().pin_memory(), torch.empty(layers, kv * g, 128).pin_memory()
    ca.certified_decode_token_host(one, host[0], g, out, **KNOBS)
    spaces = one[0]._decode_token_plan[2]
    common = spaces[0].struct.out

    def with_common_rows(fill):
        def fill_struct(blocks):
            record = fill(blocks)
            record.out = common
            return record
        return fill_struct

    for space in spaces:
        object.__setattr__(space, "fill_struct", with_common_rows(space.fill_struct))
    for l in range(layers):
        _step_rows(each[l], qkv[0, l], kv, g)
    out.fill_(float("nan"))
    ca.certified_decode_token_host(one, host[1], g, out, **KNOBS)
    for l in range(layers):
        assert torch.equal(out[l], _step_rows(each[l], qkv[1, l], kv, g).view(kv * g, 128)), l
