"""Rotary embedding and cache append of a whole prompt against the torch operations that define it, bit for bit."""

import pytest
import torch

from fdk import native
from fdk.llama import ROPE_ROW_ORDER

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,tokens,q_heads,kv_heads,spare", [(1, 1, 1, 1, 0), (1, 37, 24, 8, 5), (3, 130, 4, 2, 1), (2, 1000, 32, 8, 64)])
def test_rope_prefill_equals_torch(batch, tokens, q_heads, kv_heads, spare):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    heads = q_heads + 2 * kv_heads
    qkv = torch.randn((batch * tokens, heads * 128), generator=gen, device="cuda").bfloat16()
    angles = torch.arange(tokens, device="cuda")[:, None] * 10000.0 ** (-torch.arange(0, 128, 2, device="cuda") / 128)[None]
    cos, sin = angles.cos().bfloat16(), angles.sin().bfloat16()
    q = torch.full((batch, tokens, q_heads, 128), float("nan"), device="cuda", dtype=torch.bfloat16)
    caches = [torch.full((batch, kv_heads, tokens + spare, 128), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    native.rope_prefill(qkv, torch.stack((cos, sin), dim=-1), q, *caches)

    unpair = torch.argsort(torch.tensor(ROPE_ROW_ORDER, device="cuda"))
    c, s = (torch.cat((t, t), dim=-1)[None, None] for t in (cos, sin))
    x = qkv.view(batch, tokens, heads, 128).transpose(1, 2)
    qk = x[:, : q_heads + kv_heads][..., unpair]
    want = qk * c + torch.cat((-qk[..., 64:], qk[..., :64]), dim=-1) * s
    assert torch.equal(q.view(torch.int16), want[:, :q_heads].transpose(1, 2).contiguous().view(torch.int16))
    assert torch.equal(caches[0][:, :, :tokens].contiguous().view(torch.int16), want[:, q_heads:].contiguous().view(torch.int16))
    assert torch.equal(caches[1][:, :, :tokens], x[:, q_heads + kv_heads:])
    assert all(bool((cache[:, :, tokens:] == 7.0).all()) for cache in caches)
