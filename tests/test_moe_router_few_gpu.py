"""Routing of few tokens (one CTA per token) gives to the last bit what routing of many gives, and follows the reference."""
import pytest
import torch

from tokenweave_b200 import ops
from tokenweave_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,topk", [(4, 2), (8, 2), (16, 4), (32, 8)])
@pytest.mark.parametrize("H", [8, 264, 2048, 3072])
def test_few_tokens_as_many(E, topk, H):
    many = 8192 // E + 200
    x = torch.randn(many, H, device="cuda").bfloat16()
    g = (torch.randn(E, H, device="cuda") * H ** -0.5).bfloat16()
    w, ids, logits = ops.moe_router(x, g, topk, want_logits=True)
    for T in (1, 7, 8192 // E, 8192 // E + 1):
        for renormalize in (True, False):
            a = ops.moe_router(x[:T], g, topk, renormalize, want_logits=True)
            if renormalize:
                assert torch.equal(a[0], w[:T])
            assert torch.equal(a[1], ids[:T]) and torch.equal(a[2], logits[:T])
            want = ref.moe_router(x[:T].float(), g.float(), topk, renormalize)
            # sums of H fp32 terms of size H^-0.5: off by sqrt(H) 2^-24 at most, here with a wide margin
            assert (a[2] - want[2]).abs().max().item() < 1e-4
            same = (a[1].long() == want[1].long()).all(1)
            assert same.float().mean().item() > 0.99 and (a[0] - want[0])[same].abs().max().item() < 1e-4
