"""The producer kernel takes four heads of a token at a time: head counts around that, and fewer
groups than a CTA holds, bit for bit against the restatement."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens, heads", [(1, 1), (3, 2), (7, 3), (5, 4), (19, 5), (33, 7), (2, 56)])
@pytest.mark.parametrize("d, rotary, dtype", [(64, 32, torch.float16), (128, 64, torch.bfloat16),
                                              (128, 128, torch.float16)])
def test_head_counts(native_library, tokens, heads, d, rotary, dtype):
    from anemoi_b200.producer import fused_qknorm_rope
    from oracle.producer import qknorm_rope

    gen = torch.Generator().manual_seed(tokens + heads)
    x = torch.randn(tokens, heads, d, generator=gen).to(dtype)
    w = (1 + 0.1 * torch.randn(d, generator=gen)).to(dtype)
    cos, sin = torch.randn(2, tokens, rotary, generator=gen)
    got = fused_qknorm_rope(x.cuda().unsqueeze(0), w.cuda(), cos.cuda(), sin.cuda(), 1e-6)
    want = qknorm_rope(x, w, cos.numpy(), sin.numpy(), 1e-6)
    assert torch.equal(got[0].cpu().view(torch.int16), want.view(torch.int16))
