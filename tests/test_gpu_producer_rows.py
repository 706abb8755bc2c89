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


def test_more_threads_than_32_bits_count(native_library):
    """2^28 + 64 rows of one head, 16 lanes each: 2^32 + 1,024 threads. The same 64 rows over and over:
    every one of them is normed, and once."""
    from anemoi_b200.producer import fused_qknorm_rope

    tokens, d = (1 << 28) + 64, 128
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < tokens * d * 2 + (8 << 30):
        pytest.skip("needs 72 GiB of free device memory")
    gen = torch.Generator(device="cuda").manual_seed(1)
    rows = torch.randn(64, d, generator=gen, device="cuda").to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(d, generator=gen, device="cuda")).to(torch.bfloat16)
    want = fused_qknorm_rope(rows.clone().view(1, 64, 1, d), w, torch.empty(64, 0, device="cuda"),
                             torch.empty(64, 0, device="cuda"), 1e-6).view(-1)
    x = torch.empty(tokens // 64, 64 * d, dtype=torch.bfloat16, device="cuda")
    try:
        x.copy_(rows.view(1, -1).expand_as(x))
        none = torch.empty(tokens, 0, device="cuda")
        fused_qknorm_rope(x.view(1, tokens, 1, d), w, none, none, 1e-6)
        for part in x.split(1 << 17):
            assert (part == want).all()
    finally:
        del x
        torch.cuda.empty_cache()
