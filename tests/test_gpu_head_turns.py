"""Query tiles of several heads that start in turns: every tile of every head runs once, whatever the grid's shape."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks, heads, dim, query_block", [
    (5, 29, 64, 128),     # 145 CTAs: heads one after the other
    (149, 1, 64, 128),    # one head, its first 148 lists shortest first
    (10, 29, 64, 128),    # 290 and 300 CTAs: with and without
    (10, 30, 64, 128),
    (11, 32, 64, 64),     # pairs, the last one a block alone
    (300, 11, 128, 128),  # groups of five heads: four, four and three
])
def test_tiles_of_heads_in_turns_equal_the_heads_alone(native_library, blocks, heads, dim, query_block):
    from anemoi_b200 import executor

    gen = torch.Generator(device="cuda").manual_seed(heads)
    q, k, v = (torch.randn(1, blocks * query_block, heads, dim, generator=gen, device="cuda").to(torch.float16)
               for _ in range(3))
    q *= torch.linspace(0.2, 3.0, heads, device="cuda")[None, None, :, None].to(torch.float16)
    kw = dict(prefix_tokens=0, sparsity_ratio=0.8, retained_nvfp4_ratio=0.0, retained_int8_ratio=0.0,
              retained_fp16_ratio=1.0, video_shape=(blocks, 8, query_block // 8), layer=0, query_block_size=query_block,
              prefix_kv_precision="fp16", prefix_query_precision="fp16")
    together = executor.sm100_ragged_attention(q, k, v, **kw)
    for h in {0, heads // 2, heads - 1}:
        alone = executor.sm100_ragged_attention(*(t[:, :, h:h + 1].contiguous() for t in (q, k, v)), **kw)
        assert torch.equal(together[:, :, h:h + 1], alone)
    assert torch.equal(together, executor.sm100_ragged_attention(q, k, v, **kw))
    assert executor.last_status() == 0
