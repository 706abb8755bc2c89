"""Query tiles of several heads that start in turns: every tile of every head runs once, whatever the grid's shape."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks, heads, dim, query_block, groups", [
    (5, 29, 64, 128, 29),     # 145 CTAs: heads one after the other
    (149, 1, 64, 128, 1),     # one head, its first 148 lists shortest first
    (10, 29, 64, 128, 1),     # 290 and 300 CTAs: with and without
    (10, 30, 64, 128, 1),
    (11, 32, 64, 64, 1),      # pairs, the last one a block alone
    (300, 11, 64, 128, 3),    # groups of four heads, the last one a head short
    (600, 11, 64, 64, 3),     # pairs
    (300, 11, 128, 128, 6),   # groups of two, the last one a head short
    (800, 3, 128, 128, 3),    # a head's keys and values as large as all that are kept in use
])
def test_tiles_of_heads_in_turns_equal_the_heads_alone(native_library, blocks, heads, dim, query_block, groups):
    from anemoi_b200 import executor

    gen = torch.Generator(device="cuda").manual_seed(heads)
    q, k, v = (torch.randn(1, blocks * query_block, heads, dim, generator=gen, device="cuda").to(torch.float16)
               for _ in range(3))
    q *= torch.linspace(0.2, 3.0, heads, device="cuda")[None, None, :, None].to(torch.float16)
    kw = dict(prefix_tokens=0, sparsity_ratio=0.8, retained_nvfp4_ratio=0.0, retained_int8_ratio=0.0,
              retained_fp16_ratio=1.0, video_shape=(blocks, 8, query_block // 8), layer=0, query_block_size=query_block,
              prefix_kv_precision="fp16", prefix_query_precision="fp16")
    shape = executor.make_shape(q, prefix_tokens=0, video_blocks=blocks, query_block_size=query_block, active=("fp16",),
                                native_prefix=False, has_maxpool=False)
    assert native_library.anemoi_sm100_head_groups(C.byref(shape), 1) == groups
    alone = [executor.sm100_ragged_attention(*(t[:, :, h:h + 1].contiguous() for t in (q, k, v)), **kw)
             for h in range(heads)]
    # (a row that no CTA writes must not be one that an earlier call has written)
    held = torch.cuda.memory_reserved()
    waste = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(held >> 22)]
    del waste
    together = executor.sm100_ragged_attention(q, k, v, **kw)
    for h in range(heads):
        assert torch.equal(together[:, :, h:h + 1], alone[h]), h
    assert torch.equal(together, executor.sm100_ragged_attention(q, k, v, **kw))
    assert executor.last_status() == 0
