"""Kernels built for two of the three cells give what the kernel for all of them gives, bit for bit."""

import pytest
import torch

pytestmark = pytest.mark.gpu

FLAGS = ("has_nvfp4", "has_int8", "has_fp16")


@pytest.mark.parametrize("cells", [(0.5, 0.5, 0.0), (0.0, 0.5, 0.5), (0.5, 0.0, 0.5), (1.0, 0.0, 0.0), (0.0, 1.0, 0.0), (0.0, 0.0, 1.0)])
@pytest.mark.parametrize("query_block", [64, 128])
@pytest.mark.parametrize("dim", [64, 128])
def test_same_rows(native_library, dim, query_block, cells):
    from anemoi_b200 import executor, native

    heads, video, prefix = 2, (3, 13, 21), 70   # ragged blocks, an odd number of them
    gen = torch.Generator(device="cuda").manual_seed(dim + query_block)
    q, k, v = (torch.randn(1, prefix + 819, heads, dim, generator=gen, device="cuda").bfloat16() for _ in range(3))
    phase = ("nvfp4", "int8", "fp16")[[c > 0 for c in cells].index(True)]
    _, parts = executor.sm100_ragged_attention(
        q, k, v, prefix_tokens=prefix, sparsity_ratio=0.6, retained_nvfp4_ratio=cells[0], retained_int8_ratio=cells[1],
        retained_fp16_ratio=cells[2], video_shape=video, layer=0, query_block_size=query_block, prefix_kv_precision=phase,
        prefix_query_precision="int8" if cells[1] else "fp16", nvfp4_scales=(0.01, 0.01, 0.002), return_parts=True)
    shape, lists, valid_k, status = (parts[n] for n in ("shape", "lists", "valid_k", "status"))
    assert [getattr(shape, f) for f in FLAGS] == [int(c > 0) for c in cells]
    every = native.Shape(**{name: getattr(shape, name) for name, _ in shape._fields_})
    for flag in FLAGS:
        setattr(every, flag, 1)
    every.q_global_scale, every.k_global_scale, every.v_global_scale = 0.01, 0.01, 0.002
    store = native.allocate_operands(every, q.device)
    native.prepare(every, q, k, v, parts["layout"].indices, parts["layout"].counts, store)
    pairs = native.pair_lists(shape, lists) if query_block == 64 else None
    own = native.attention(shape, parts["store"], lists, valid_k, status, pairs)
    assert torch.equal(own, native.attention(every, store, lists, valid_k, status, pairs))
    if cells[1]:  # prefix tiles walk in the call's kernel
        rows = native.prefix_attention(shape, parts["store"], valid_k, status)
        assert torch.equal(rows, native.prefix_attention(every, store, valid_k, status))
    assert executor.last_status() == 0
