"""FP16 prefix queries in the FP16 cell: against dense attention in 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("query_block, dim, dtype, cells, prefix, packed", [
    (64, 64, torch.float16, (0.4, 0.4, 0.2), 62, True),       # the strided views of an exchange's buffer
    (64, 128, torch.bfloat16, (0.0, 0.0, 1.0), 1, False),
    (64, 128, torch.bfloat16, (0.0, 0.0, 1.0), 129, False),   # three tiles of 64 rows, the last one alone
    (128, 64, torch.bfloat16, (0.0, 0.5, 0.5), 128, False),
    (128, 128, torch.float16, (0.5, 0.0, 0.5), 300, False),
    (128, 128, torch.bfloat16, (0.0, 0.0, 1.0), 65, True),
])
def test_prefix_rows_are_dense_attention(native_library, query_block, dim, dtype, cells, prefix, packed):
    from anemoi_b200 import executor

    video, heads = (3, 13, 21), 3
    tokens = prefix + 3 * 13 * 21
    gen = torch.Generator(device="cuda").manual_seed(prefix)
    buffer = torch.randn(1, tokens, heads, 3 * dim, generator=gen, device="cuda").to(dtype)
    q, k, v = buffer.split(dim, dim=3)
    if not packed:
        q, k, v = (t.contiguous() for t in (q, k, v))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.7, retained_nvfp4_ratio=cells[0], retained_int8_ratio=cells[1],
              retained_fp16_ratio=cells[2], video_shape=video, layer=0, query_block_size=query_block,
              prefix_kv_precision="fp16", prefix_query_precision="fp16", nvfp4_scales=(0.01, 0.01, 0.002))
    out = executor.sm100_ragged_attention(q, k, v, **kw)
    staged, _ = executor.sm100_ragged_attention(q, k, v, return_parts=True, **kw)
    assert torch.equal(out, staged)
    scores = torch.einsum("bqhd,bkhd->bhqk", q[:, :prefix].double(), k.double()) / dim ** 0.5
    want = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), v.double())
    off = (out[:, :prefix].double() - want).norm() / want.norm()
    # probabilities and results rounded to fp16 (2^-12 each on average over a sum), results of bf16 once more
    assert off < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -10)
    assert executor.last_status() == 0
