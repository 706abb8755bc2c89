"""FP16 prefix queries: dense attention of the caller's tensors, whatever their range and whichever heads are together."""

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


def _prefix_call(q, k, v, prefix, cells, query_block, **extra):
    from anemoi_b200 import executor

    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.8, retained_nvfp4_ratio=cells[0], retained_int8_ratio=cells[1],
              retained_fp16_ratio=cells[2], video_shape=((q.size(1) - prefix) // 64, 8, 8), layer=0,
              query_block_size=query_block, prefix_kv_precision="fp16", prefix_query_precision="fp16",
              nvfp4_scales=(0.01, 0.01, 0.002), **extra)
    return executor.sm100_ragged_attention(q, k, v, **kw)


@pytest.mark.parametrize("query_block, dim, cells", [(64, 64, (0.0, 0.0, 1.0)), (128, 128, (0.0, 0.5, 0.5))])
@pytest.mark.parametrize("factor", [1.0e5, 1.0e-7])
def test_bf16_prefix_rows_keep_the_range_of_bf16(native_library, query_block, dim, cells, factor):
    """Values past fp16's 65,504, and below its smallest 6e-8: prefix rows are finite, and no further off than at 1."""
    prefix, heads, tokens = 70, 2, 70 + 12 * 64
    gen = torch.Generator(device="cuda").manual_seed(dim)
    q, k, v = (torch.randn(1, tokens, heads, dim, generator=gen, device="cuda") for _ in range(3))
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v * factor))
    out = _prefix_call(q, k, v, prefix, cells, query_block)[:, :prefix].double()
    scores = torch.einsum("bqhd,bkhd->bhqk", q[:, :prefix].double(), k.double()) / dim ** 0.5
    want = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), v.double())
    # probabilities and results rounded to bf16 (2^-9 each)
    assert (out - want).norm() / want.norm() < 2 ** -8


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_prefix_rows_of_very_low_scores(native_library, dtype):
    """Every score below -5e6 (in powers of two): all weight on the one key that is nearest, whatever its size."""
    prefix, heads, tokens, dim = 70, 2, 70 + 12 * 64, 64
    gen = torch.Generator(device="cuda").manual_seed(3)
    v = torch.randn(1, tokens, heads, dim, generator=gen, device="cuda").to(dtype)
    q = torch.full_like(v, 896.0)
    k = torch.full_like(v, -896.0)
    k[:, 131] = -832.0    # 896 x 832 x 64 / 8 / ln 2 = 8.6e6
    out = _prefix_call(q, k, v, prefix, (0.0, 0.0, 1.0), 64)
    assert torch.equal(out[:, :prefix], v[:, 131:132].expand(1, prefix, heads, dim))


@pytest.mark.parametrize("query_block, dim, dtype, cells, prefix, blocks, heads", [
    (64, 128, torch.bfloat16, (0.0, 0.0, 1.0), 200, 60, 40),      # few and many prefix rows of the whole call
    (128, 128, torch.bfloat16, (0.4, 0.4, 0.2), 200, 60, 90),
    (64, 64, torch.float16, (0.0, 0.5, 0.5), 70, 60, 150),
])
def test_heads_alone_and_in_host_groups_equal_one_call(native_library, query_block, dim, dtype, cells, prefix, blocks,
                                                       heads):
    from anemoi_b200 import HostAttention, NVFP4Calibration, QuantConfig, SparseConfig, VisualLayout

    tokens = prefix + blocks * 64
    gen = torch.Generator(device="cuda").manual_seed(blocks)
    q, k, v = (torch.randn(1, tokens, heads, dim, generator=gen, device="cuda").to(dtype) for _ in range(3))
    whole = _prefix_call(q, k, v, prefix, cells, query_block)
    for first, last in ((0, 1), (heads // 2, heads // 2 + 2), (heads - 4, heads)):
        part = _prefix_call(*(t[:, :, first:last] for t in (q, k, v)), prefix, cells, query_block)
        assert torch.equal(whole[:, :, first:last], part)
    host = [t.cpu().pin_memory() for t in (q, k, v)]
    out = torch.empty_like(host[0]).pin_memory()
    runner = HostAttention("cuda", group_heads=8)
    runner(*host, out, layout=VisualLayout((blocks, 8, 8), prefix), layer=0, sparse_config=SparseConfig(query_block, 0.8),
           quant_config=QuantConfig(*cells, "fp16", "fp16"), calibration=NVFP4Calibration(0.01, 0.01, 0.002))
    torch.cuda.synchronize()
    assert torch.equal(out, whole.cpu())


@pytest.mark.parametrize("prefix, tokens, library", [(384, 8192, False), (385, 8171, True), (385, 8170, False)])
def test_both_sides_of_the_library_rule(native_library, prefix, tokens, library):
    """Prefixes on both sides of the line from which they are left to torch: the same rows to rounding, in both paths of a
    call, with the heads together or alone."""
    from anemoi_b200 import executor

    heads, dim = 2, 128
    gen = torch.Generator(device="cuda").manual_seed(prefix)
    q, k, v = (torch.randn(1, tokens, heads, dim, generator=gen, device="cuda").bfloat16() for _ in range(3))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.9, retained_nvfp4_ratio=0.0, retained_int8_ratio=0.0,
              retained_fp16_ratio=1.0, video_shape=(1, 1, tokens - prefix), layer=0, query_block_size=128,
              prefix_kv_precision="fp16", prefix_query_precision="fp16")
    assert executor._library_prefix(False, prefix, tokens, dim) == library
    out = executor.sm100_ragged_attention(q, k, v, **kw)
    staged, _ = executor.sm100_ragged_attention(q, k, v, return_parts=True, **kw)
    assert torch.equal(out, staged)
    assert torch.equal(out[:, :, 1:], executor.sm100_ragged_attention(q[:, :, 1:], k[:, :, 1:], v[:, :, 1:], **kw))
    scores = torch.einsum("bqhd,bkhd->bhqk", q[:, :prefix].double(), k.double()) / dim ** 0.5
    want = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), v.double())
    assert (out[:, :prefix].double() - want).norm() / want.norm() < 2 ** -8
