"""Which FP16 prefix rows are the library's own and which torch's, and how many CTAs share the own ones' keys."""

import pytest
import torch


@pytest.mark.parametrize("prefix, tokens, dim, library", [
    (384, 9_984, 128, True), (384, 17_664, 128, True),         # calls in which the own kernel costs up to 5 %
    (512, 9_872, 64, True), (1_000, 4_960, 64, True), (700, 6_912, 64, True),
    (257, 12_241, 64, True), (257, 12_240, 64, False),         # the line
    (257, 12_241, 128, True), (257, 12_240, 128, False),
    (256, 85_000, 64, False), (256, 85_000, 128, False),       # never up to two tiles
    (512, 3_072, 128, False), (1_000, 2_080, 64, False),
])
def test_line(prefix, tokens, dim, library):
    from anemoi_b200 import executor

    assert executor._library_prefix(False, prefix, tokens, dim) == library
    assert not executor._library_prefix(True, prefix, tokens, dim)


@pytest.mark.parametrize("tokens, rows, parts", [
    (31 * 64, 1, 1), (31 * 64 + 1, 1, 2), (95 * 64, 128, 2), (95 * 64 + 1, 128, 4), (255 * 64, 128, 4), (255 * 64 + 1, 128, 8),
    (31 * 64, 384, 1), (31 * 64 + 1, 129, 2), (255 * 64, 384, 2), (255 * 64 + 1, 129, 4), (85_000, 384, 4),
    (2_080, 1_000, 1), (2_592, 392, 1), (95 * 64, 385, 1), (95 * 64 + 1, 385, 2), (85_000, 1_000, 2),   # many heads: see the rule
    (10, 0, -1), (10, 11, -1),
])
def test_parts(native_library, tokens, rows, parts):
    assert native_library.anemoi_sm100_dense_parts(tokens, rows) == parts


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dim, prefix, tokens, heads", [(64, 1_000, 4_960, 24), (64, 257, 12_250, 9), (128, 300, 10_700, 40),
                                                        (128, 512, 16_112, 40)])
def test_rows_left_to_torch_do_not_depend_on_other_heads(native_library, dtype, dim, prefix, tokens, heads):
    """Dense attention to rounding, and the same bits for one head, eight and all of them."""
    from anemoi_b200 import executor

    assert executor._library_prefix(False, prefix, tokens, dim)
    gen = torch.Generator(device="cuda").manual_seed(prefix)
    q, k, v = (torch.randn(1, tokens, heads, dim, generator=gen, device="cuda").to(dtype) for _ in range(3))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.9, retained_nvfp4_ratio=0.0, retained_int8_ratio=0.0,
              retained_fp16_ratio=1.0, video_shape=(1, 1, tokens - prefix), layer=0, query_block_size=128,
              prefix_kv_precision="fp16", prefix_query_precision="fp16")
    out = executor.sm100_ragged_attention(q, k, v, **kw)
    for first, last in ((0, 1), (heads - 8, heads)):
        part = executor.sm100_ragged_attention(*(t[:, :, first:last] for t in (q, k, v)), **kw)
        assert torch.equal(part, out[:, :, first:last])
    scores = torch.einsum("qd,kd->qk", q[0, :prefix, 0].double(), k[0, :, 0].double()) / dim ** 0.5
    want = scores.softmax(-1) @ v[0, :, 0].double()
    # probabilities and results rounded once each (bf16: 2^-9, fp16: 2^-12 at most)
    assert (out[0, :prefix, 0].double() - want).norm() / want.norm() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
    assert executor.last_status() == 0
