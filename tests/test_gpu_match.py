"""Q64 pairs chosen by what the blocks' lists share: bit for bit one block per CTA."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _options(blocks, prefix, cells, drop):
    return dict(prefix_tokens=prefix, sparsity_ratio=drop, retained_nvfp4_ratio=cells[0], retained_int8_ratio=cells[1],
                retained_fp16_ratio=cells[2], video_shape=(blocks, 8, 8), query_block_size=64,
                prefix_kv_precision="fp16" if cells[2] else "int8" if cells[1] else "nvfp4",
                prefix_query_precision="int8" if cells[1] else "fp16")


def _chosen(native_library, q, kw):
    """Whether a call of this shape has its pairs chosen."""
    from anemoi_b200 import executor

    plan = executor._Plan(q.device, q.size(1), q.size(2), q.size(3), q.dtype, kw["prefix_tokens"], kw["sparsity_ratio"],
                          kw["retained_nvfp4_ratio"], kw["retained_int8_ratio"], kw["retained_fp16_ratio"],
                          kw["video_shape"], 64, kw["prefix_kv_precision"], kw["prefix_query_precision"], 0.0, True)
    return native_library.anemoi_sm100_matches_pairs(C.byref(plan.struct))


@pytest.mark.parametrize("blocks, heads, dim, prefix, cells, drop", [
    (33, 400, 64, 0, (0.0, 1.0, 0.0), 0.8),      # a word and a bit per row; a block alone at the end
    (64, 128, 64, 70, (0.4, 0.4, 0.2), 0.7),     # three phases
    (127, 60, 64, 37, (0.0, 1.0, 0.0), 0.9),     # one less than a group and a piece of columns, a group, one more
    (128, 20, 128, 0, (1.0, 0.0, 0.0), 0.7),
    (129, 160, 64, 0, (0.5, 0.0, 0.5), 0.9),
    (129, 150, 64, 0, (0.0, 1.0, 0.0), 0.96),    # blocks with empty lists
    (255, 7, 128, 300, (0.0, 0.0, 1.0), 0.8),
    (256, 4, 64, 0, (0.4, 0.4, 0.2), 0.0),       # every list whole: ties everywhere
    (257, 8, 64, 64, (0.0, 1.0, 0.0), 0.8),      # three groups
    (1025, 1, 64, 0, (0.0, 1.0, 0.0), 0.9),      # more than 32 words per row, routing in several kernels
    (2049, 1, 64, 20, (0.0, 1.0, 0.0), 0.97),
])
def test_chosen_pairs_equal_one_block_per_cta(native_library, blocks, heads, dim, prefix, cells, drop):
    from anemoi_b200 import executor

    gen = torch.Generator(device="cuda").manual_seed(blocks)
    shape = (1, prefix + blocks * 64, heads, dim)
    q, k, v = (torch.randn(shape, generator=gen, device="cuda") for _ in range(3))
    q[..., 5] *= 6.0   # a loud channel: lists that are much alike, far from each other
    k[..., 5] *= 6.0
    q[:, prefix:] += 2.0 * torch.randn(blocks, 1, dim, generator=gen, device="cuda").repeat_interleave(64, 0)
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    kw = _options(blocks, prefix, cells, drop)
    assert _chosen(native_library, q, kw) == 1
    kw.update(layer=0, nvfp4_scales=(0.01, 0.01, 0.002))
    paired = [executor.sm100_ragged_attention(q, k, v, **kw) for _ in range(2)]
    executor._PAIR_Q64 = False
    try:
        single = executor.sm100_ragged_attention(q, k, v, **kw)
    finally:
        executor._PAIR_Q64 = True
    assert torch.isfinite(single).all()
    assert torch.equal(paired[0], single) and torch.equal(paired[1], single)
    assert executor.last_status() == 0


@pytest.mark.parametrize("blocks, heads, cells, chosen", [
    (200, 9, (0.0, 1.0, 0.0), 0), (200, 10, (0.0, 1.0, 0.0), 1),      # 80,000 stages of one cell
    (200, 19, (0.0, 0.5, 0.5), 0), (200, 20, (0.0, 0.5, 0.5), 1),     # 160,000 of several
    (32, 400, (0.0, 1.0, 0.0), 0), (4097, 1, (0.0, 1.0, 0.0), 0),     # blocks of a head
])
def test_where_pairs_are_chosen(native_library, blocks, heads, cells, chosen):
    q = torch.empty((1, 1, 1, 1), device="cuda", dtype=torch.bfloat16).expand(1, blocks * 64, heads, 64)
    assert _chosen(native_library, q, _options(blocks, 0, cells, 0.8)) == chosen
