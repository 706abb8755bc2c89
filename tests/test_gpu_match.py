"""Q64 pairs chosen by what the blocks' lists share: bit for bit one block per CTA."""

import ctypes as C
import math

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


def _two_kinds(blocks, heads, dim, first_peaked, columns):
    """Q/K/V in which every other block of queries has half its weight on one block of keys, or nearly all of it on two (of the
    second less), and the others attend to all blocks about alike."""
    gen = torch.Generator(device="cuda").manual_seed(blocks + heads)
    # (orthogonal: the shares are what is asked for)
    u = torch.linalg.qr(torch.randn(heads, dim, dim, generator=gen, device="cuda"))[0][:, :blocks]
    u = u.permute(1, 0, 2)[:, None] * dim ** 0.5
    q = 0.3 * torch.randn(blocks, 64, heads, dim, generator=gen, device="cuda")
    for i in range(0 if first_peaked else 1, blocks, 2):
        for c in range(columns):
            q[i] += (math.log(blocks) if columns == 1 else 16.0 - 0.5 * c) * dim ** -0.5 * u[(i * 7 + c * 5) % blocks]
    k = u + 0.3 * torch.randn(blocks, 64, heads, dim, generator=gen, device="cuda")
    v = torch.randn(blocks, 64, heads, dim, generator=gen, device="cuda")
    return tuple(t.reshape(1, blocks * 64, heads, dim).to(torch.float16) for t in (q, k, v))


@pytest.mark.parametrize("first_peaked", [True, False])
@pytest.mark.parametrize("columns, int8, fp16, without, partner", [
    (2, 16, 0, (16, 0, 0), (14, 2, 0)),      # no INT8 phase, NVFP4 before it
    (1, 128, 8, (15, 0, 1), (0, 16, 0)),     # no middle phase: three cells
    (2, 8, 8, (16, 0, 0), (14, 1, 1)),       # the first phase alone
])
@pytest.mark.parametrize("dim", [64, 128])
def test_rows_do_not_depend_on_the_phases_of_the_other_block(native_library, dim, first_peaked, columns, int8, fp16,
                                                             without, partner):
    """Pairs in which a block has no stage of a phase that its partner has: bit for bit one block per CTA."""
    from anemoi_b200 import executor

    blocks, heads = 16, 6
    q, k, v = _two_kinds(blocks, heads, dim, first_peaked, columns)
    int8, fp16 = int8 / blocks ** 2, fp16 / blocks ** 2
    kw = _options(blocks, 0, (1.0 - int8 - fp16, int8, fp16), 0.0)
    kw.update(layer=0, nvfp4_scales=(0.01, 0.01, 0.002))
    paired, parts = executor.sm100_ragged_attention(q, k, v, return_parts=True, **kw)
    own = parts["lists"].row_counts[..., :3].cpu()
    kinds = [tuple(own[0, i].tolist()) for i in (0, 1)]
    assert set(kinds) == {without, partner}, kinds
    assert all(tuple(own[h, i].tolist()) == kinds[i % 2] for h in range(heads) for i in range(blocks))
    called = executor.sm100_ragged_attention(q, k, v, **kw)
    executor._PAIR_Q64 = False
    try:
        single = executor.sm100_ragged_attention(q, k, v, **kw)
    finally:
        executor._PAIR_Q64 = True
    assert torch.isfinite(single).all()
    assert torch.equal(paired, single) and torch.equal(called, single)


def test_heads_alone_equal_one_call_with_chosen_pairs(native_library):
    """The whole call chooses its pairs, a head alone takes neighbours; every block of one kind has no INT8 phase."""
    from anemoi_b200 import executor

    blocks, heads = 128, 10
    q, k, v = _two_kinds(blocks, heads, 128, True, 1)
    kw = _options(blocks, 0, (63.5 / 128, 64 / 128, 0.5 / 128), 0.0)
    assert _chosen(native_library, q, kw) == 1 and _chosen(native_library, q[:, :, :1], kw) == 0
    kw.update(layer=0, nvfp4_scales=(0.01, 0.01, 0.002))
    whole = executor.sm100_ragged_attention(q, k, v, **kw)
    for h in range(heads):
        assert torch.equal(whole[:, :, h:h + 1], executor.sm100_ragged_attention(*(t[:, :, h:h + 1] for t in (q, k, v)), **kw))


@pytest.mark.parametrize("blocks, heads, prefix, cells, counted", [
    (129, 64, 37, (0.4, 0.4, 0.2), 2),
    (1025, 1, 0, (0.0, 1.0, 0.0), 6),      # routing in several kernels
    (64, 2, 0, (0.0, 1.0, 0.0), 1),        # neighbours
])
def test_stages_take_the_pairs_of_the_call(native_library, blocks, heads, prefix, cells, counted):
    """Stage by stage (NVTX ranges, stage events) a call walks the lists that it walks in one."""
    from anemoi_b200 import executor, native

    gen = torch.Generator(device="cuda").manual_seed(blocks)
    q, k, v = (torch.randn(1, prefix + blocks * 64, heads, 64, generator=gen, device="cuda").to(torch.bfloat16)
               for _ in range(3))
    kw = _options(blocks, prefix, cells, 0.8)
    assert _chosen(native_library, q, kw) == (counted > 1)
    kw.update(layer=0, nvfp4_scales=(0.01, 0.01, 0.002))
    whole = executor.sm100_ragged_attention(q, k, v, **kw)
    before = dict(native.LAUNCHES)
    staged = executor.sm100_ragged_attention(q, k, v, profile_nvtx=True, **kw)
    assert torch.equal(staged, whole)
    assert native.LAUNCHES["route"] - before.get("route", 0) == counted
    assert native.LAUNCHES.get("pair_lists", 0) - before.get("pair_lists", 0) == (2 if counted == 1 else 0)
    assert executor.last_status() == 0


@pytest.mark.parametrize("cells, prefix_kv", [((0.0, 1.0, 0.0), "fp16"), ((0.0, 1.0, 0.0), "nvfp4"), ((1.0, 0.0, 0.0), "int8"),
                                              ((0.5, 0.0, 0.5), "int8"), ((0.0, 0.5, 0.5), "nvfp4")])
def test_prefix_stages_in_a_phase_of_their_own(native_library, cells, prefix_kv):
    """The prefix is all that the lists have of its phase: in front of the others, between or behind them."""
    from anemoi_b200 import executor

    blocks, heads, prefix = 129, 50, 150
    gen = torch.Generator(device="cuda").manual_seed(blocks)
    q, k, v = (torch.randn(1, prefix + blocks * 64, heads, 64, generator=gen, device="cuda").to(torch.bfloat16)
               for _ in range(3))
    kw = dict(_options(blocks, prefix, cells, 0.8), prefix_kv_precision=prefix_kv)
    assert _chosen(native_library, q, kw) == 1
    kw.update(layer=0, nvfp4_scales=(0.01, 0.01, 0.002))
    paired = executor.sm100_ragged_attention(q, k, v, **kw)
    executor._PAIR_Q64 = False
    try:
        single = executor.sm100_ragged_attention(q, k, v, **kw)
    finally:
        executor._PAIR_Q64 = True
    assert torch.isfinite(single).all() and torch.equal(paired, single)
    assert executor.last_status() == 0
