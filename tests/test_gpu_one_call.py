"""The one-call layer and its one-kernel routing at the sizes where they can go wrong."""

import numpy as np
import pytest
import torch

from tests.helpers import smooth_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads, blocks", [(1, 1), (3, 2), (2, 31), (5, 33), (40, 97), (2, 257), (3, 671)])
@pytest.mark.parametrize("cells, prefix, phase", [((0.4, 0.4, 0.2), 70, 1), ((0.0, 1.0, 0.0), 0, -1),
                                                  ((0.5, 0.0, 0.5), 130, 2), ((1.0, 0.0, 0.0), 64, 0)])
def test_routing_lists_equal_the_oracle(native_library, heads, blocks, cells, prefix, phase):
    """One to eight CTAs per head, rows that do not divide evenly, maps shorter and longer than the
    pieces a warp reads ahead, many equal probabilities; lists, counts and launch order are exact."""
    from anemoi_b200 import native
    from anemoi_b200.routing import route_counts
    from oracle import route as R

    gen = torch.Generator(device="cuda").manual_seed(blocks)
    prob = torch.softmax(2 * torch.randn(heads, blocks, blocks, generator=gen, device="cuda"), -1)
    prob = (prob * 512).round().div(512).half()      # few distinct values: the boundaries fall among ties
    n16, n8, n4 = route_counts(blocks * blocks, sparsity_ratio=0.7, nvfp4_ratio=cells[0], int8_ratio=cells[1],
                               fp16_ratio=cells[2])
    stages = -(-prefix // 64)
    for block in (64, 128):
        shape = native.Shape(heads=heads, head_dim=128, query_block=block, seq_tokens=prefix + blocks * block,
                             prefix_tokens=prefix, video_blocks=blocks, has_nvfp4=1, has_int8=1, has_fp16=1,
                             has_prefix_query_int8=0, has_maxpool=0, input_is_bf16=1, q_global_scale=1.0,
                             k_global_scale=1.0, v_global_scale=1.0)
        lists = native.route(shape, prob, n16, n8, n4, phase)
        counts, offset, ids = (t.cpu().numpy() for t in (lists.row_counts, lists.row_offset, lists.stage_ids))
        for h in sorted({0, heads - 1}):
            out = R.route(prob[h].cpu().numpy(), n16, n8, n4)
            want = R.stage_lists(*out, query_block=block, prefix_stages=stages,
                                 prefix_phase=None if phase < 0 else ("nvfp4", "int8", "fp16")[phase])
            for i in range(blocks):
                n = [len(x) for x in want[i]]
                assert counts[h, i, :3].tolist() == n
                got = ids[h, offset[h, i]:offset[h, i] + sum(n)]
                assert np.array_equal(got, np.concatenate([np.asarray(x, dtype=np.int64) for x in want[i]]))
            total = counts[h, :, :3].sum(1)
            assert np.array_equal(counts[h, :, 3] - 1, np.lexsort((np.arange(blocks), -total)))
        if block == 128 or not native.library().anemoi_sm100_routes_in_one_kernel(shape):
            continue
        pairs = native.pair_lists(shape, lists)
        half = (blocks + 1) // 2
        offset2, counts2 = torch.empty_like(lists.row_offset), torch.empty_like(lists.row_counts)
        pc, ids2 = torch.empty_like(pairs.pair_counts), torch.empty_like(pairs.pair_ids)
        p = native._ptr
        assert native.library().anemoi_sm100_route_pairs(
            shape, p(prob), n16, n8, n4, phase, p(offset2), p(counts2), p(pc), p(ids2), lists.capacity,
            native._stream(prob.device)) == 0
        assert torch.equal(offset2, lists.row_offset) and torch.equal(counts2[..., :3], lists.row_counts[..., :3])
        assert torch.equal(pc, pairs.pair_counts)
        a, b, pc = pairs.pair_ids.cpu().numpy(), ids2.cpu().numpy(), pc.cpu().numpy()
        for h in sorted({0, heads - 1}):
            for t in range(half):
                at = offset[h, 2 * t]
                for c in range(3):
                    assert np.array_equal(a[h, at:at + pc[h, t, c]], b[h, at:at + pc[h, t, c]])
                    at += counts[h, 2 * t:2 * t + 2, c].sum()


@pytest.mark.parametrize("query_block, dim, dtype, heads, cells, prefix, prefix_query, maxpool", [
    (64, 64, torch.float16, 3, (0.4, 0.4, 0.2), 0, "int8", 0.0),
    (64, 128, torch.bfloat16, 2, (0.0, 1.0, 0.0), 75, "int8", 0.5),
    (128, 64, torch.bfloat16, 2, (0.0, 0.0, 1.0), 30, "fp16", 0.0),
    (128, 128, torch.float16, 5, (0.4, 0.4, 0.2), 129, "int8", 1.0),
    (128, 128, torch.bfloat16, 80, (0.0, 0.5, 0.5), 200, "int8", 0.0),      # prefix tiles start after routing
    (64, 64, torch.bfloat16, 4, (0.5, 0.0, 0.5), 64, "fp16", 0.0),
])
@pytest.mark.parametrize("drop", [0.5, 0.98])
def test_one_call_equals_the_stages(native_library, query_block, dim, dtype, heads, cells, prefix, prefix_query, maxpool,
                                    drop):
    """The call that runs everything in one native function, with the results written straight to
    their tokens, against the same call stage by stage with the assembly pass: bit for bit (at 98 %
    dropped with query blocks that keep nothing)."""
    from anemoi_b200 import executor

    vs = (3, 9, 21)
    q, k, v = (t.cuda() for t in smooth_fields(*vs, heads, dim, prefix, seed=3, outliers=(5, 41), dtype=dtype))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=drop, retained_nvfp4_ratio=cells[0], retained_int8_ratio=cells[1],
              retained_fp16_ratio=cells[2], video_shape=vs, layer=0, query_block_size=query_block,
              prefix_kv_precision="fp16" if cells[2] else "int8", prefix_query_precision=prefix_query,
              maxpool_weight=maxpool, nvfp4_scales=(0.01, 0.01, 0.002))
    one = executor.sm100_ragged_attention(q, k, v, **kw)
    staged, _ = executor.sm100_ragged_attention(q, k, v, return_parts=True, **kw)
    assert torch.equal(one.view(torch.int16), staged.view(torch.int16))
    assert executor.last_status() == 0
