"""A set status word: every CTA of a later launch leaves before it allocates or waits for anything."""

import pytest
import torch

from tests.helpers import smooth_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("query_block, dim, cells", [(64, 64, (0.4, 0.4, 0.2)), (128, 128, (0.0, 1.0, 0.0)),
                                                     (64, 128, (0.0, 0.5, 0.5))])
def test_set_word_leaves_the_output_alone(native_library, query_block, dim, cells):
    """Video tiles (pairs and single blocks) and prefix tiles, with a status word of the test's own:
    set, the kernels return without a write; clear, the same launches give the call's rows."""
    from anemoi_b200 import executor, native

    vs, prefix = (4, 16, 16), 70
    q, k, v = (t.cuda() for t in smooth_fields(*vs, 3, dim, prefix, seed=5, dtype=torch.bfloat16))
    _, parts = executor.sm100_ragged_attention(
        q, k, v, prefix_tokens=prefix, sparsity_ratio=0.5, retained_nvfp4_ratio=cells[0], retained_int8_ratio=cells[1],
        retained_fp16_ratio=cells[2], video_shape=vs, layer=0, query_block_size=query_block,
        nvfp4_scales=(0.01, 0.01, 0.002), return_parts=True)
    shape, store, lists, valid_k = (parts[n] for n in ("shape", "store", "lists", "valid_k"))
    lib, p, stream = native.library(), native._ptr, native._stream(q.device)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    packed, rows = torch.empty_like(parts["packed"]), torch.empty_like(parts["prefix_out"])
    pairs = native.pair_lists(shape, lists) if query_block == 64 else None

    def launch():
        packed.fill_(-7.0)
        rows.fill_(-7.0)
        if pairs is not None:
            code = lib.anemoi_sm100_attention_pairs(
                shape, store.struct, p(lists.row_offset), p(lists.row_counts), p(pairs.pair_counts), p(pairs.pair_ids),
                lists.capacity, p(valid_k), p(packed), p(status), stream)
        else:
            code = lib.anemoi_sm100_attention(
                shape, store.struct, p(lists.row_offset), p(lists.row_counts), p(lists.stage_ids), lists.capacity,
                p(valid_k), p(packed), p(status), stream)
        assert code == 0
        assert lib.anemoi_sm100_prefix_attention(shape, store.struct, p(valid_k), p(rows), p(status), stream) == 0
        torch.cuda.synchronize()

    status.fill_(5)
    launch()
    assert (packed == -7.0).all() and (rows == -7.0).all() and int(status.item()) == 5
    status.zero_()
    launch()
    live = (lists.row_counts[..., :3].sum(-1) > 0).view(-1)
    got, want = (t.view(live.numel(), query_block, dim)[live] for t in (packed, parts["packed"]))
    counts = parts["layout"].counts.repeat(shape.heads)[live]
    real = torch.arange(query_block, device="cuda") < counts[:, None]
    assert torch.equal(got[real], want[real])
    assert torch.equal(rows[:, :prefix], parts["prefix_out"][:, :prefix])
    assert int(status.item()) == 0 and executor.last_status() == 0
