"""HostAttention: the shrinking last groups."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_host_call_with_shrinking_groups(native_library):
    """Large heads: the last group is split (4, 2, 1, 1 heads here, views of the group's buffers);
    bit-equal to one call on the device, twice in a row on the same buffers."""
    from anemoi_b200 import HostAttention, QuantConfig, SparseConfig, VisualLayout, anemoi_attention

    layout, heads = VisualLayout((6, 40, 60), 100), 8
    q, k, v = (torch.randn(1, layout.sequence_tokens, heads, 128, dtype=torch.bfloat16).pin_memory() for _ in range(3))
    out = torch.empty_like(q).pin_memory()
    runner = HostAttention("cuda", group_heads=4)
    assert runner._groups(heads, 3 * layout.sequence_tokens * 256) == [(0, 4), (4, 6), (6, 7), (7, 8)]
    how = dict(layout=layout, layer=0, sparse_config=SparseConfig(128, 0.8), quant_config=QuantConfig(0.0, 0.5, 0.5))
    want = anemoi_attention(*(t.cuda() for t in (q, k, v)), **how).cpu()
    for _ in range(2):
        out.zero_()
        runner(q, k, v, out, **how)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
