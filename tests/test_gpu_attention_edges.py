"""Stage lists at the edges of the attention kernel's rings, and every kernel of its dispatch.

With nothing dropped, a video of ``blocks`` 8x8 frames gives every query block a list of exactly
``blocks`` (Q64) or ``2 * blocks`` (Q128, every second stage fully masked) stages: one stage (one of
the two softmax warpgroups has none), an even and an odd few, and one less than, exactly and one more
than the eight entries of the per-stage rings and twice that.  The one-cell kernels and the mixed
one, both head dims and both query blocks.

Bound: output values are means of N(0,1) values, at most about 4.5 in size; the largest relative
rounding step of a probability is half an e2m1 step (1/6 at 3) in the NVFP4 cell, of which the oracle
and the kernel take the same, so what differs is the accumulation order and the exponential's last
bits: the 2e-2 of the other parity tests."""

import pytest
import torch

from tests.helpers import compare_metrics, smooth_fields

pytestmark = pytest.mark.gpu

CELLS = {"nvfp4": (1.0, 0.0, 0.0), "int8": (0.0, 1.0, 0.0), "fp16": (0.0, 0.0, 1.0), "mixed": (0.4, 0.3, 0.3)}


@pytest.mark.parametrize("cell", CELLS)
@pytest.mark.parametrize("dim, query_block", [(64, 64), (128, 64), (64, 128), (128, 128)])
@pytest.mark.parametrize("blocks", [1, 2, 3, 7, 8, 9, 17])
def test_short_lists_against_the_oracle(native_library, blocks, dim, query_block, cell):
    from anemoi_b200 import executor
    from anemoi_b200.partition import make_ragged_2d_partition
    from oracle import pipeline as PL, prep as P

    q, k, v = smooth_fields(blocks, 8, 8, 2, dim, 0, seed=blocks, dtype=torch.float16)
    scales = tuple(float(t.float().abs().max()) / (6 * 448) for t in (q, k, v))
    ratios = CELLS[cell]
    out = executor.sm100_ragged_attention(
        q.cuda(), k.cuda(), v.cuda(), prefix_tokens=0, sparsity_ratio=0.0, retained_nvfp4_ratio=ratios[0],
        retained_int8_ratio=ratios[1], retained_fp16_ratio=ratios[2], video_shape=(blocks, 8, 8), layer=0,
        query_block_size=query_block, nvfp4_scales=scales)
    assert executor.last_status() == 0
    geo = P.make_geometry(make_ragged_2d_partition(8, 8, query_block, include_adjacency=False).blocks, blocks, 8, 8,
                          query_block, 0)
    for h in range(2):
        want = PL.head_attention(q[0, :, h], k[0, :, h], v[0, :, h], geo, sparsity=0.0, ratios=ratios,
                                 prefix_kv_precision="int8", prefix_query_precision="int8", maxpool_weight=0.0,
                                 global_scales=scales)
        max_abs, cos, _ = compare_metrics(out[0, :, h].float().cpu().numpy(), want)
        assert max_abs <= 2e-2 and cos >= 0.999
