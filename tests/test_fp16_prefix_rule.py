"""Which FP16 prefix queries take the FP16 cell's kernel: both sides of each line."""

import pytest

from anemoi_b200.executor import _fp16_prefix


@pytest.mark.parametrize("prefix, heads, dim, query_block, blocks, active, sparsity, kernel", [
    (0, 4, 64, 64, 100, ("fp16",), 0.8, False),
    (62, 5, 64, 64, 592, ("nvfp4", "int8", "fp16"), 0.8, True),
    (62, 5, 64, 64, 592, ("nvfp4", "int8"), 0.8, False),          # no FP16 keys and values
    (100, 147, 64, 128, 8, ("fp16",), 0.8, True),                 # tiles: fewer than one per SM
    (100, 148, 64, 128, 8, ("fp16",), 0.8, False),
    (500, 12, 64, 128, 160, ("fp16",), 0.8, True),                # 15,744 and 20,992 steps of 20,000
    (500, 16, 64, 128, 160, ("fp16",), 0.8, False),
    (500, 12, 128, 128, 61, ("int8", "fp16"), 0.8, True),         # 6,240 steps: of 10,000, and of 5,000
    (500, 12, 128, 128, 61, ("fp16",), 0.8, False),
    (427, 2, 128, 128, 168, ("int8", "fp16"), 0.9, False),        # the prefix's walk is the longest of the call
    (427, 6, 128, 128, 168, ("int8", "fp16"), 0.5, True),
    (427, 2, 64, 128, 168, ("int8", "fp16"), 0.9, True),
])
def test_rule(prefix, heads, dim, query_block, blocks, active, sparsity, kernel):
    assert _fp16_prefix(prefix, heads, dim, query_block, blocks, active, sparsity) is kernel
