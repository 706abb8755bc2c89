"""The NVFP4 scales of the executor's call, in every form that indexing and conversion to float take."""

import numpy as np
import pytest
import torch


def test_scales_are_read_at_every_call():
    from anemoi_b200.executor import _scale_array

    want = [0.5, 0.25, 2.0]
    for form in (tuple(want), want, np.array(want), want + [9.0], [torch.tensor(v) for v in want]):
        assert list(_scale_array(form)) == want
    held = tuple(torch.tensor(v) for v in want)
    assert list(_scale_array(held)) == want
    held[1].fill_(4.0)
    assert list(_scale_array(held)) == [0.5, 4.0, 2.0]
    for bad, error in (((0.5, 0.25), IndexError), (None, TypeError), (("0.5", 0.25, 2.0), TypeError)):
        with pytest.raises(error):
            _scale_array(bad)


@pytest.mark.gpu
def test_forms_of_the_scales(native_library):
    """A list and tensors give the tuple's bits; tensors changed in place give those of their new values."""
    from anemoi_b200 import executor

    q, k, v = (torch.randn(1, 2 * 10 * 14, 2, 128, device="cuda", dtype=torch.bfloat16) for _ in range(3))

    def call(scales, nvfp4=0.5):
        return executor.sm100_ragged_attention(
            q, k, v, prefix_tokens=0, sparsity_ratio=0.5, retained_nvfp4_ratio=nvfp4, retained_int8_ratio=1.0 - nvfp4,
            retained_fp16_ratio=0.0, video_shape=(2, 10, 14), layer=0, query_block_size=64, nvfp4_scales=scales)

    one, two = (0.01, 0.01, 0.002), (0.02, 0.005, 0.001)
    assert not torch.equal(call(one), call(two))
    assert torch.equal(call(list(one)), call(one))
    held = [torch.tensor(s, device="cuda") for s in one]
    assert torch.equal(call(held), call(one))
    for t, s in zip(held, two):
        t.fill_(s)
    assert torch.equal(call(held), call(two)) and torch.equal(call(tuple(held)), call(two))
    with pytest.raises(RuntimeError):
        call((0.0, 0.01, 0.01))
    with pytest.raises(TypeError):
        call(None, nvfp4=0.0)
