"""The public call finds its plan by the values of the configuration."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_equal_objects_share_a_plan(native_library):
    """Newly made configuration objects of equal values, integers beside floats, and a calibration of its
    own for each of 70 layers: one plan, the bits of the staged call.  Other values: another plan."""
    from anemoi_b200 import NVFP4Calibration, QuantConfig, SparseConfig, VisualLayout, anemoi_attention, executor

    vs, prefix = (2, 10, 14), 30
    q, k, v = (torch.randn(1, prefix + 280, 3, 128, device="cuda", dtype=torch.bfloat16) for _ in range(3))

    def call(scale, layer=0, drop=0.5, bands=()):
        return anemoi_attention(
            q, k, v, layout=VisualLayout(vs, prefix), layer=layer, sparse_config=SparseConfig(64, drop, bands, 0),
            quant_config=QuantConfig(0.5, 0.5, 0), calibration=NVFP4Calibration(scale, scale, 1))

    def staged(scale, drop=0.5):
        return executor.sm100_ragged_attention(
            q, k, v, prefix_tokens=prefix, sparsity_ratio=drop, retained_nvfp4_ratio=0.5, retained_int8_ratio=0.5,
            retained_fp16_ratio=0.0, video_shape=vs, layer=0, query_block_size=64, nvfp4_scales=(scale, scale, 1.0),
            return_parts=True)[0]

    executor._public_plan.cache_clear()
    for layer in range(70):
        out = call(0.01 + 0.001 * layer, layer)
        if layer % 23 == 0:
            assert torch.equal(out, staged(0.01 + 0.001 * layer))
    found = executor._public_plan.cache_info()
    assert (found.misses, found.hits) == (1, 69)
    bands = [(0, 1, 0.5), (1, 2, 0.8)]            # a list, which does not hash, and may change
    assert torch.equal(call(0.01, 1, bands=bands), staged(0.01, 0.8))
    bands[1] = (1, 2, 0.9)
    assert torch.equal(call(0.01, 1, bands=bands), staged(0.01, 0.9))
    assert torch.equal(call(0.01, 0, bands=bands), staged(0.01, 0.5))
    assert executor._public_plan.cache_info().misses == 3


def test_refusals_do_not_depend_on_earlier_calls(native_library):
    from anemoi_b200 import QuantConfig, SparseConfig, VisualLayout, anemoi_attention

    vs, prefix = (2, 10, 14), 30
    q, k, v = (torch.randn(1, prefix + 280, 2, 128, device="cuda", dtype=torch.bfloat16) for _ in range(3))

    def call(*tensors, quant=QuantConfig(), sparse=SparseConfig()):
        return anemoi_attention(*tensors, layout=VisualLayout(vs, prefix), layer=0, sparse_config=sparse,
                                quant_config=quant)

    for _ in range(2):
        want = call(q, k, v)
        with pytest.raises(RuntimeError, match="active INT8 phase"):
            call(q, k, v, quant=QuantConfig(0.0, 0.0, 1.0, "fp16", "int8"))
        with pytest.raises(ValueError):
            call(q.float(), k.float(), v.float())
        with pytest.raises(ValueError):
            call(*(t.expand(2, -1, -1, -1) for t in (q, k, v)))
        with pytest.raises(ValueError, match="share"):
            call(q, k[0], v)
        with pytest.raises(RuntimeError):
            call(q.cpu(), k.cpu(), v.cpu())
        twin = SimpleNamespace(query_block_size=64, sparsity_ratio=0.8, layer_sparsity_bands=(), maxpool_weight=0.0,
                               sparsity_for_layer=lambda layer: 0.8)
        assert torch.equal(call(q, k, v, sparse=twin), want)
        twin.maxpool_weight = 2.0
        with pytest.raises(ValueError):
            call(q, k, v, sparse=twin)


def test_block_size_of_another_type(native_library):
    """Refused before and after the same call with an integer."""
    from anemoi_b200 import executor

    q, k, v = (torch.randn(1, 280, 2, 64, device="cuda", dtype=torch.float16) for _ in range(3))

    def call(block):
        return executor.sm100_ragged_attention(
            q, k, v, prefix_tokens=0, sparsity_ratio=0.5, retained_nvfp4_ratio=0.0, retained_int8_ratio=1.0,
            retained_fp16_ratio=0.0, video_shape=(2, 10, 14), layer=0, query_block_size=block)

    executor._plan.cache_clear()
    for _ in range(2):
        with pytest.raises(TypeError):
            call(64.0)
        call(64)
