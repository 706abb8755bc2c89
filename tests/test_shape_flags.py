"""The shape's switches are flags: every value but 0 means the same."""

import pytest


def _shape(**flags):
    from anemoi_b200 import native

    fields = dict(has_nvfp4=0, has_int8=1, has_fp16=1, has_prefix_query_int8=1)
    fields.update(flags)
    return native.Shape(heads=3, head_dim=64, query_block=64, seq_tokens=200 + 9 * 64, prefix_tokens=200, video_blocks=9,
                        has_maxpool=0, input_is_bf16=1, q_global_scale=1.0, k_global_scale=1.0, v_global_scale=1.0,
                        **fields)


@pytest.mark.parametrize("prefix_query_int8", [0, 1])
@pytest.mark.parametrize("flag", ["has_nvfp4", "has_int8", "has_fp16"])
@pytest.mark.parametrize("value", [2, -1, 255])
def test_any_true_value(native_library, flag, value, prefix_query_int8):
    import ctypes as C

    from anemoi_b200 import native

    one = _shape(**{"has_prefix_query_int8": prefix_query_int8, flag: 1})
    other = _shape(**{"has_prefix_query_int8": prefix_query_int8, flag: value})
    for which in range(native.BUF_COUNT):
        size = native_library.anemoi_sm100_operand_bytes(C.byref(one), which)
        assert size >= 0 and native_library.anemoi_sm100_operand_bytes(C.byref(other), which) == size
    assert (native_library.anemoi_sm100_prepare_kernels(C.byref(other))
            == native_library.anemoi_sm100_prepare_kernels(C.byref(one)) > 0)
