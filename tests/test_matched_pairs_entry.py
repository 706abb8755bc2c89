"""The stages of a call whose pairs are chosen: what their entry points refuse (on the host, before any launch)."""

import ctypes as C

import pytest

PTRS = dict(prob=0x10000, scratch=0x20000, row_offset=0x30000, row_counts=0x40000, bits=0x50000, table=0x60000, ids=0x70000)


def _plan(native, library, blocks, heads, query_block=64, pair_q64=1):
    shape = native.Shape(heads=heads, head_dim=64, query_block=query_block, seq_tokens=blocks * query_block, prefix_tokens=0,
                         video_blocks=blocks, has_nvfp4=0, has_int8=1, has_fp16=0, has_prefix_query_int8=0, has_maxpool=0,
                         input_is_bf16=1, q_global_scale=1.0, k_global_scale=1.0, v_global_scale=1.0)
    n8 = blocks * blocks // 5
    capacity = library.anemoi_sm100_route_list_capacity(C.byref(shape), 0, n8, 0, -1)
    return native.LayerPlan(shape=shape, indices=0x1000, counts=0x2000, valid_k=0x3000, status=0x4000, n16=0, n8=n8, n4=0,
                            list_capacity=capacity, prefix_phase=-1, pair_q64=pair_q64, maxpool_weight=0.0)


def _route(library, plan, short=0, **ptrs):
    p = {**PTRS, **ptrs}
    size = library.anemoi_sm100_route_scratch_bytes(C.byref(plan.shape)) - short
    return library.anemoi_sm100_route_matched(C.byref(plan), p["prob"], p["scratch"], size, p["row_offset"],
                                              p["row_counts"], p["bits"], p["table"], p["ids"], None)


def test_bits_are_a_word_per_32_columns_in_pieces_of_128(native_library):
    from anemoi_b200 import native

    plan = _plan(native, native_library, 200, 10)
    assert native_library.anemoi_sm100_pair_bits_bytes(C.byref(plan)) == 10 * 1 * 200 * 8 * 4


@pytest.mark.parametrize("blocks, heads, query_block, pair_q64", [(200, 9, 64, 1), (200, 10, 128, 1), (200, 10, 64, 0)])
def test_plans_without_chosen_pairs_are_refused(native_library, blocks, heads, query_block, pair_q64):
    from anemoi_b200 import native

    plan = _plan(native, native_library, blocks, heads, query_block, pair_q64)
    assert native_library.anemoi_sm100_pair_bits_bytes(C.byref(plan)) == -1
    assert _route(native_library, plan) == -1


@pytest.mark.parametrize("wrong", [dict(row_counts=0x40004), dict(bits=0x50008), dict(table=0x60004), dict(prob=None),
                                   dict(scratch=None), dict(row_offset=None), dict(ids=None), dict(short=1)])
def test_pointers_that_do_not_fit_are_refused(native_library, wrong):
    from anemoi_b200 import native

    assert _route(native_library, _plan(native, native_library, 200, 10), **wrong) == -1


@pytest.mark.parametrize("table", [None, 0x60004])
def test_attention_refuses_a_table_off_16_bytes(native_library, table):
    from anemoi_b200 import native

    plan = _plan(native, native_library, 200, 10)
    ops = native.Operands(**{name: 0x100000 for name, _ in native.Operands._fields_})
    assert native_library.anemoi_sm100_attention_matched(C.byref(plan.shape), C.byref(ops), 0x30000, 0x40000, table, 0x70000,
                                                         plan.list_capacity, 0x3000, 0x80000, 0x4000, None) == -1
