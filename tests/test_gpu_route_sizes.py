"""Routing and the order of the launches where their rules change."""

import ctypes as C

import pytest
import torch

from tests.test_gpu_one_call import test_routing_lists_equal_the_oracle as lists_equal_the_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads, blocks, one_kernel", [
    (75, 1100, 1),      # one CTA per head with more rows than threads: a second round of the scans
    (16, 592, 1),       # clusters of four
    (33, 400, 1),
    (34, 400, 0),       # 68 CTAs in clusters of two, long maps: five kernels
    (36, 672, 0),
    (37, 400, 1),       # 74 CTAs
    (2, 500, 1),        # few heads, clusters of eight: up to 65,536 pairs per CTA
    (2, 800, 0),
])
def test_each_side_of_the_one_kernel_rule(native_library, heads, blocks, one_kernel):
    from anemoi_b200 import native

    shape = native.Shape(heads=heads, head_dim=128, query_block=64, seq_tokens=70 + blocks * 64, prefix_tokens=70,
                         video_blocks=blocks, has_nvfp4=1, has_int8=1, has_fp16=1, has_prefix_query_int8=0,
                         has_maxpool=0, input_is_bf16=1, q_global_scale=1.0, k_global_scale=1.0, v_global_scale=1.0)
    assert native.library().anemoi_sm100_routes_in_one_kernel(C.byref(shape)) == one_kernel
    lists_equal_the_oracle(native_library, heads, blocks, (0.4, 0.4, 0.2), 70, 1)


@pytest.mark.parametrize("heads, query_block", [(18, 128), (19, 128), (18, 64), (19, 64)])
def test_prefix_tiles_beside_and_after_routing(native_library, heads, query_block):
    """A prefix of 1,000 tokens is eight tiles per head: 144 of them start before routing, whose clusters need SMs
    of their own, 152 after it.  Bit for bit the stages."""
    from anemoi_b200 import executor

    vs, prefix = (5, 30, 52), 1000
    gen = torch.Generator(device="cuda").manual_seed(heads)
    q, k, v = (torch.randn(1, prefix + 7800, heads, 128, generator=gen, device="cuda").to(torch.bfloat16)
               for _ in range(3))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.8, retained_nvfp4_ratio=0.0, retained_int8_ratio=0.5,
              retained_fp16_ratio=0.5, video_shape=vs, layer=0, query_block_size=query_block)
    staged, _ = executor.sm100_ragged_attention(q, k, v, return_parts=True, **kw)
    for _ in range(3):
        assert torch.equal(executor.sm100_ragged_attention(q, k, v, **kw), staged)
    assert executor.last_status() == 0


@pytest.mark.parametrize("video, query_block, dim, weight, prefix, one_launch", [
    ((1, 8, 16), 64, 64, 0.0, 0, 1),       # two blocks
    ((31, 8, 8), 64, 128, 0.5, 0, 1),      # 31 blocks, both maps, pairs with a single block at the end
    ((32, 8, 16), 128, 64, 1.0, 0, 1),     # 32 blocks, the max pools' map alone
    ((32, 8, 16), 128, 128, 0.5, 0, 1),
    ((32, 8, 16), 128, 128, 0.5, 20, 0),   # a draft launch of its own: beside prefix tiles
    ((33, 8, 8), 64, 64, 0.5, 0, 0),       # and for more blocks
])
def test_map_and_routing_in_one_launch(native_library, video, query_block, dim, weight, prefix, one_launch):
    """Calls whose routing kernel forms the draft map, up to 32 blocks per head and no prefix: bit for bit the stages."""
    from anemoi_b200 import executor, native

    frames, height, width = video
    tokens = prefix + frames * height * width
    shape = native.Shape(heads=3, head_dim=dim, query_block=query_block, seq_tokens=tokens, prefix_tokens=prefix,
                         video_blocks=frames * height * width // query_block, has_nvfp4=0, has_int8=1, has_fp16=1,
                         has_prefix_query_int8=0, has_maxpool=int(weight != 0.0), input_is_bf16=0, q_global_scale=1.0,
                         k_global_scale=1.0, v_global_scale=1.0)
    assert native.library().anemoi_sm100_drafts_in_routing(C.byref(shape)) == one_launch
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    q, k, v = (torch.randn(1, tokens, 3, dim, generator=gen, device="cuda").half() for _ in range(3))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.7, retained_nvfp4_ratio=0.0, retained_int8_ratio=0.6,
              retained_fp16_ratio=0.4, video_shape=video, layer=0, query_block_size=query_block, maxpool_weight=weight)
    staged, _ = executor.sm100_ragged_attention(q, k, v, return_parts=True, **kw)
    for _ in range(3):
        assert torch.equal(executor.sm100_ragged_attention(q, k, v, **kw), staged)
    assert executor.last_status() == 0


@pytest.mark.parametrize("video, query_block, dim, weight", [
    ((1, 8, 16), 64, 64, 0.0), ((17, 8, 8), 64, 128, 0.5), ((31, 8, 8), 64, 64, 1.0), ((32, 8, 16), 128, 128, 0.5),
])
@pytest.mark.parametrize("values", ["plain", "ties", "overflow"])
def test_map_of_the_one_launch(native_library, video, query_block, dim, weight, values):
    """The map that the routing kernel forms (it lies in the layer's workspace), bit for bit the draft kernel's and
    the oracle's on the same pools: rows of ties, logits far below the maximum, and ones that overflow to infinity."""
    import numpy as np

    from anemoi_b200 import executor, native
    from oracle import route as R

    heads, tokens = 3, video[0] * video[1] * video[2]
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    q, k, v = (torch.randn(1, tokens, heads, dim, generator=gen, device="cuda") for _ in range(3))
    if values == "ties":
        q[:, ::2] = 0.0
        q[:, 1::2] *= 40.0
        k[:, tokens // 2:] = k[:, :tokens - tokens // 2].clone()
    elif values == "overflow":
        q, k = q.abs() * 900.0, k * 900.0        # mean pools too have entries of some hundreds
    q, k, v = (t.half() for t in (q, k, v))
    plan = executor._Plan(q.device, tokens, heads, dim, q.dtype, 0, 0.7, 0.0, 0.6, 0.4, video, query_block, "int8",
                          "int8", weight, True)
    lib, shape = native.library(), plan.struct.shape
    assert lib.anemoi_sm100_drafts_in_routing(C.byref(shape)) == 1
    workspace = torch.empty(plan.bytes, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(q)
    strides = executor._stride_array(*(heads * dim, dim) * 3)
    assert plan.call(plan.ref, q.data_ptr(), k.data_ptr(), v.data_ptr(), strides, executor._scale_array((1.0, 1.0, 1.0)),
                     None, 0, 1, out.data_ptr(), workspace.data_ptr(), plan.bytes,
                     torch.cuda.current_stream().cuda_stream, None) == 0
    # the workspace is cut in this order, each piece a multiple of 256 bytes
    at = 0
    for which in (native.BUF_V_AMAX, native.BUF_Q_FP16, native.BUF_KV_FP16, native.BUF_Q_INT8, native.BUF_KV_INT8,
                  native.BUF_Q_NVFP4, native.BUF_KV_NVFP4, native.BUF_Q_INT8_SCALE, native.BUF_K_INT8_SCALE,
                  native.BUF_V_E4M3_SCALE):
        at += -(-lib.anemoi_sm100_operand_bytes(C.byref(shape), which) // 256) * 256
    blocks, pools = shape.video_blocks, {}

    def take(*size):
        nonlocal at
        n = 2 * int(np.prod(size))
        piece = workspace[at:at + n].view(torch.float16).view(size)
        at += -(-n // 256) * 256
        return piece

    for name in ("q_pool", "k_pool", "q_max_pool", "k_max_pool")[:4 if weight else 2]:
        pools[name] = take(heads, blocks, dim)
    got = take(heads, blocks, blocks)
    pools = {n: pools.get(n) for n in ("q_pool", "k_pool", "q_max_pool", "k_max_pool")}
    store = native.OperandStore(shape=shape, struct=native.Operands(), buffers=pools)
    assert torch.equal(got.view(torch.int16), native.draft_probability(shape, store, weight).view(torch.int16))
    if values != "overflow":
        for h in range(heads):
            want = R.draft_probability(*(None if t is None else t[h].cpu().numpy() for t in pools.values()), weight)
            assert np.array_equal(got[h].cpu().numpy().view(np.uint16), want.view(np.uint16))
    else:
        assert torch.isfinite(got).all()
    assert executor.last_status() == 0


@pytest.mark.parametrize("heads, blocks", [(3, 1), (3, 2), (2, 31), (2, 32), (2, 33), (5, 63), (150, 64), (2, 65)])
@pytest.mark.parametrize("cells, prefix, phase", [((0.4, 0.4, 0.2), 0, -1), ((0.0, 1.0, 0.0), 200, 1), ((0.5, 0.0, 0.5), 70, 2)])
def test_short_maps(native_library, heads, blocks, cells, prefix, phase):
    """Up to 64 blocks a head's map is held in registers: one and two columns per lane, and the kernel past it."""
    lists_equal_the_oracle(native_library, heads, blocks, cells, prefix, phase)


@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("heads, blocks", [(3, 7), (3, 40), (3, 64), (3, 101), (1, 1100)])
def test_arrays_on_four_bytes(native_library, heads, blocks, pairs):
    """The caller's arrays start at any int: the same lists as in arrays on 16 bytes."""
    from anemoi_b200 import native

    shape = native.Shape(heads=heads, head_dim=64, query_block=64, seq_tokens=blocks * 64, prefix_tokens=0, video_blocks=blocks,
                         has_nvfp4=0, has_int8=1, has_fp16=1, has_prefix_query_int8=0, has_maxpool=0, input_is_bf16=1,
                         q_global_scale=1.0, k_global_scale=1.0, v_global_scale=1.0)
    if pairs and not native.library().anemoi_sm100_routes_in_one_kernel(C.byref(shape)):
        pytest.skip("pairs of their own launches")
    gen = torch.Generator(device="cuda").manual_seed(blocks)
    prob = torch.rand(heads, blocks, blocks, generator=gen, device="cuda").to(torch.float16)
    n16, n8 = blocks * blocks // 10, blocks * blocks // 10 + 1
    capacity = native_library.anemoi_sm100_route_list_capacity(C.byref(shape), n16, n8, 0, -1)
    scratch = torch.empty(native_library.anemoi_sm100_route_scratch_bytes(C.byref(shape)), dtype=torch.uint8, device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    tiles = (blocks + 1) // 2
    sizes = [heads * blocks, heads * blocks * 4] + ([heads * tiles * 4] if pairs else []) + [heads * capacity]
    got = []
    for shift in (0, 1, 2, 3):
        out = [torch.full((n + 4,), -7, dtype=torch.int32, device="cuda")[shift:shift + n] for n in sizes]
        ptr = [C.c_void_p(t.data_ptr()) for t in out]
        if pairs:
            code = native_library.anemoi_sm100_route_pairs(C.byref(shape), C.c_void_p(prob.data_ptr()), n16, n8, 0, -1, *ptr,
                                                           capacity, stream)
        else:
            code = native_library.anemoi_sm100_route(C.byref(shape), C.c_void_p(prob.data_ptr()), n16, n8, 0, -1,
                                                     C.c_void_p(scratch.data_ptr()), scratch.numel(), *ptr, capacity, stream)
        assert code == 0
        got.append(out)
    torch.cuda.synchronize()
    for out in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(out, got[0]))
