"""Kernels whose split of the work follows the size of the grid: each branch of the rule."""

import ctypes as C

import numpy as np
import pytest
import torch

from tests.helpers import Records, smooth_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads, blocks, dim, weight", [
    (1, 1, 64, 0.0),       # one query block per warp: a grid of at most 148 CTAs
    (29, 40, 128, 0.5),
    (60, 17, 64, 0.25),    # two: 180 CTAs of one, 120 of two
    (2, 1185, 128, 0.5),   # two: four would not leave room for two CTAs on an SM
    (7, 273, 128, 0.5),    # two, three key tiles
    (80, 20, 128, 0.0),    # four
    (75, 33, 64, 1.0),     # four, the last CTA with one block
    (20, 300, 128, 0.5),   # four, three key tiles: the query rows change with the map
    (16, 672, 128, 0.0),   # four, six key tiles, exponentials kept
    (20, 385, 64, 0.5),    # four key tiles: the row's words are swizzled
    (18, 512, 128, 0.5),   # the last size of four rows with two maps
    (10, 1024, 128, 0.0),  # and with one, eight key tiles
    (10, 1025, 128, 0.0),  # past it
])
def test_draft_rows_per_warp(native_library, heads, blocks, dim, weight):
    """The draft map of pooled blocks, bit for bit the oracle's, first and last head."""
    from anemoi_b200 import native
    from oracle import route as R

    shape = native.Shape(heads=heads, head_dim=dim, query_block=128, seq_tokens=blocks * 128, prefix_tokens=0,
                         video_blocks=blocks, has_nvfp4=0, has_int8=1, has_fp16=0, has_prefix_query_int8=0,
                         has_maxpool=int(weight != 0.0), input_is_bf16=1, q_global_scale=1.0, k_global_scale=1.0,
                         v_global_scale=1.0)
    g = torch.Generator().manual_seed(5)
    pools = [torch.randn(heads, blocks, dim, generator=g).half() for _ in range(4)]
    q, k, qx, kx = (t.cuda() for t in pools)
    prob = torch.empty(heads, blocks, blocks, dtype=torch.float16, device="cuda")
    p = native._ptr
    assert native.library().anemoi_sm100_draft_probability(
        shape, p(q), p(k), p(qx), p(kx), weight, p(prob), native._stream(prob.device)) == 0
    for h in sorted({0, heads - 1}):
        want = R.draft_probability(*(t[h].numpy() for t in pools), weight)
        assert np.array_equal(prob[h].cpu().numpy().view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("blocks, weight", [
    (128, 0.0), (129, 0.5),                # one and two loads of four values per lane
    (384, 0.5), (385, 0.0), (512, 0.5),    # words in order, and swizzled
    (768, 0.5), (769, 0.5),                # exponentials kept, and formed twice
    (1000, 0.5), (2048, 0.0),              # eight and sixteen words swizzled
])
def test_draft_row_lengths(native_library, blocks, weight):
    """Rows around the steps of the softmax's layout, with logits far below the maximum among them, bit for bit."""
    from anemoi_b200 import native
    from oracle import route as R

    shape = native.Shape(heads=1, head_dim=64, query_block=64, seq_tokens=blocks * 64, prefix_tokens=0,
                         video_blocks=blocks, has_nvfp4=0, has_int8=1, has_fp16=0, has_prefix_query_int8=0,
                         has_maxpool=int(weight != 0.0), input_is_bf16=1, q_global_scale=1.0, k_global_scale=1.0,
                         v_global_scale=1.0)
    g = torch.Generator().manual_seed(blocks)
    pools = [torch.randn(1, blocks, 64, generator=g).half() for _ in range(4)]
    pools[0][:, ::7] *= 40.0
    pools[1][:, ::5] *= 3.0
    q, k, qx, kx = (t.cuda() for t in pools)
    prob = torch.empty(1, blocks, blocks, dtype=torch.float16, device="cuda")
    p = native._ptr
    assert native.library().anemoi_sm100_draft_probability(
        shape, p(q), p(k), p(qx), p(kx), weight, p(prob), native._stream(prob.device)) == 0
    want = R.draft_probability(*(t[0].numpy() for t in pools), weight)
    assert np.array_equal(prob[0].cpu().numpy().view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("dim, dtype", [(64, torch.float16), (128, torch.bfloat16)])
def test_preparation_of_many_q64_heads(native_library, dim, dtype):
    """32 heads of 9 Q64 blocks and a prefix (640 key and value tasks: one CTA per block for both)
    against each head alone (20 tasks: a CTA each): the same records, scales and pools."""
    from anemoi_b200 import executor

    vs, heads, prefix = (3, 9, 21), 32, 70
    q, k, v = (t.cuda() for t in smooth_fields(*vs, heads, dim, prefix, seed=2, outliers=(5, 41), dtype=dtype))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.5, retained_nvfp4_ratio=0.4, retained_int8_ratio=0.4,
              retained_fp16_ratio=0.2, video_shape=vs, layer=0, query_block_size=64, maxpool_weight=0.5,
              nvfp4_scales=(0.01, 0.01, 0.002), return_parts=True)

    def prepared(*tensors):
        _, parts = executor.sm100_ragged_attention(*tensors, **kw)
        torch.cuda.synchronize()
        return parts["store"], parts["shape"]

    many = prepared(q, k, v)
    assert (2 * many[1].video_blocks + 2) * heads == 640
    for h in (0, heads - 1):
        a = Records(*many, h)
        b = Records(*prepared(*(t[:, :, h:h + 1].contiguous() for t in (q, k, v))), 0)
        views = [(r.q_fp16(), *r.kv_fp16(), *r.q_int8(), *r.kv_int8(), *r.q_int8(prefix=True), *r.q_nvfp4(),
                  *r.kv_nvfp4(), *(r.b[n][r.h] for n in ("q_pool", "k_pool", "q_max_pool", "k_max_pool")))
                 for r in (a, b)]
        for x, y in zip(*views):
            assert x.dtype == y.dtype and x.tobytes() == y.tobytes()


@pytest.mark.parametrize("dim, query_block, heads, video, dtype", [
    (64, 64, 2, (3, 9, 21), torch.float16),       # keys and values in CTAs of their own; maxima found by those of values
    (128, 64, 2, (3, 30, 40), torch.bfloat16),    # the same after a kernel for the maxima
    (64, 64, 32, (3, 9, 21), torch.bfloat16),     # one CTA per block for both
    (128, 64, 32, (3, 9, 21), torch.float16),
    (64, 128, 2, (3, 9, 21), torch.bfloat16),     # 128-row blocks, either way to the maxima
    (64, 128, 32, (3, 9, 21), torch.float16),
    (128, 128, 2, (2, 9, 21), torch.float16),
    (128, 128, 32, (3, 9, 21), torch.bfloat16),
])
def test_records_do_not_depend_on_the_other_cells(native_library, dim, query_block, heads, video, dtype):
    """A preparation kernel holds the cells that its call may have (FP16 alone, no NVFP4, all): each cell's records,
    scales and the pools are those of every other kernel that writes them."""
    from anemoi_b200 import native
    from anemoi_b200.executor import make_shape
    from anemoi_b200.layout import materialize_ragged_2d_layout

    prefix = 70
    q, k, v = (t.cuda() for t in smooth_fields(*video, heads, dim, prefix, seed=3, outliers=(5, 41), dtype=dtype))
    layout = materialize_ragged_2d_layout(q.device, frames=video[0], height=video[1], width=video[2],
                                          logical_block=query_block)
    seen = {}
    for maxpool in (False, True):
        for cells in (("fp16",), ("int8",), ("int8", "fp16"), ("nvfp4",), ("nvfp4", "fp16"), ("nvfp4", "int8", "fp16")):
            shape = make_shape(q, prefix_tokens=prefix, video_blocks=layout.video_blocks, query_block_size=query_block,
                               active=cells, native_prefix=False, has_maxpool=maxpool, nvfp4_scales=(0.01, 0.01, 0.002))
            store = native.allocate_operands(shape, q.device)
            for t in store.buffers.values():
                if t is not None:
                    t.zero_()        # the bytes between the rows of a scale block are nobody's
            native.prepare(shape, q, k, v, layout.indices, layout.counts, store)
            torch.cuda.synchronize()
            for name, t in store.buffers.items():
                if t is not None:
                    bits = t.view(torch.uint8) if t.dtype != torch.uint8 else t
                    assert torch.equal(seen.setdefault(name, bits), bits), (name, cells, maxpool)
    assert len(seen) == len(native.Operands._fields_)


@pytest.mark.parametrize("cells", [("int8",), ("nvfp4",), ("fp16",)])
def test_layout_written_just_before(native_library, cells):
    """Slot tables that a kernel in front of the preparation writes (no kernel for the maxima between the two)."""
    from anemoi_b200 import native
    from anemoi_b200.executor import make_shape
    from anemoi_b200.layout import materialize_ragged_2d_layout

    video = (3, 9, 21)
    q, k, v = (t.cuda() for t in smooth_fields(*video, 4, 64, 0, seed=4))
    layout = materialize_ragged_2d_layout(q.device, frames=video[0], height=video[1], width=video[2], logical_block=64)
    shape = make_shape(q, prefix_tokens=0, video_blocks=layout.video_blocks, query_block_size=64, active=cells,
                       native_prefix=False, has_maxpool=False, nvfp4_scales=(0.01, 0.01, 0.002))
    assert native.library().anemoi_sm100_prepare_kernels(C.byref(shape)) == 1
    store = native.allocate_operands(shape, q.device)
    native.prepare(shape, q, k, v, layout.indices, layout.counts, store)
    want = {n: t.clone() for n, t in store.buffers.items() if n in ("q_pool", "k_pool", "k_int8_scale") and t is not None}
    for _ in range(20):
        counts, indices = torch.ones_like(layout.counts), torch.zeros_like(layout.indices)
        torch.cuda.synchronize()
        counts.copy_(layout.counts)
        indices.add_(layout.indices)
        native.prepare(shape, q, k, v, indices, counts, store)
        for n, t in want.items():
            assert torch.equal(store.buffers[n], t)


def test_repeated_public_calls(native_library):
    """A call with configuration objects seen before skips their checks, not the tensors': other
    strides, heads and types give what the staged path gives, and bad tensors still raise."""
    from anemoi_b200 import QuantConfig, SparseConfig, VisualLayout, anemoi_attention, executor

    vs, prefix = (2, 10, 14), 30
    layout, sparse = VisualLayout(vs, prefix), SparseConfig(64, 0.5, ((0, 1, 0.5), (1, 2, 0.8)))
    quant = QuantConfig(0.0, 0.5, 0.5)
    tokens = layout.sequence_tokens

    def call(q, k, v, layer=0):
        return anemoi_attention(q, k, v, layout=layout, layer=layer, sparse_config=sparse, quant_config=quant)

    def staged(q, k, v, layer=0):
        return executor.sm100_ragged_attention(
            q, k, v, prefix_tokens=prefix, sparsity_ratio=sparse.sparsity_for_layer(layer),
            retained_nvfp4_ratio=0.0, retained_int8_ratio=0.5, retained_fp16_ratio=0.5, video_shape=vs, layer=layer,
            query_block_size=64, return_parts=True)[0]

    packed = torch.randn(1, tokens, 3, 3, 128, device="cuda", dtype=torch.bfloat16)
    sets = [tuple(packed[:, :, i] for i in range(3)),
            tuple(packed[:, :, i].contiguous() for i in range(3)),
            tuple(packed[:, :, i, :2].half() for i in range(3))]
    for _ in range(2):
        for t in sets:
            for layer in (0, 1):
                assert torch.equal(call(*t, layer), staged(*t, layer))
    q, k, v = sets[1]
    shifted = torch.zeros(q.numel() + 1, dtype=q.dtype, device="cuda")[1:].view(q.shape)
    for bad in ((q[:, :-1], k, v), (q, k[:, :-1], v), (q, k, v.half()), (q, k, v.cpu()), (q[..., :64], k, v),
                (q, k, shifted)):
        with pytest.raises(ValueError):
            call(*bad)
    assert torch.equal(call(q, k, v), staged(q, k, v))


@pytest.mark.parametrize("video, heads, dim, dtype", [
    ((1, 8, 16), 1, 64, torch.float16),        # one range of tokens
    ((3, 12, 9), 5, 128, torch.bfloat16),      # three ranges and a half-empty group of channels
    ((4, 16, 16), 3, 64, torch.bfloat16),      # eight: the largest cluster
    ((3, 19, 18), 3, 64, torch.float16),       # nine: atomics
    ((2, 8, 16), 130, 128, torch.float16),     # many heads
    ((3, 16, 16), 12, 128, torch.bfloat16),    # found by the CTAs of values: 144 CTAs, the longest heads
    ((3, 16, 16), 13, 128, torch.bfloat16),    # 156: the kernel of six ranges
    ((1, 16, 96), 3, 64, torch.float16),       # 96 K values of a head: the last such length
    ((1, 16, 97), 3, 64, torch.float16),       # past it
    ((4, 16, 16), 3, 128, torch.bfloat16),     # the kernel's eight ranges
])
def test_value_maxima(native_library, video, heads, dim, dtype):
    """max |v| per head and channel, with the largest value at either end of the sequence, twice."""
    from anemoi_b200 import executor

    tokens = int(np.prod(video))
    q, k, v = (torch.randn(1, tokens, heads, dim, device="cuda").to(dtype) for _ in range(3))
    for at in (0, tokens - 1):
        v[0, at, :, 3:40:7] *= -8.0
        _, parts = executor.sm100_ragged_attention(
            q, k, v, prefix_tokens=0, sparsity_ratio=0.5, retained_nvfp4_ratio=0.0, retained_int8_ratio=1.0,
            retained_fp16_ratio=0.0, video_shape=video, layer=0, query_block_size=64, return_parts=True)
        got = parts["store"].buffers["v_amax"].view(heads, dim)
        assert torch.equal(got, v[0].abs().amax(0).half().float())


@pytest.mark.parametrize("video, prefix, heads, dim, query_block, dtype, kernels", [
    ((4, 16, 16), 0, 4, 64, 64, torch.bfloat16, 1),
    ((3, 16, 16), 0, 12, 128, 64, torch.float16, 1),      # 144 CTAs of values, 96 K values of a head
    ((3, 16, 16), 0, 13, 128, 64, torch.float16, 2),
    ((1, 16, 97), 0, 1, 64, 128, torch.bfloat16, 2),      # a row more than 96 K values
    ((5, 15, 17), 200, 5, 64, 128, torch.bfloat16, 1),    # prefix stages count, and their values
    ((2, 9, 21), 70, 16, 128, 128, torch.float16, 1),
    ((2, 9, 21), 70, 25, 128, 128, torch.float16, 2),
])
def test_value_maxima_of_short_sequences(native_library, video, prefix, heads, dim, query_block, dtype, kernels):
    """Where CTAs of values find the maxima themselves and where a kernel does: q|k|v views of one buffer, NaNs among
    the values (they win no maximum), the largest in the prefix or the last token.  The same records as the same
    heads among enough others for the kernel."""
    from anemoi_b200 import native
    from anemoi_b200.executor import make_shape
    from anemoi_b200.layout import materialize_ragged_2d_layout

    tokens, many = prefix + int(np.prod(video)), max(heads, 160)
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    base = torch.randn(1, tokens, heads, 3 * dim, generator=gen, device="cuda").to(dtype)
    base[0, 0, :, 2 * dim + 3] = 9.0
    base[0, tokens - 1, :, 2 * dim + 5] = -11.0
    base[0, 7::50, :, 2 * dim + 8] = float("nan")
    layout = materialize_ragged_2d_layout(base.device, frames=video[0], height=video[1], width=video[2],
                                          logical_block=query_block)

    def prepared(buffer):
        q, k, v = buffer.split(dim, dim=3)
        shape = make_shape(q, prefix_tokens=prefix, video_blocks=layout.video_blocks, query_block_size=query_block,
                           active=("int8",), native_prefix=prefix > 0, has_maxpool=False)
        store = native.allocate_operands(shape, q.device)
        native.prepare(shape, q, k, v, layout.indices, layout.counts, store)
        return native.library().anemoi_sm100_prepare_kernels(C.byref(shape)), store.buffers

    launched, own = prepared(base)
    assert launched == kernels
    v = base[0, :, :, 2 * dim:].float()
    want = torch.nan_to_num(v, nan=0.0).abs().amax(0)
    assert torch.equal(own["v_amax"].view(heads, dim), want) and want[0, 3] == 9.0 and want[0, 5] == 11.0
    launched, other = prepared(base.repeat(1, 1, -(-many // heads), 1))
    assert launched == 2
    for name in ("v_amax", "v_e4m3_scale", "kv_int8", "k_int8_scale", "q_int8", "q_int8_scale"):
        bits = own[name].view(torch.uint8)
        assert torch.equal(bits, other[name].view(torch.uint8)[:bits.numel()]), name


def _scalar_map(q, k, q_max, k_max, weight):
    """The map of one head with the kernel's maxima, which a NaN does not win (the oracle's does)."""
    from oracle import route as R

    def softmax(logit16):
        x = logit16.astype(np.float32)
        m = np.fmax.reduce(x, axis=1, keepdims=True, initial=-np.inf)
        y = np.fmax(((x - m) * R.LOG2E).astype(np.float32), np.float32(-125.0))
        n = np.rint(y).astype(np.float32)
        f = (y - n).astype(np.float32)
        p = np.full_like(f, R.EXP2_COEFFS[7])
        for c in R.EXP2_COEFFS[6::-1]:
            p = ((p * f).astype(np.float32) + c).astype(np.float32)
        e = np.ldexp(p, n.astype(np.int32)).astype(np.float32)
        return (e * (np.float32(1.0) / R._row_sum32(e)).astype(np.float32)[:, None]).astype(np.float32)

    with np.errstate(all="ignore"):
        if weight in (0.0, 1.0):
            return softmax(R._logits16(*((q, k) if weight == 0.0 else (q_max, k_max)))).astype(np.float16)
        w = np.float32(weight)
        a = ((np.float32(1.0) - w) * softmax(R._logits16(q, k))).astype(np.float32)
        return (a + (w * softmax(R._logits16(q_max, k_max))).astype(np.float32)).astype(np.float32).astype(np.float16)


@pytest.mark.parametrize("heads, blocks, dim, weight", [
    (2, 45, 64, 0.0), (3, 130, 128, 0.5),      # one row per warp
    (7, 273, 128, 0.5),                        # two
    (20, 300, 64, 1.0), (12, 800, 64, 0.0),    # four, exponentials kept and formed twice
])
def test_draft_map_of_infinities_and_nans(native_library, heads, blocks, dim, weight):
    """Pools with infinities and NaNs, and logits that overflow: bit for bit the scalar arithmetic."""
    from anemoi_b200 import native

    shape = native.Shape(heads=heads, head_dim=dim, query_block=64, seq_tokens=blocks * 64, prefix_tokens=0,
                         video_blocks=blocks, has_nvfp4=0, has_int8=1, has_fp16=0, has_prefix_query_int8=0,
                         has_maxpool=int(weight != 0.0), input_is_bf16=1, q_global_scale=1.0, k_global_scale=1.0,
                         v_global_scale=1.0)
    g = torch.Generator().manual_seed(blocks)
    pools = [torch.randn(heads, blocks, dim, generator=g).half() for _ in range(4)]
    for t in pools[::2]:
        t[:, 1] = float("nan")                    # a row of NaNs
        t[:, 2, 5] = float("inf")
        t[:, 3] *= 3000.0                         # logits past 65,504 once the keys are as large
        t[:, 4] = 0.0                             # a row of ties
    for t in pools[1::2]:
        t[:, 7, 3] = float("nan")                 # a column of NaNs
        t[:, 9, 5] = float("-inf")
        t[:, 11::13] *= 3000.0
    q, k, qx, kx = (t.cuda() for t in pools)
    prob = torch.empty(heads, blocks, blocks, dtype=torch.float16, device="cuda")
    p = native._ptr
    assert native.library().anemoi_sm100_draft_probability(
        shape, p(q), p(k), p(qx), p(kx), weight, p(prob), native._stream(prob.device)) == 0
    for h in (0, heads - 1):
        want = _scalar_map(*(t[h].numpy() for t in pools), weight)
        assert np.isfinite(want).all()
        assert np.array_equal(prob[h].cpu().numpy().view(np.uint16), want.view(np.uint16))
