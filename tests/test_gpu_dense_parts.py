"""Dense rows whose keys are shared by up to eight CTAs: every length of the merge, and infinities in one part of it."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense(q, k, v, rows):
    scores = torch.einsum("bqhd,bkhd->bhqk", q[:, :rows].double(), k.double()) / q.size(3) ** 0.5
    return torch.einsum("bhqk,bkhd->bhqd", scores.softmax(-1), v.double())[0]


# one row and a whole tile of eight parts, the last stage of one key; four, two and one part at more tiles
@pytest.mark.parametrize("tokens, rows, parts", [(255 * 64 + 1, 1, 8), (256 * 64 + 5, 127, 8), (40_000, 128, 8), (40_000, 256, 4),
                                                 (255 * 64 + 1, 384, 4), (200 * 64 + 63, 128, 4), (255 * 64, 200, 2),
                                                 (97 * 64, 513, 2), (95 * 64, 513, 1)])
@pytest.mark.parametrize("dim, dtype", [(64, torch.float16), (128, torch.bfloat16), (128, torch.float16)])
def test_rows(native_library, tokens, rows, parts, dim, dtype):
    from anemoi_b200 import executor, native

    assert native_library.anemoi_sm100_dense_parts(tokens, rows) == parts
    gen = torch.Generator(device="cuda").manual_seed(tokens + rows)
    q, k, v = (torch.randn(1, tokens, 2, dim, generator=gen, device="cuda").to(dtype) for _ in range(3))
    status = executor._status_word(q.device)
    out = native.dense_rows(q, k, v, rows, status)
    want = _dense(q, k, v, rows)
    # probabilities and results rounded once each (bf16: 2^-9, fp16: 2^-12 at most)
    assert (out.double() - want).norm() / want.norm() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
    assert torch.equal(native.dense_rows(*(t[:, :, 1:] for t in (q, k, v)), rows, status)[0], out[1])
    assert executor.last_status() == 0


@pytest.mark.parametrize("tokens, parts", [(2_500, 2), (9_000, 4), (17_000, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_infinities_in_one_part(native_library, tokens, parts, dtype):
    """A key of infinities (weightless where the score is -inf, NaN where it is +inf), a part whose keys have all scores
    at -inf beside finite ones, and one key above all others."""
    from anemoi_b200 import executor, native

    heads, dim, rows = 2, 64, 100
    assert native_library.anemoi_sm100_dense_parts(tokens, rows) == parts
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    q, k, v = (torch.randn(1, tokens, heads, dim, generator=gen, device="cuda").to(dtype) for _ in range(3))
    q[:, :rows, :, 5] = torch.where(torch.arange(rows, device="cuda")[:, None] % 3 == 0, 1.0, -1.0).to(dtype)
    status = executor._status_word(q.device)
    stages = (tokens + 63) // 64
    for part in (0, parts // 2, parts - 1):
        first, last = (64 * (stages * n // parts) for n in (part, part + 1))
        one, whole, high = k.clone(), k.clone(), k.clone()
        one[:, first + 70, :, 5] = float("inf")
        whole[:, first:last, :, 5] = float("inf")
        high[:, first + 3] = q[:, 7] * 60
        for name, keys in (("one", one), ("whole", whole), ("high", high)):
            out = native.dense_rows(q, keys, v, rows, status).double()
            want = _dense(q, keys, v, rows)
            assert torch.equal(out.isnan(), want.isnan()), (part, name)
            fine = ~want.isnan()
            assert 0 < fine.sum() and (name == "high") == bool(fine.all())
            assert (out - want)[fine].norm() / want[fine].norm() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
    assert executor.last_status() == 0


@pytest.mark.parametrize("video, prefix, dim, cells, staged", [
    ((4, 20, 40), 77, 64, (0.0, 1.0, 0.0), False), ((9, 30, 52), 256, 128, (0.4, 0.4, 0.2), False),
    ((4, 20, 40), 512, 128, (0.0, 0.0, 1.0), False), ((4, 20, 40), 77, 64, (0.0, 1.0, 0.0), True),
    ((9, 30, 52), 300, 128, (0.0, 0.5, 0.5), False),    # left to torch
])
def test_counted_launches(native_library, video, prefix, dim, cells, staged):
    """A call with FP16 prefix queries counts the library's kernels, and none of torch's."""
    from anemoi_b200 import executor, native
    from tests.test_gpu_launch_count import _kernel_nodes

    tokens = prefix + video[0] * video[1] * video[2]
    q, k, v = (torch.randn(1, tokens, 6, dim, device="cuda").to(torch.bfloat16) for _ in range(3))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.8, retained_nvfp4_ratio=cells[0], retained_int8_ratio=cells[1],
              retained_fp16_ratio=cells[2], video_shape=video, layer=0, query_block_size=128, return_parts=staged,
              prefix_kv_precision="int8" if cells[1] else "fp16", prefix_query_precision="fp16",
              nvfp4_scales=(0.01, 0.01, 0.002))

    def kernels(f):
        f()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        before = native.launches_total()
        with torch.cuda.graph(graph):
            kept = f()
        del kept
        return native.launches_total() - before, _kernel_nodes(graph)

    counted, launched = kernels(lambda: executor.sm100_ragged_attention(q, k, v, **kw))
    foreign = 0
    if executor._library_prefix(False, prefix, tokens, dim):
        foreign = kernels(lambda: executor._library_rows(q, k, v, prefix))[1]
    assert counted == launched - foreign
