"""A set status word and dense rows: every CTA of a cluster leaves, and the next call finds nothing amiss."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens, rows, parts", [(700, 200, 1), (2_500, 130, 2), (9_000, 70, 4), (16_500, 129, 4), (16_500, 100, 8)])
@pytest.mark.parametrize("dim, dtype", [(64, torch.float16), (128, torch.bfloat16)])
def test_set_word_leaves_the_output_alone(native_library, tokens, rows, parts, dim, dtype):
    """Set, no row is written and the word is kept; clear, the same launch gives the rows."""
    import ctypes as C

    from anemoi_b200 import native

    assert native_library.anemoi_sm100_dense_parts(tokens, rows) == parts
    heads = 3
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    q, k, v = (torch.randn(1, tokens, heads, dim, generator=gen, device="cuda").to(dtype) for _ in range(3))
    status = torch.full((1,), 5, dtype=torch.int32, device="cuda")
    out = torch.full((heads, rows, dim), -7.0, dtype=dtype, device="cuda")
    strides = (C.c_int64 * 6)(*(heads * dim, dim) * 3)

    def launch():
        code = native_library.anemoi_sm100_dense_rows(
            heads, dim, tokens, rows, int(dtype == torch.bfloat16), q.data_ptr(), k.data_ptr(), v.data_ptr(), strides,
            out.data_ptr(), dim, rows * dim, status.data_ptr(), native._stream(q.device))
        assert code == 0
        torch.cuda.synchronize()

    launch()
    assert (out == -7.0).all() and int(status.item()) == 5
    status.zero_()
    launch()
    scores = torch.einsum("bqhd,bkhd->bhqk", q[:, :rows].double(), k.double()) / dim ** 0.5
    want = torch.einsum("bhqk,bkhd->bhqd", scores.softmax(-1), v.double())[0]
    # probabilities and results rounded once each (bf16: 2^-9, fp16: 2^-12 at most)
    assert (out.double() - want).norm() / want.norm() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
    assert int(status.item()) == 0
