"""Dense rows of the caller's tensors (prefix queries kept out of the cells) against 64 bits."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _tensors(layout, tokens, heads, dim, dtype, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if layout == "packed":      # the strided views of an exchange's buffer
        return torch.randn(1, tokens, heads, 3 * dim, generator=gen, device="cuda").to(dtype).split(dim, dim=3)
    if layout == "head_major":  # [H][S][D] in memory
        return tuple(torch.randn(1, heads, tokens, dim, generator=gen, device="cuda").to(dtype).transpose(1, 2)
                     for _ in range(3))
    if layout == "padded":      # tokens further apart than heads x channels, values not where keys are
        return tuple(torch.randn(1, tokens, heads + n, dim + 8 * n, generator=gen, device="cuda").to(dtype)
                     [:, :, :heads, :dim] for n in (1, 0, 2))
    return tuple(torch.randn(1, tokens, heads, dim, generator=gen, device="cuda").to(dtype) for _ in range(3))


def _dense(q, k, v, rows):
    scores = torch.einsum("bqhd,bkhd->bhqk", q[:, :rows].double(), k.double()) / q.size(3) ** 0.5
    return torch.einsum("bhqk,bkhd->bhqd", scores.softmax(-1), v.double())[0]


# lengths on both sides of a stage's end and of every rule of the parts (32, 96 and 256 stages), rows of a tile's
@pytest.mark.parametrize("tokens, rows", [(2, 1), (63, 62), (64, 64), (65, 1), (31 * 64, 127), (32 * 64, 128), (95 * 64 + 1, 129),
                                          (96 * 64 + 63, 300), (255 * 64, 40), (255 * 64 + 1, 257), (20_001, 1_000)])
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("layout, dtype, heads", [("contiguous", torch.bfloat16, 1), ("packed", torch.float16, 3),
                                                  ("head_major", torch.bfloat16, 2), ("padded", torch.float16, 2)])
def test_rows(native_library, tokens, rows, dim, layout, dtype, heads):
    from anemoi_b200 import executor, native

    q, k, v = _tensors(layout, tokens, heads, dim, dtype, tokens)
    status = executor._status_word(q.device)
    out = native.dense_rows(q, k, v, rows, status)
    want = _dense(q, k, v, rows)
    # probabilities and results rounded once each (bf16: 2^-9, fp16: 2^-12 at most)
    assert (out.double() - want).norm() / want.norm() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -11)
    for h in range(heads):  # a head's rows do not depend on the others
        assert torch.equal(native.dense_rows(*(t[:, :, h:h + 1] for t in (q, k, v)), rows, status)[0], out[h])
    assert executor.last_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_infinities_and_nans(native_library, dtype):
    """A key of infinities: rows whose score is -inf have no weight there, those of +inf are NaN, as of softmax; a NaN
    query is its own row's; rows without any score above -inf are NaN."""
    from anemoi_b200 import executor, native

    tokens, rows, heads, dim = 700, 200, 2, 64
    q, k, v = _tensors("contiguous", tokens, heads, dim, dtype, 1)
    k[:, 333, :, 5] = float("inf")
    q[:, 7] = float("nan")
    out = native.dense_rows(q, k, v, rows, executor._status_word(q.device)).double()
    want = _dense(q, k, v, rows)
    assert torch.equal(out.isnan(), want.isnan()) and 0 < want.isnan().sum() < want.numel()
    fine = ~want.isnan()
    assert (out - want)[fine].norm() / want[fine].norm() < 2 ** -8
    k[..., 5] = float("inf")
    q[:, :rows, :, 5] = -1.0
    assert native.dense_rows(q, k, v, rows, executor._status_word(q.device)).isnan().all()
    assert executor.last_status() == 0


def test_refusals(native_library):
    from anemoi_b200 import executor, native

    q, k, v = _tensors("contiguous", 100, 2, 64, torch.float16, 1)
    out = torch.empty(2, 10, 64, dtype=torch.float16, device="cuda")
    status = executor._status_word(q.device)
    good = dict(heads=2, dim=64, tokens=100, rows=10, q=q.data_ptr(), strides=(128, 64) * 3, out=out.data_ptr(), out_token=64)

    def call(**other):
        a = dict(good, **other)
        strides = (C.c_int64 * 6)(*a["strides"])
        return native.library().anemoi_sm100_dense_rows(
            a["heads"], a["dim"], a["tokens"], a["rows"], 0, a["q"], k.data_ptr(), v.data_ptr(), strides, a["out"],
            a["out_token"], 640, status.data_ptr(), torch.cuda.current_stream().cuda_stream)

    assert call() == 0
    for other in (dict(rows=0), dict(rows=101), dict(dim=96), dict(heads=0), dict(q=None), dict(q=q.data_ptr() + 8),
                  dict(out=out.data_ptr() + 2), dict(out_token=60), dict(strides=(128, 0) * 3),
                  dict(strides=(-128, 64) * 3), dict(strides=(132, 64) * 3)):
        assert call(**other) == -1, other
    torch.cuda.synchronize()
