"""The draft map reads its key pools 16 bytes at a time: elsewhere they are refused.  Query pools may start anywhere."""

import ctypes as C

import pytest
import torch


def _shape(heads, blocks, dim, maxpool):
    from anemoi_b200 import native

    return native.Shape(heads=heads, head_dim=dim, query_block=128, seq_tokens=blocks * 128, prefix_tokens=0,
                        video_blocks=blocks, has_nvfp4=0, has_int8=1, has_fp16=0, has_prefix_query_int8=0,
                        has_maxpool=maxpool, input_is_bf16=1, q_global_scale=1.0, k_global_scale=1.0,
                        v_global_scale=1.0)


@pytest.mark.parametrize("weight, at, off", [
    (0.0, 1, 2), (0.0, 1, 8), (0.0, 0, 1), (0.0, 4, 1),
    (0.5, 1, 2), (0.5, 3, 8), (0.5, 2, 1), (1.0, 3, 2), (1.0, 2, 1),
])
def test_entry_point_refuses_misaligned_pointers(native_library, weight, at, off):
    """Refused on the host, before any launch (the addresses are never used)."""
    ptrs = [0x10000, 0x20000, 0x30000, 0x40000, 0x50000]      # mean q, k, max q, k, map
    ptrs[at] += off
    q, k, qx, kx, prob = (C.c_void_p(p) for p in ptrs)
    assert native_library.anemoi_sm100_draft_probability(_shape(2, 4, 64, int(weight != 0.0)), q, k, qx, kx, weight,
                                                         prob, None) == -1


@pytest.mark.parametrize("at, off", [(0, 1), (1, 2), (2, 1), (3, 8), (4, 1)])
def test_jensen_refuses_misaligned_pointers(native_library, at, off):
    ptrs = [0x10000, 0x20000, 0x30000, 0x40000, 0x50000]
    ptrs[at] += off
    q, k, q2, k2, prob = (C.c_void_p(p) for p in ptrs)
    assert native_library.anemoi_sm100_draft_probability_jensen(_shape(2, 4, 64, 2), q, k, q2, k2, prob, None) == -1


@pytest.mark.gpu
@pytest.mark.parametrize("heads, blocks, dim", [(3, 45, 64), (20, 300, 128), (3, 33, 128)])
@pytest.mark.parametrize("weight", [0.0, 0.5, 1.0])
def test_query_pools_that_start_anywhere(native_library, heads, blocks, dim, weight):
    """Contiguous query pools at any storage offset give the bits of aligned ones, through the operator;
    key pools off a boundary raise."""
    from anemoi_b200 import torch_ops

    torch_ops.load()
    gen = torch.Generator(device="cuda").manual_seed(blocks)
    q, k, qx, kx = ((torch.randn(heads, blocks, dim, generator=gen, device="cuda") * 0.5).half() for _ in range(4))

    def shifted(t, by):
        flat = torch.zeros(t.numel() + by, dtype=t.dtype, device=t.device)
        flat[by:] = t.reshape(-1)
        return flat[by:].view(t.shape)

    run = torch.ops.anemoi_sm100.draft_probability
    want = run(q, k, qx, kx, weight, 128)
    for by, byx in ((1, 0), (0, 3), (4, 4), (7, 8)):
        assert torch.equal(run(shifted(q, by), k, shifted(qx, byx), kx, weight, 128), want)
    keys = (k, shifted(kx, 4)) if weight == 1.0 else (shifted(k, 4), kx)
    with pytest.raises(RuntimeError):
        run(q, keys[0], qx, keys[1], weight, 128)
    assert torch.equal(run(q, k, qx, kx, weight, 128), want)
