"""The producer reads and writes 16 bytes at a time: what starts elsewhere is refused or copied."""

import ctypes as C

import pytest
import torch


def test_entry_point_refuses_misaligned_pointers(native_library):
    """Refused on the host, before any launch (the addresses are never used)."""
    strides = (C.c_int64 * 2)(256, 128)
    good = [0x10000, 0x20000, 0x30000, 0x40000]
    for at, off in ((0, 2), (0, 8), (1, 2), (2, 4), (3, 8)):
        ptrs = list(good)
        ptrs[at] += off
        code = native_library.anemoi_sm100_qknorm_rope(*(C.c_void_p(p) for p in ptrs), 4, 2, 128, 64, 1e-6, 1, strides,
                                                       None)
        assert code == -1


def test_tensors_elsewhere_are_refused():
    from anemoi_b200.producer import fused_qknorm_rope

    x, table = torch.zeros(1, 4, 2, 128, dtype=torch.bfloat16), torch.zeros(4, 64)
    with pytest.raises(ValueError):
        fused_qknorm_rope(x, torch.ones(128, dtype=torch.bfloat16), table, table, 1e-6)


@pytest.mark.gpu
def test_slices_that_start_anywhere(native_library):
    """Weights and tables that are slices of larger tensors give the same bits; an x that is one is refused,
    as is a weight on the host."""
    from anemoi_b200.producer import fused_qknorm_rope

    gen = torch.Generator(device="cuda").manual_seed(1)

    def shifted(t, by):
        flat = torch.zeros(t.numel() + by, dtype=t.dtype, device=t.device)
        flat[by:] = t.reshape(-1)
        return flat[by:].view(t.shape)

    x = torch.randn(1, 9, 5, 128, generator=gen, device="cuda").to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(128, generator=gen, device="cuda")).to(torch.bfloat16)
    cos, sin = torch.randn(2, 9, 64, generator=gen, device="cuda")
    want = fused_qknorm_rope(x.clone(), w, cos, sin, 1e-6)
    for args in ((shifted(w, 1), cos, sin), (w, shifted(cos, 1), sin), (w, cos, shifted(sin, 2)),
                 (shifted(w, 4), shifted(cos, 3), shifted(sin, 3))):
        assert torch.equal(fused_qknorm_rope(x.clone(), *args, 1e-6), want)
    with pytest.raises(RuntimeError):
        fused_qknorm_rope(shifted(x, 4), w, cos, sin, 1e-6)
    with pytest.raises(ValueError):
        fused_qknorm_rope(x.clone(), w.cpu(), cos, sin, 1e-6)
