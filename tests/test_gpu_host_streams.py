"""HostAttention called from several streams."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(seed=0):
    from anemoi_b200 import QuantConfig, SparseConfig, VisualLayout, anemoi_attention

    layout, heads = VisualLayout((3, 20, 30), 50), 6
    gen = torch.Generator().manual_seed(seed)
    shape = (1, layout.sequence_tokens, heads, 128)
    qkv = [torch.randn(shape, generator=gen).to(torch.bfloat16).pin_memory() for _ in range(3)]
    how = dict(layout=layout, layer=0, sparse_config=SparseConfig(128, 0.6), quant_config=QuantConfig(0.0, 0.5, 0.5))
    want = anemoi_attention(*(t.cuda() for t in qkv), **how).cpu()
    return qkv, torch.zeros_like(qkv[0]).pin_memory(), how, want


def _slowly(monkeypatch, cycles):
    """Each group's layer starts ``cycles`` late on its stream."""
    from anemoi_b200 import host

    layer = host.anemoi_attention

    def late(*args, **kw):
        torch.cuda._sleep(cycles)
        return layer(*args, **kw)

    monkeypatch.setattr(host, "anemoi_attention", late)


def test_runner_dropped_while_another_stream_computes(native_library, monkeypatch):
    """Buffers of the first call's stream, a second call on another stream, the runner dropped when its
    copies in are through and that stream's layers are not: the first stream must not get the memory."""
    from anemoi_b200 import HostAttention

    (q, k, v), out, how, want = _setup()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    runner = HostAttention("cuda", group_heads=4)
    with torch.cuda.stream(first):
        runner(q, k, v, out, **how)
    torch.cuda.synchronize()
    out.zero_()
    _slowly(monkeypatch, 100_000_000)            # some 50 ms
    with torch.cuda.stream(second):
        runner(q, k, v, out, **how)
    runner.copy_in.synchronize()
    sizes = [t.shape for buffers in runner._buffers.values() for t in buffers]
    del runner
    with torch.cuda.stream(first):
        taken = [torch.full(s, float("nan"), dtype=torch.bfloat16, device="cuda") for s in sizes]
    torch.cuda.synchronize()
    assert len(taken) == 6 and torch.equal(out, want)


def test_calls_from_two_streams_take_turns(native_library, monkeypatch):
    """A call from a second stream while the first one's layers wait: its copies in must not overwrite the
    slots that those layers still have to read."""
    from anemoi_b200 import HostAttention

    (q, k, v), out, how, want = _setup(1)
    (q2, k2, v2), out2, _, want2 = _setup(2)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    runner = HostAttention("cuda", group_heads=4)
    runner(q, k, v, out, **how)
    torch.cuda.synchronize()
    out.zero_()
    _slowly(monkeypatch, 50_000_000)
    with torch.cuda.stream(first):
        runner(q, k, v, out, **how)
    with torch.cuda.stream(second):
        runner(q2, k2, v2, out2, **how)
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(out2, want2)
