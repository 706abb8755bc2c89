"""The side stream of FP16 prefix rows is nobody else's."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_not_of_the_callers_streams(native_library):
    from anemoi_b200 import HostAttention, executor

    device = torch.device("cuda", torch.cuda.current_device())
    side = executor._dense_stream(device)
    assert side.device == device and side is executor._dense_stream(device)
    runner = HostAttention(device)
    others = [torch.cuda.Stream(device) for _ in range(70)] + [runner.copy_in, runner.copy_out]
    assert side.cuda_stream not in {s.cuda_stream for s in others} | {0, torch.cuda.current_stream(device).cuda_stream}


def test_no_wait_for_the_default_stream(native_library):
    """It runs beside the default stream, as torch's own do, and is ordered by events."""
    from anemoi_b200 import executor

    device = torch.device("cuda", torch.cuda.current_device())
    side = executor._dense_stream(device)
    x = torch.zeros(1 << 20, device=device)
    x += 0    # (a kernel's first use may wait for all streams)
    torch.cuda._sleep(1)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)    # some 100 ms of the default stream
    held = torch.cuda.Event()
    held.record()
    with torch.cuda.stream(side):
        x += 1
        done = torch.cuda.Event()
        done.record()
    done.synchronize()
    assert not held.query()
    torch.cuda.current_stream(device).wait_stream(side)
    assert (x == 1).all()
