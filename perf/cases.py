"""The workloads this library's speed is judged on, as a user's program meets them.

Three public entry points carry the work: ``anemoi_attention`` (one sparse mixed-precision layer
on the device), ``HostAttention`` (the same layer for Q/K/V in pinned host memory) and
``fused_qknorm_rope`` (the producer step on Q and K in front of it).  The listed cases go from one
call over a thousand tokens, where latency counts, to the 85,184-token, 56-head layer the benchmark
is quoted on; ``draw`` gives more of the same ranges: 1-40 frames of ragged sizes with or without
a packed prefix, 1-56 heads, both head dims, query blocks and data types, every mix of the
precision cells, 50-90 % dropped blocks and the three draft maps.
"""

from __future__ import annotations

import math

import torch

from anemoi_b200 import NVFP4Calibration, QuantConfig, SparseConfig, VisualLayout, anemoi_attention
from anemoi_b200.host import HostAttention
from anemoi_b200.producer import fused_qknorm_rope

_MOST_PAIRS = 85_184 ** 2 * 56 * 128 * 0.2    # dot products of the largest listed layer, dense share
_MOST_VALUES = 85_184 * 56 * 128              # values of one of its tensors


def _layer(name, video, prefix, heads, dim, dtype, query_block, drop, cells, *, maxpool=0.0,
           prefix_kv="int8", prefix_query="int8", packed=False, path="attention"):
    case = dict(path=path, frames=video[0], height=video[1], width=video[2], prefix=prefix, heads=heads, dim=dim,
                dtype=dtype, query_block=query_block, drop=drop, nvfp4=cells[0], int8=cells[1], fp16=cells[2],
                maxpool=maxpool, prefix_kv=prefix_kv, prefix_query=prefix_query, packed=packed)
    return dict(case, name=name) if name else case


def _producer(name, tokens, heads, dim, dtype, rotary):
    case = dict(path="producer", tokens=tokens, heads=heads, dim=dim, dtype=dtype, rotary=rotary)
    return dict(case, name=name) if name else case


def listed():
    return [
        # a preview-sized call with the default configuration: a thousand tokens, latency only
        _layer("preview_1k_q64", (4, 16, 16), 0, 4, 64, "float16", 64, 0.8, (0.0, 1.0, 0.0)),
        # one image with a short prompt in front of it, as a still-frame request sends it
        _layer("image_q128", (1, 48, 84), 77, 8, 128, "bfloat16", 128, 0.8, (0.0, 0.5, 0.5), maxpool=0.5),
        # odd everything: ragged frames, odd prefix, odd head count, small heads, all three cells
        _layer("ragged_d64_mixed", (13, 27, 45), 333, 5, 64, "float16", 64, 0.7, (0.4, 0.4, 0.2)),
        # prefix queries and a whole layer kept in FP16 (the cautious setting of a quality check)
        _layer("fp16_cells", (9, 30, 52), 256, 16, 128, "bfloat16", 64, 0.8, (0.0, 0.0, 1.0),
               prefix_kv="fp16", prefix_query="fp16"),
        # visual-only NVFP4 layer at the large video shape, max-pooled draft map: the kernel sweep's point
        _layer("sweep_nvfp4_d64", (21, 48, 84), 0, 4, 64, "bfloat16", 128, 0.9, (1.0, 0.0, 0.0), maxpool=1.0),
        # one rank's share (7 of 56 heads) of the 832x480 layer after the sequence<->head exchange, on the
        # strided q|k|v views of its receive buffer
        _layer("rank_share_832x480", (21, 30, 52), 512, 7, 128, "bfloat16", 128, 0.8, (0.0, 0.5, 0.5),
               maxpool=0.5, packed=True),
        # the same share of the 1344x768 layer
        _layer("rank_share_1344x768", (21, 48, 84), 512, 7, 128, "bfloat16", 128, 0.8, (0.4, 0.4, 0.2), packed=True),
        # the model adapter's default request: Q64 blocks, INT8 cells, 951-token prefix
        _layer("adapter_default_q64", (37, 24, 42), 951, 56, 128, "bfloat16", 64, 0.8, (0.0, 1.0, 0.0)),
        # the whole 832x480 layer on one GPU
        _layer("layer_832x480", (21, 30, 52), 512, 56, 128, "bfloat16", 128, 0.8, (0.0, 0.5, 0.5), maxpool=0.5),
        # the whole 1344x768 layer on one GPU (the benchmark's configuration)
        _layer("layer_1344x768", (21, 48, 84), 512, 56, 128, "bfloat16", 128, 0.8, (0.4, 0.4, 0.2)),
        # a layer whose Q/K/V and output live in pinned host memory
        _layer("host_832x480", (21, 30, 52), 512, 16, 128, "bfloat16", 128, 0.8, (0.4, 0.4, 0.2), path="host"),
        # qk-norm and partial rotary on Q and K of a layer, in place
        _producer("producer_832x480", 33_272, 56, 128, "bfloat16", 64),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.random()
    dtype = rng.choice(("bfloat16", "bfloat16", "float16"))
    dim = rng.choice((128, 128, 64))
    if kind < 0.1:
        heads = _log(rng, 1, 56)
        tokens = min(_log(rng, 500, 85_000), _MOST_VALUES // (heads * dim) // 2)
        return _producer(None, tokens, heads, dim, dtype, rng.choice((32, 64)))
    path = "host" if kind < 0.2 else "attention"
    query_block = rng.choice((64, 128))
    cells = rng.choice(((0.0, 1.0, 0.0), (1.0, 0.0, 0.0), (0.0, 0.0, 1.0), (0.0, 0.5, 0.5), (0.5, 0.5, 0.0),
                        (0.4, 0.4, 0.2), (0.3, 0.3, 0.4)))
    active = [name for name, share in zip(("nvfp4", "int8", "fp16"), cells) if share]
    prefix = rng.choice((0, _log(rng, 20, 1_000)))
    prefix_query = "int8" if "int8" in active and rng.random() < 0.85 else "fp16"
    drop = rng.choice((0.5, 0.8, 0.8, 0.9))
    maxpool = rng.choice((0.0, 0.0, 0.5, 1.0))
    while True:
        # frames, frame sizes and heads over their whole range, until the call is no larger than the largest listed
        video = (_log(rng, 1, 40), _log(rng, 12, 60), _log(rng, 12, 90))
        heads = _log(rng, 1, 56) if path == "attention" else _log(rng, 4, 24)
        tokens = math.prod(video) + prefix
        dense = (1.0 - drop) + 2.0 * prefix / tokens
        blocks = math.prod(video) / query_block
        if 1_000 <= tokens <= 86_000 and blocks <= 1_600 and tokens ** 2 * heads * dim * dense <= _MOST_PAIRS \
                and (path == "attention" or tokens * heads * dim <= 1 << 27):
            break
    return _layer(None, video, prefix, heads, dim, dtype, query_block, drop, cells, maxpool=maxpool,
                  prefix_kv=rng.choice(active), prefix_query=prefix_query,
                  packed=path == "attention" and rng.random() < 0.3, path=path)


def _blur(n, device):
    """Gaussian blur (sigma 2) over an axis of ``n`` tokens with reflected ends, as a matrix."""
    radius = min(6, n - 1)
    taps = torch.exp(-0.5 * (torch.arange(-radius, radius + 1, dtype=torch.float32) / 2.0) ** 2)
    taps = taps / taps.sum()
    m = torch.zeros(n, n)
    for i in range(n):
        for t in range(-radius, radius + 1):
            j = abs(i + t)
            m[i, 2 * (n - 1) - j if j > n - 1 else j] += taps[t + radius]
    return m.to(device)


def _field(case, gen, dtype, out):
    """Q or K: N(0,1) smoothed over each frame plus half as much noise, two loud channels in bf16
    (prefix rows and the layout as the model's activations have them)."""
    f, h, w, prefix, heads, dim = (case[k] for k in ("frames", "height", "width", "prefix", "heads", "dim"))
    device = out.device
    rows, cols = _blur(h, device), _blur(w, device)
    out[:prefix] = torch.randn(prefix, heads, dim, generator=gen, device=device).to(dtype)
    video = out[prefix:].view(f, h, w, heads, dim) if out.is_contiguous() else None
    step = max(1, (1 << 27) // (f * h * w * dim))
    for h0 in range(0, heads, step):
        n = min(step, heads - h0)
        x = torch.randn(f, h, w * n * dim, generator=gen, device=device)
        x = torch.matmul(rows, x).view(f * h, w, n * dim)
        x = torch.matmul(cols, x)
        x += 0.5 * torch.randn(f * h, w, n * dim, generator=gen, device=device)
        x = x.view(f, h, w, n, dim)
        if dtype == torch.bfloat16:
            x[..., 17] *= 8.0
            x[..., dim - 35] *= 8.0
        if video is not None:
            video[:, :, :, h0:h0 + n] = x.to(dtype)
        else:
            out[prefix:, h0:h0 + n] = x.reshape(f * h * w, n, dim).to(dtype)


def _qkv(case, seed):
    device = torch.device("cuda")
    dtype = getattr(torch, case["dtype"])
    gen = torch.Generator(device=device).manual_seed(seed)
    heads, dim = case["heads"], case["dim"]
    tokens = case["prefix"] + case["frames"] * case["height"] * case["width"]
    if case["packed"]:
        buffer = torch.empty(tokens, heads, 3 * dim, dtype=dtype, device=device)
        q, k, v = buffer.split(dim, dim=2)
    else:
        q, k, v = (torch.empty(tokens, heads, dim, dtype=dtype, device=device) for _ in range(3))
    _field(case, gen, dtype, q)
    _field(case, gen, dtype, k)
    step = max(1, (1 << 28) // (heads * dim))
    for t in range(0, tokens, step):
        part = v[t:t + step]
        part.copy_(torch.randn(part.shape, generator=gen, device=device).to(dtype))
    return q.unsqueeze(0), k.unsqueeze(0), v.unsqueeze(0)


def prepare(case, seed):
    device = torch.device("cuda")
    dtype = getattr(torch, case["dtype"])
    if case["path"] == "producer":
        gen = torch.Generator(device=device).manual_seed(seed)
        shape = (1, case["tokens"], case["heads"], case["dim"])
        q, k = (torch.randn(shape, generator=gen, device=device).to(dtype) for _ in range(2))
        wq, wk = ((1.0 + 0.05 * torch.randn(case["dim"], generator=gen, device=device)).to(dtype) for _ in range(2))
        half = case["rotary"] // 2
        speed = 10_000.0 ** (-torch.arange(half, device=device, dtype=torch.float32) / half)
        angle = torch.arange(case["tokens"], device=device, dtype=torch.float32)[:, None] * speed
        angle = torch.cat((angle, angle), dim=1)
        return dict(path="producer", q=q, k=k, wq=wq, wk=wk, cos=angle.cos(), sin=angle.sin())
    q, k, v = _qkv(case, seed)
    scales = None
    if case["nvfp4"] > 0 or (case["prefix"] and case["prefix_kv"] == "nvfp4"):
        # per-layer scales come out of a calibration pass, long before the call
        scales = NVFP4Calibration(*(float(t.abs().amax()) / (6 * 448) for t in (q, k, v)))
    state = dict(
        path=case["path"], layout=VisualLayout((case["frames"], case["height"], case["width"]), case["prefix"]),
        sparse=SparseConfig(case["query_block"], case["drop"], (), case["maxpool"]),
        quant=QuantConfig(case["nvfp4"], case["int8"], case["fp16"], case["prefix_kv"], case["prefix_query"]),
        scales=scales)
    if case["path"] == "host":
        host = []
        for t in (q, k, v):
            pinned = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
            pinned.copy_(t)
            host.append(pinned)
        state.update(q=host[0], k=host[1], v=host[2], out=torch.empty(q.shape, dtype=dtype, pin_memory=True),
                     call=HostAttention(device))
    else:
        state.update(q=q, k=k, v=v)
    return state


def run(state):
    if state["path"] == "producer":
        q = fused_qknorm_rope(state["q"], state["wq"], state["cos"], state["sin"], 1e-6)
        k = fused_qknorm_rope(state["k"], state["wk"], state["cos"], state["sin"], 1e-6)
        return q, k
    how = dict(layout=state["layout"], layer=0, sparse_config=state["sparse"], quant_config=state["quant"],
               calibration=state["scales"])
    if state["path"] == "host":
        return state["call"](state["q"], state["k"], state["v"], state["out"], **how)
    return anemoi_attention(state["q"], state["k"], state["v"], **how)


def work(case):
    heads, dim = case["heads"], case["dim"]
    if case["path"] == "producer":
        values = case["tokens"] * heads * dim
        return {"bytes": 2 * 2 * 2 * values + 2 * 4 * case["tokens"] * case["rotary"], "flops": 2 * 8 * values}
    video = case["frames"] * case["height"] * case["width"]
    tokens = video + case["prefix"]
    # kept pairs of video tokens, video rows against the prefix, prefix rows against everything; QK and PV
    pairs = (1.0 - case["drop"]) * video * video + video * case["prefix"] + case["prefix"] * tokens
    return {"bytes": 4 * 2 * tokens * heads * dim, "flops": 4 * dim * heads * pairs}


def tolerance(case):
    if case["path"] == "producer":
        return {"rel": 2e-3}    # one rounding to 16 bits; the sums inside are fp32
    # probabilities are rounded to e2m1 in the NVFP4 cell, to e4m3 or fp16 in the others
    return {"rel": 2e-2} if case["nvfp4"] > 0 else {"rel": 1e-2}
