"""The launches that are counted for a call are the kernels that it puts on the stream."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernel_nodes(graph) -> int:
    runtime = C.CDLL("libcudart.so.12")
    handle, count = C.c_void_p(graph.raw_cuda_graph()), C.c_size_t()
    assert runtime.cudaGraphGetNodes(handle, None, C.byref(count)) == 0
    nodes, kind, kernels = (C.c_void_p * count.value)(), C.c_int(), 0
    assert runtime.cudaGraphGetNodes(handle, nodes, C.byref(count)) == 0
    for node in nodes:
        assert runtime.cudaGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        kernels += kind.value == 0    # cudaGraphNodeTypeKernel
    return kernels


@pytest.mark.parametrize("video, prefix, heads, query_block, cells, maxpool", [
    ((4, 8, 32), 0, 4, 64, (0.0, 1.0, 0.0), 0.0),       # the CTAs of values find the maxima; the map in the routing
    ((1, 48, 84), 77, 8, 128, (0.0, 0.5, 0.5), 0.5),    # the maxima start at zero by a kernel
    ((1, 25, 40), 0, 40, 64, (0.0, 1.0, 0.0), 0.0),     # the maxima by clusters
    ((9, 30, 52), 0, 4, 64, (1.0, 0.0, 0.0), 0.0),      # no maxima
    ((200, 8, 8), 20, 10, 64, (0.0, 1.0, 0.0), 0.0),    # pairs are chosen
    ((1025, 8, 8), 0, 1, 64, (0.0, 1.0, 0.0), 0.0),     # and routing takes several kernels
    ((1025, 8, 8), 0, 1, 64, (0.0, 0.5, 0.5), 0.0),     # neighbours
    ((1025, 8, 16), 30, 1, 128, (0.4, 0.4, 0.2), 0.0),
])
def test_counted_launches(native_library, video, prefix, heads, query_block, cells, maxpool):
    from anemoi_b200 import executor, native

    tokens = prefix + video[0] * video[1] * video[2]
    q, k, v = (torch.randn(1, tokens, heads, 64, device="cuda").to(torch.bfloat16) for _ in range(3))
    kw = dict(prefix_tokens=prefix, sparsity_ratio=0.8, retained_nvfp4_ratio=cells[0], retained_int8_ratio=cells[1],
              retained_fp16_ratio=cells[2], video_shape=video, layer=0, query_block_size=query_block, maxpool_weight=maxpool,
              prefix_kv_precision="int8" if cells[1] else "nvfp4", nvfp4_scales=(0.01, 0.01, 0.002))
    executor.sm100_ragged_attention(q, k, v, **kw)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    before = native.launches_total()
    with torch.cuda.graph(graph):
        executor.sm100_ragged_attention(q, k, v, **kw)
    assert native.launches_total() - before == _kernel_nodes(graph)
