"""Helpers shared by the tests: bit views, seeded inputs, numpy bridges."""
from __future__ import annotations

import ctypes

import numpy as np
import torch


def u8(t: torch.Tensor) -> torch.Tensor:
    return t.contiguous().view(torch.uint8)


def to_np_f32(t: torch.Tensor) -> np.ndarray:
    """Exact widening of a float tensor to a numpy fp32 array."""
    return t.detach().float().cpu().numpy()


def codes_np(t: torch.Tensor) -> np.ndarray:
    return u8(t).cpu().numpy()


def from_bits16(bits: np.ndarray, dtype=torch.bfloat16) -> torch.Tensor:
    return torch.from_numpy(bits.view(np.int16).copy()).view(dtype)


def from_bits32(bits: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(bits.view(np.int32).copy()).view(torch.float32)


def f32_bits(t: torch.Tensor) -> int:
    return int(t.detach().float().cpu().view(torch.int32).reshape(-1)[0].item()) & 0xFFFFFFFF


def randn_cpu(shape, seed, dtype=torch.bfloat16, scale=1.0) -> torch.Tensor:
    """Seeded on the CPU so that CPU and GPU arms see identical bits."""
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g, dtype=torch.float32) * scale).to(dtype)


def config1_inputs(seed: int = 0):
    """BASELINE config 1 inputs, generated exactly as tests/golden/make_golden.py does."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(8, 4096, generator=g, dtype=torch.float32)
    mask = torch.rand(8, 4096, generator=g) < 1e-3
    x = torch.where(mask, x * 50.0, x).to(torch.bfloat16)
    w = (torch.randn(4096, 4096, generator=g, dtype=torch.float32) * 0.02).to(torch.bfloat16)
    return x, w


def max_rel(y: torch.Tensor, ref: torch.Tensor) -> float:
    y, ref = y.double(), ref.double()
    return float((y - ref).abs().max() / ref.abs().max().clamp_min(1e-300))


def captured_kernels(fn):
    """The kernels that `fn()` launches, captured and not run: per kernel its (mangled) name, CTAs, threads and CTAs per cluster; and how
    many of the edges between them are programmatic."""
    from cuda.bindings import driver

    def ok(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:] if len(result) > 2 else result[1]

    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    handle = driver.CUgraph(graph.raw_cuda_graph())
    nodes, _ = ok(driver.cuGraphGetNodes(handle, ok(driver.cuGraphGetNodes(handle))[1]))
    found = []
    for node in nodes:
        if ok(driver.cuGraphNodeGetType(node)) != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        params = ok(driver.cuGraphKernelNodeGetParams(node))
        name = ok(driver.cuFuncGetName(params.func)) if int(params.func) else ok(driver.cuKernelGetName(params.kern))
        cluster = ok(driver.cuGraphKernelNodeGetAttribute(node, driver.CUlaunchAttributeID.CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION))
        found.append({"name": name.decode(), "ctas": params.gridDimX * params.gridDimY, "threads": params.blockDimX,
                      "cluster": cluster.clusterDim.x})
    # cuda-python hands out edge data that it has freed
    libcuda, n = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t(len(nodes) ** 2)
    ends = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)()
    data = (ctypes.c_uint8 * (8 * n.value))()         # from port, to port, type, five reserved
    assert libcuda.cuGraphGetEdges_v2(ctypes.c_void_p(graph.raw_cuda_graph()), *ends, data, ctypes.byref(n)) == 0
    programmatic = sum(data[8 * i + 2] == int(driver.CUgraphDependencyType.CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC) for i in range(n.value))
    return found, programmatic
