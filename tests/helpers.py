"""Shared builders for the parity tests: seeded synthetic NF4 weights plus their oracle views."""
from __future__ import annotations

import numpy as np
import torch

from aila_b200 import synth


def make_weight(seed, N, K, blocksize=64, nested=True):
    return synth.synth_linear(seed, N, K, blocksize, nested)


def oracle_absmax(O, w):
    """fp32 absmax as Bnb4BitLinear::init computes it (Bnb4BitLinear.cpp:472-488)."""
    if w.nested:
        return O.expand_absmax(w.absmax_codes, w.nested_quant_map, w.nested_absmax,
                               w.nested_blocksize, w.nested_offset)
    return np.asarray(w.absmax_f32, np.float32)


def bf16_bits(t: torch.Tensor) -> np.ndarray:
    return t.detach().cpu().contiguous().view(torch.uint16).numpy()


def from_bits(a: np.ndarray, device=None) -> torch.Tensor:
    t = torch.from_numpy(np.ascontiguousarray(a, np.uint16)).view(torch.bfloat16)
    return t.to(device) if device is not None else t


def bits_to_f32(a: np.ndarray) -> np.ndarray:
    return (np.ascontiguousarray(a, np.uint16).astype(np.uint32) << 16).view(np.float32)


def assert_close_norm(got_bits, want_bits, rel=2e-2, what=""):
    """max |err| <= rel * ||want||_inf : the acceptance bound for GEMV/GEMM outputs."""
    g, w = bits_to_f32(got_bits).astype(np.float64), bits_to_f32(want_bits).astype(np.float64)
    assert g.shape == w.shape, (g.shape, w.shape)
    assert np.isfinite(g).all(), f"{what}: non-finite output"
    err = np.abs(g - w).max() if g.size else 0.0
    bound = rel * (np.abs(w).max() if w.size else 0.0)
    assert err <= bound + 1e-30, f"{what}: max err {err:.4g} > {rel} * |y|inf = {bound:.4g}"
    return err, bound


def concat_rows(ws):
    """Row concatenation of quantised weights with fp32 absmax, as init_fused_rows does
    (Bnb4BitLinear.cpp:604-615). Returns (packed, absmax_f32_list_placeholder)."""
    return np.concatenate([np.asarray(w.packed, np.uint8).reshape(-1) for w in ws])


def captured(call, stream=None):
    """Captures call() in a CUDA graph: (mangled names of the kernels it launches, how many of them may start
    before the launch before has ended)."""
    from cuda.bindings import driver
    torch.cuda.synchronize()
    stream = stream or torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph, stream=stream):
            call()
    torch.cuda.synchronize()

    def ask(fn, *args):
        err, *rest = fn(*args)
        assert int(err) == 0, (fn.__name__, err)
        return rest
    raw = driver.CUgraph(graph.raw_cuda_graph())
    nodes, count = ask(driver.cuGraphGetNodes, raw, 1024)
    names = []
    for node in nodes[:count]:
        if ask(driver.cuGraphNodeGetType, node)[0] == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = ask(driver.cuGraphKernelNodeGetParams, node)[0]
            name = ask(driver.cuKernelGetName, params.kern) if int(params.kern) else ask(driver.cuFuncGetName, params.func)
            names.append(name[0].decode())
    edges, count = ask(driver.cuGraphGetEdges_v2, raw, 1024)[2:]
    programmatic = int(driver.CUgraphDependencyType.CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC)
    return names, sum(int(e.type) == programmatic for e in edges[:count])
