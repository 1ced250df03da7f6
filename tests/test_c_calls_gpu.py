"""Calls of the C library in forms that the Python entry points do not produce."""

import ctypes

import pytest
import torch

from selective_attention_b200 import _lib, kernels, mixers

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _problem(q, k, v):
    return kernels._problem(q, k, v, _lib.ENGINE_TCGEN05, 1)


@pytest.mark.parametrize("heads,dim", [(1, 64), (3, 64), (1, 128), (3, 128)])
def test_backward_writes_gradients_at_any_element(heads, dim):
    """dq, dk and dv of the plain backward are contiguous; where they begin is the caller's affair."""
    lib = _lib.load()
    g = torch.Generator("cpu").manual_seed(dim + heads)
    b, t = 2, 200
    q, k, v, d_out = (torch.randn(b, heads, t, dim, generator=g).bfloat16().cuda() for _ in range(4))
    out, lse2, carry, *_ = kernels._forward(q, k, v, True, 1, 0, 0)
    p = _problem(q, k, v)
    need = lib.sa_backward_workspace_bytes(ctypes.byref(p))
    workspace = torch.empty(need, dtype=torch.uint8, device="cuda")
    n = q.numel()
    got = []
    for first in (8, 9, 11, 12):                   # elements of 2 bytes: at 16, 2, 6 and 8 bytes of a boundary
        flat = [torch.full((n + 32,), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
        ptrs = [x.data_ptr() + 2 * first for x in flat]
        _lib.check("sa_backward", lib.sa_backward(ctypes.byref(p), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                                                  lse2.data_ptr(), carry.data_ptr(), d_out.data_ptr(), _lib.DTYPE_BF16, *ptrs,
                                                  workspace.data_ptr(), need, _stream()))
        torch.cuda.synchronize()
        for x in flat:
            assert (x[:first] == 7).all() and (x[first + n:] == 7).all()
        got.append([x[first:first + n].float() for x in flat])
    assert _lib.device_status() == 0
    for other in got[1:]:
        for a, ref in zip(other, got[0]):
            assert float((a - ref).norm() / ref.norm()) < 2e-3         # the order of the fp32 reductions


def _pointer_arguments(driver, node):
    """The 8-byte arguments of a graph's kernel node."""
    err, params = driver.cuGraphKernelNodeGetParams(node)
    assert err == 0
    values = ctypes.cast(params.kernelParams, ctypes.POINTER(ctypes.c_void_p))
    found, i = [], 0
    while True:
        err, _, size = driver.cuFuncGetParamInfo(params.func, i)
        if err != 0:
            return found
        if size == 8:
            found.append(ctypes.cast(values[i], ctypes.POINTER(ctypes.c_uint64))[0])
        i += 1


@pytest.mark.parametrize("heads,dim,per_head,skip", [(2, 64, False, False), (2, 64, True, True), (160, 64, False, True), (2, 128, False, False)])
def test_the_history_of_a_cache_moves_on_last(heads, dim, per_head, skip):
    """A chunk whose call fails must not leave its selection behind, or trying again would count it twice: nothing but the last
    launch of the call is given the history to write."""
    driver = pytest.importorskip("cuda.bindings.driver")
    g = torch.Generator("cpu").manual_seed(3)
    first, total = 300, 330
    q, k, v = (torch.randn(1, heads, total, dim, generator=g).bfloat16().cuda() for _ in range(3))
    slot = mixers.SelectiveAttentionSlot(n_heads=heads, context_length=total, per_head=per_head)
    _, cache = slot.begin_cache(*(x[:, :, :first] for x in (q, k, v)))
    new = [x[:, :, first:] for x in (q, k, v)]
    want = {key: (x.clone() if torch.is_tensor(x) else x) for key, x in cache.items()}
    slot.extend_cache(*new, want, skip_dead_tiles=skip)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        slot.extend_cache(*new, cache, skip_dead_tiles=skip)
    raw = driver.CUgraph(graph.raw_cuda_graph())
    nodes = {int(n): n for n in driver.cuGraphGetNodes(raw, driver.cuGraphGetNodes(raw)[2])[1]}
    _, sources, targets, *_ = driver.cuGraphGetEdges(raw, driver.cuGraphGetEdges(raw)[-1])
    follows = {int(a): int(b) for a, b in zip(sources, targets)}
    node = next(n for n in nodes if n not in set(follows.values()))
    order = [node]
    while node in follows:
        order.append(node := follows[node])
    assert len(order) == len(nodes)                             # one stream: a chain
    kernel, copy = driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL, driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_MEMCPY
    types = [driver.cuGraphNodeGetType(nodes[n])[1] for n in order]
    history = cache["selected"].data_ptr()
    given = sum(_pointer_arguments(driver, nodes[n]).count(history) for n, kind in zip(order, types) if kind == kernel)
    assert given == 1                                           # the scan reads it
    assert types[-1] == copy and int(driver.cuGraphMemcpyNodeGetParams(nodes[order[-1]])[1].dstDevice) == history
    graph.replay()
    assert torch.equal(cache["selected"], want["selected"])
