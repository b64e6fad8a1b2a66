"""How the recurrences over portions are launched: their few blocks walk a sequence's tokens for the whole of the kernel, and started
while the kernel before drains they pile up on the SMs that it leaves first. Read off the edges of a captured graph; so is that
single calls wait for the end of the call before."""
import ctypes

import pytest
import torch

from dryft_challenge_htn_2026_b200.csrc import api

pytestmark = pytest.mark.gpu
DEV = "cuda"
H, T = 2, 80


def f32(*shape):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(len(shape)), dtype=torch.float32).to(DEV) * 0.1


def i32(*v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def rows(portion):
    """(rows, cu_q, seq_pos0, seq_slot, sequences) of one portion of T tokens, or of T single tokens."""
    return (i32(0, T), i32(0), i32(0), 1) if portion else (None, torch.zeros(T, dtype=torch.int32, device=DEV),
                                                          torch.arange(T, dtype=torch.int32, device=DEV), T)


def linear(dtype, D, portion):
    cu, pos, slot, n = rows(portion)
    q, k, v = (f32(T, H * D).to(dtype) for _ in range(3))
    out, state, decay = f32(T, H * D), f32(T, H, D, D), torch.full((H,), 0.9, device=DEV)
    return lambda: api.linear_attention(q, k, v, out, state, cu, pos, slot, decay, n, H, D, D, T if portion else 1)


def gated(dtype, D, portion):
    cu, pos, slot, n = rows(portion)
    q, k, v = (f32(T, H * D).to(dtype) for _ in range(3))
    out, state, z, bias = f32(T, H * D), f32(T, H, D, D), f32(T, H * D), f32(H * D)
    return lambda: api.gated_linear_attention(q, k, v, out, state, cu, pos, slot, z, bias, 4.0, 1.0, n, H, D, D)


def given(dtype, D, portion):
    cu, pos, slot, n = rows(portion)
    q, k, v, decay = api.recurrence_operands(T, H * D, H * D, torch.device(DEV))
    q.normal_(), k.normal_(), v.normal_(), decay.fill_(0.9)
    out, state = f32(T, H * D), f32(T, H, D, D)
    return lambda: api.recurrence(q, k, decay, v, out, state, cu, pos, slot, n, H, D, D)


def memory(dtype, D, portion):
    cu, pos, slot, n = rows(portion)
    q, k, v, g = (f32(T, H * D).to(dtype) for _ in range(4))
    proj = f32(T, 2 * H).to(dtype)
    states, out = (f32(T, H, D, D), f32(T, H, D), f32(T, H)), torch.empty(T, H * D, dtype=dtype, device=DEV)
    row_pos = torch.arange(T, dtype=torch.int32, device=DEV)
    bias, w = f32(H), f32(H * D)
    buf = torch.cat([q, k, v, g, proj], 1).contiguous()
    cut = [buf[:, a:b] for a, b in ((0, H * D), (H * D, 2 * H * D), (2 * H * D, 3 * H * D), (3 * H * D, 4 * H * D),
                                    (4 * H * D, 4 * H * D + H), (4 * H * D + H, 4 * H * D + 2 * H))]
    return lambda: api.matrix_memory(*cut, bias, bias, 8.0, states, w, 1e-5, 1.0, out, 1.0, cu, pos, slot, row_pos, n, H, D, D)


class Edge(ctypes.Structure):
    """CUgraphEdgeData."""
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


PROGRAMMATIC = 1                                 # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC


def edges(graph):
    """[(from, to, whether the second may start before the first has ended)] of a captured graph."""
    get, n = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2, ctypes.c_size_t(0)
    graph = ctypes.c_void_p(graph)
    assert get(graph, None, None, None, ctypes.byref(n)) == 0
    start, end, data = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (Edge * n.value)()
    assert get(graph, start, end, data, ctypes.byref(n)) == 0
    return [(s, e, d.type == PROGRAMMATIC) for s, e, d in zip(start, end, data)]


def chain(call, steps):
    """For the kernels behind two small ones, in order: whether each may start before the one in front of it has ended."""
    h, a = f32(4, 64), torch.empty(4, 64, device=DEV)
    call()                                       # builds and sizes everything
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        if steps:
            with api.dependent_launches():
                api.cast_rows(h, a), api.cast_rows(h, a)
                call()
        else:
            api.cast_rows(h, a), api.cast_rows(h, a)
            call()
    after = {s: (e, early) for s, e, early in edges(graph.raw_cuda_graph())}
    assert len(after) == len(edges(graph.raw_cuda_graph()))      # one behind the other
    at, out = (set(after) - {e for e, _ in after.values()}).pop(), []
    while at in after:
        at, early = after[at]
        out.append(early)
    return out[0], out[1:]


OPS = [(linear, torch.float32, 24), (linear, torch.bfloat16, 64), (gated, torch.float32, 24), (gated, torch.bfloat16, 64),
       (gated, torch.float32, 128), (given, torch.float32, 24), (given, torch.float32, 64), (memory, torch.float32, 24),
       (memory, torch.bfloat16, 24)]


@pytest.mark.parametrize("op,dtype,D", OPS)
def test_a_recurrence_over_a_portion_starts_behind_the_end_of_the_kernel_before(op, dtype, D):
    first, kernels = chain(op(dtype, D, True), steps=True)
    assert first and kernels.count(False) == 1                  # the recurrence; gates, decays and norms around it start early
    assert all(chain(op(dtype, D, False), steps=True)[1])       # single tokens: all of them do


@pytest.mark.parametrize("op,dtype,D", OPS[:2])
def test_single_calls_wait_for_the_end_of_the_call_before(op, dtype, D):
    first, kernels = chain(op(dtype, D, True), steps=False)
    assert not first and not any(kernels)
