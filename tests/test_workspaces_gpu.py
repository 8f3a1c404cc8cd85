"""gemm() calls without a workspace of their own that overlap on the GPU: streams side by side, graphs replayed beside one
another and beside eager calls.  Every result has to be bit-identical to the same call made alone (both reductions add partial
sums in a fixed order)."""
import time

import pytest

import fp8_quant_matmul_b200 as f
from fp8_quant_matmul_b200 import api
import helpers as h
from test_gemm_gpu import to_dev

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (M, N, K), splits, tile_n: two that leave partial sums in the workspace, of different sizes, and stream-K
SPLIT_A = ((1024, 512, 7168), 4, 128 | f.SPLIT_WORKSPACE)
SPLIT_B = ((1024, 576, 7168), 3, 128 | f.SPLIT_WORKSPACE)
STREAM_K = ((1024, 576, 7168), 1, 128 | f.STREAM_K)


def prepare(config, seed):
    """call(C): one gemm() call; and its result when it is alone, with a workspace of its own."""
    (M, N, K), splits, tile_n = config
    operands = to_dev(*h.make_inputs(M, N, K, seed=seed))
    kw = dict(path=f.PATH_MN_SMALL, splits=splits, tile_n=tile_n)

    def call(C=None, **more):
        return f.gemm(*operands, C, M, N, K, **kw, **more)

    ws = torch.zeros(f.workspace_bytes(M, N, K, **kw), dtype=torch.uint8, device="cuda")
    want = call(workspace=ws).view(torch.int16)
    f.last_device_status()
    return call, want


@pytest.mark.parametrize("pair", [(SPLIT_A, SPLIT_A), (SPLIT_A, SPLIT_B), (STREAM_K, SPLIT_B)],
                         ids=["same split", "two splits", "stream-K and split"])
def test_two_streams_at_once(pair):
    calls = [prepare(c, seed=61 + i) for i, c in enumerate(pair)]
    streams = [torch.cuda.Stream() for _ in pair]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(25):
        for (call, _), stream, out in zip(calls, streams, got):
            with torch.cuda.stream(stream):
                out.append(call())
    torch.cuda.synchronize()
    f.last_device_status()
    for (_, want), out in zip(calls, got):
        assert all(torch.equal(C.view(torch.int16), want) for C in out)


def test_graphs_beside_one_another_and_beside_eager_calls():
    calls = [prepare(SPLIT_A, seed=71), prepare(SPLIT_B, seed=72)]
    graphs, outs = [], []
    held = len(api._graph_workspaces)
    for call, want in calls:                                    # both captured on torch's one capture stream
        C = [torch.zeros(want.shape, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for c in C:
                call(c)
        graphs.append(graph)
        outs.append(C)
    assert len(api._graph_workspaces) == held + 2               # one for each graph, not one for each call
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    eager = []
    for _ in range(10):
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
        with torch.cuda.stream(streams[2]):
            eager.append(calls[0][0]())
    torch.cuda.synchronize()
    f.last_device_status()
    for (_, want), C in zip(calls, outs):
        assert all(torch.equal(c.view(torch.int16), want) for c in C)
    assert all(torch.equal(c.view(torch.int16), calls[0][1]) for c in eager)
    # the workspace of a graph is given back when the graph is gone
    graph = None
    graphs.clear()
    for _ in range(100):
        api._drop_graph_workspaces()
        if len(api._graph_workspaces) <= held:
            break
        time.sleep(0.05)
    assert len(api._graph_workspaces) <= held


def test_an_eager_call_after_a_capture_on_the_same_stream():
    call, want = prepare(SPLIT_A, seed=81)
    stream = torch.cuda.Stream()
    C = torch.zeros(want.shape, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call(C)
    with torch.cuda.stream(stream):
        first = call()
        graph.replay()
        second = call()
    torch.cuda.synchronize()
    f.last_device_status()
    assert all(torch.equal(c.view(torch.int16), want) for c in (first, C, second))
