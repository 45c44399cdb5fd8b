"""Scratch of captured linears and experts: a graph's own, whatever its stream runs afterwards, and given back with it."""
import pytest
import torch

from mindpipe_b200 import _lib, ops
from mindpipe_b200.modules import SmoothQuantLinear, SmoothQuantPackedMoeExperts, VllmPackedInt4Linear

pytestmark = pytest.mark.gpu


def _linear(cls, n, k):
    lin = torch.nn.Linear(k, n, bias=False, device="meta", dtype=torch.float16)
    lin.weight = torch.nn.Parameter((torch.randn(n, k, device="cuda") * 0.02).half(), requires_grad=False)
    mod = cls.from_float(lin)
    mod.process_weights_after_loading()
    return mod


def _experts():
    e, h, i = 4, 512, 512
    mod = SmoothQuantPackedMoeExperts((torch.randn(e, 2 * i, h, device="cuda") * 0.02).half(),
                                      (torch.randn(e, h, i, device="cuda") * 0.02).half())
    x = torch.randn(48, h, device="cuda").half()
    index, weights = ops.moe_router_topk(torch.randn(48, e, device="cuda"), 2)
    return lambda: mod(x, index, weights)


def _call(kind, m, n, k):
    if kind == "experts":
        return _experts()
    mod = _linear({"w4": VllmPackedInt4Linear, "w8": SmoothQuantLinear}[kind], n, k)
    x = torch.randn(m, k, device="cuda").half()
    return lambda: mod(x)


def _capture(fn, stream):
    """The graph, its result and the scratch its launches hold."""
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = fn()
        held = ops._workspace(1, torch.device("cuda"))
    return graph, out, held


CALLS = [("w4", 1, 4096, 4096), ("w4", 8, 8192, 8192), ("w4", 16, 4096, 2048), ("w4", 77, 4096, 4096), ("w8", 4, 4096, 4096),
         ("experts", 0, 0, 0)]


@pytest.mark.parametrize("kind,m,n,k", CALLS)
@torch.no_grad()
def test_replay_after_the_stream_s_scratch_has_grown(kind, m, n, k, new_stream):
    fn, larger = _call(kind, m, n, k), [_call("w4", 17, 4096, 4096), _call("w4", 128, 8192, 2048), _experts()]
    want = fn().clone()
    stream = new_stream()
    with torch.cuda.stream(stream):
        fn()
        own = ops._workspace(1, torch.device("cuda"))
    stream.synchronize()
    graph, got, held = _capture(fn, stream)
    assert held.data_ptr() != own.data_ptr()
    size, address = own.numel(), own.data_ptr()
    del own
    with torch.cuda.stream(stream):
        for f in larger:
            f()
        assert ops._workspace(1, torch.device("cuda")).numel() > size or size >= 9 << 20
        others = [torch.full((size,), 0x5A, dtype=torch.uint8, device="cuda") for _ in range(4)]
        for _ in range(3):
            graph.replay()
            fn()                                             # the stream's own scratch, between replays
    torch.cuda.synchronize()
    ops.check_device_errors()
    assert torch.equal(got, want) and all(bool((t == 0x5A).all()) for t in others) and held.data_ptr() != address


@pytest.mark.parametrize("kind,m,n,k", CALLS)
@torch.no_grad()
def test_graphs_of_one_stream_side_by_side(kind, m, n, k, new_stream):
    calls = [_call(kind, m, n, k) for _ in range(2)]
    want = [f().clone() for f in calls]
    stream, streams = new_stream(), [new_stream(), new_stream()]
    with torch.cuda.stream(stream):
        calls[0]()
    stream.synchronize()
    graphs = [_capture(lambda f=f: [f() for _ in range(8)], stream) for f in calls]
    assert graphs[0][2].data_ptr() != graphs[1][2].data_ptr()
    for _ in range(5):
        for (graph, _, _), st in zip(graphs, streams):
            with torch.cuda.stream(st):
                graph.replay()
    torch.cuda.synchronize()
    ops.check_device_errors()
    for (_, got, _), w in zip(graphs, want):
        assert all(torch.equal(y, w) for y in got)


@torch.no_grad()
def test_scratch_that_grows_within_a_capture(new_stream):
    """Launches captured before it grew keep what they hold."""
    calls = [_call("w4", m, 4096, 4096) for m in (8, 32, 128, 16, 77)]
    want = [f().clone() for f in calls]
    stream = new_stream()
    with torch.cuda.stream(stream):
        for f in calls:
            f()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        got = [f() for f in calls]
    for _ in range(4):
        graph.replay()
    torch.cuda.synchronize()
    ops.check_device_errors()
    assert all(torch.equal(y, w) for y, w in zip(got, want))


@torch.no_grad()
def test_scratch_goes_back_with_its_graph(new_stream):
    fn = _call("w4", 16, 4096, 4096)
    stream = new_stream()
    with torch.cuda.stream(stream):
        want = fn().clone()
    stream.synchronize()
    count, addresses = [], []
    for _ in range(8):
        graph, got, held = _capture(fn, stream)
        count.append(len(_lib.host().workspaces()))
        addresses.append(held.data_ptr())
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        del graph, got, held
    assert count[-1] <= count[1] and len(set(addresses)) <= 4       # the same memory again
    kept = [_capture(fn, stream) for _ in range(4)]
    assert len({held.data_ptr() for _, _, held in kept}) == 4       # never while the graph is there


@pytest.mark.parametrize("m", [1, 8, 16, 77])
@torch.no_grad()
def test_a_capture_on_a_fresh_stream_records_the_products_alone(m, new_stream):
    """Its scratch is cleared once, not by a fill in front of every linear."""
    from cuda.bindings import runtime
    calls = [_call("w4", m, n, k) for n, k in ((4096, 4096), (4096, 2048), (5120, 4096))]
    want = [f().clone() for f in calls]
    stream = new_stream()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        got = [f() for f in calls]
    err, _, count = runtime.cudaGraphGetNodes(runtime.cudaGraph_t(graph.raw_cuda_graph()), 0)
    assert int(err) == 0 and count == len(calls)
    graph.instantiate()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    ops.check_device_errors()
    assert all(torch.equal(y, w) for y, w in zip(got, want))
