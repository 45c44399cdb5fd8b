"""``w4a16_linear`` at the row counts where its kernels hand over and at ragged shapes, against fp32 of the expanded
weights; repeated calls give the same bits and leave the scratch buffer's tiles zero."""
import pytest
import torch

from mindpipe_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _case(n, k, m, group):
    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.02).half()
    packed, scale, zero, _ = ops.w4a16_quantize(w, group)
    sz = ops.w4a16_prepare(scale, zero, k)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    bias = torch.randn(n, generator=g, device="cuda").half()
    return x, packed, sz, bias, ops.w4a16_dequant(packed, scale, zero, n, k).float()


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32, 33, 48, 49, 64, 65, 80, 81, 96, 97, 112, 113, 128, 129])
@pytest.mark.parametrize("n,k,group", [(8200, 1664, 128), (264, 1280, 128), (4104, 512, 64), (40, 1408, 128), (2048, 2176, 128),
                                       (20480, 512, 256), (1032, 4096, 4096)])
def test_linear_at_row_count_edges(m, n, k, group):
    x, packed, sz, bias, wdq = _case(n, k, m, group)
    for b in (None, bias):
        y = ops.w4a16_linear(x, packed, sz, b)
        ref = x.float() @ wdq.t() + (0 if b is None else b.float())
        assert ((y.float() - ref).norm() / ref.norm()).item() <= 1e-3
        for _ in range(2):
            assert torch.equal(ops.w4a16_linear(x, packed, sz, b), y)
    ops.check_device_errors()
    nbytes = _lib.load().mp_w4a16_linear_workspace_bytes(min(m, 16), 28672, 8192, 128)      # counters and 16-token tiles
    assert not ops._workspace(nbytes, x.device)[:nbytes].any()


@pytest.mark.parametrize("m", [5, 16, 50, 100])
def test_linear_of_extreme_values(m):
    """Zeros, infinities and NaNs pass through the partial tiles (whose words mean "not there yet" when zero)."""
    n, k = 512, 8192
    x, packed, sz, _, wdq = _case(n, k, m, 128)
    x.zero_()
    assert not ops.w4a16_linear(x, packed, sz).any()
    x[0, 3], x[m - 1, k - 1] = float("inf"), float("nan")
    y = ops.w4a16_linear(x, packed, sz)
    assert y[m - 1].isnan().all() and not torch.isfinite(y[0]).any() and not y[1:m - 1].any()
    ops.check_device_errors()


@pytest.mark.parametrize("m", [1, 16, 17, 33, 48, 64, 77, 96, 112, 128])
@pytest.mark.parametrize("n,k", [(1024, 8192), (512, 2048), (4104, 4096)])
def test_chained_launches_with_early_weights_share_scratch(n, k, m):
    """Blocks of few stages that close a row block, behind a launch whose partial tiles lie in the same scratch: none may
    take the other's.  The same bits as one launch at a time."""
    cases = [_case(n, k, m, group)[:3] for group in (128, 64)]
    want = [ops.w4a16_linear(*c) for c in cases]
    lib = _lib.load()
    before = lib.mp_set_programmatic_launch(1)
    stream = torch.cuda.Stream()
    try:
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            ops.w4a16_linear(*cases[0])
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = [ops.w4a16_linear(*cases[i % 2]) for i in range(8)]
        for _ in range(10):
            graph.replay()
        torch.cuda.synchronize()
    finally:
        lib.mp_set_programmatic_launch(before)
    ops.check_device_errors()
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2])


@pytest.mark.parametrize("m,n,k", [(1, 4096, 4096), (8, 8192, 8192), (16, 1024, 8192), (16, 12288, 4096),
                                   (77, 4096, 4096), (100, 4096, 4096), (128, 8192, 2048)])
def test_capture_on_a_stream_without_scratch(m, n, k, new_stream):
    """A capture needs no call on its stream before; the graph has zeroed scratch of its own."""
    x, packed, sz, bias, _ = _case(n, k, m, 128)
    want = ops.w4a16_linear(x, packed, sz, bias)
    stream = new_stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        got = [ops.w4a16_linear(x, packed, sz, bias) for _ in range(3)]
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    ops.check_device_errors()
    assert all(torch.equal(y, want) for y in got)


def test_weights_that_share_memory_and_more_of_them_than_maps_are_kept():
    """Weights of other shapes and groups at the same addresses, and 160 of them in turn, again and again."""
    g = torch.Generator(device="cuda").manual_seed(5)
    codes = torch.randint(-2**31, 2**31 - 1, (4096 * 4096 // 8,), generator=g, dtype=torch.int32, device="cuda")
    pairs = (torch.rand(4096 * 4096 // 64 * 2, generator=g, device="cuda") * 0.01).half()
    forms = []
    for n, k, group in ((4096, 4096, 128), (2048, 8192, 128), (8192, 2048, 64), (4096, 4096, 64), (4096, 2048, 128)):
        packed = codes[:n * k // 8].view(n, k // 8)
        sz = pairs[:k // group * n * 2].view(k // group, n, 2)
        x = torch.randn(5, k, generator=g, device="cuda").half()
        forms.append((x, packed, sz, ops.w4a16_linear(x, packed.clone(), sz.clone())))
    many = []
    for i in range(160):
        packed, sz = codes[i * 4096:][:2048 * 2048 // 8].view(2048, 256), pairs[i * 64:][:16 * 2048 * 2].view(16, 2048, 2)
        x = torch.randn(9, 2048, generator=g, device="cuda").half()
        many.append((x, packed, sz, ops.w4a16_linear(x, packed.clone(), sz.clone())))
    for _ in range(2):
        for x, packed, sz, want in forms + many:
            assert torch.equal(ops.w4a16_linear(x, packed, sz), want)
    ops.check_device_errors()
