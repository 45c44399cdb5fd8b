"""The scratch of ``mp_w4a16_linear``: what a shape asks for is what the kernel it runs on needs, whatever other shapes have
used the same buffer before."""
import pytest
import torch

from mindpipe_b200 import _lib, ops
from mindpipe_b200.modules import VllmPackedInt4Linear

# K of half a 128-column chunk, N of half an 8-row group: the tensor-core GEMM is the only kernel that takes them
ODD_SHAPES = [(4096, 4160, 64), (1024, 2880, 64), (4100, 512, 128), (516, 2880, 64)]


@pytest.mark.parametrize("m", [17, 32, 33, 64, 77, 96])
@pytest.mark.parametrize("n,k,group", ODD_SHAPES)
def test_shapes_of_the_gemm_ask_for_its_scratch(m, n, k, group):
    lib = _lib.load()
    prev = lib.mp_set_decode_kernel(2)                       # auto
    try:
        auto = lib.mp_w4a16_linear_workspace_bytes(m, n, k, group)
        lib.mp_set_decode_kernel(0)                          # the stream kernel off: the GEMM for more than 16 rows
        assert auto == lib.mp_w4a16_linear_workspace_bytes(m, n, k, group)
    finally:
        lib.mp_set_decode_kernel(prev)


def _module(n, k, group):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.02).half()
    packed, scale, zero, _ = ops.w4a16_quantize(w, group)
    return VllmPackedInt4Linear(packed_weight=packed, scale=scale, bias=None, in_features=k, out_features=n, zero_point=zero)


@pytest.mark.gpu
@pytest.mark.parametrize("rows_before", [200, 640])
@pytest.mark.parametrize("n,k,group", ODD_SHAPES)
def test_shapes_of_the_gemm_after_other_shapes_on_one_buffer(n, k, group, rows_before):
    """A call that grows the stream's buffer by some amount, then rows that took that amount for theirs."""
    before, mod = _module(1024, 1024, 128), _module(n, k, group)
    wdq = mod.dequantize().double()
    st = torch.cuda.Stream()                                 # a buffer of its own
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st), torch.no_grad():
        before(torch.randn(rows_before, 1024, device="cuda").half())
        for m in (17, 33, 64, 77, 96):
            x = torch.randn(m, k, device="cuda").half()
            ref = x.double() @ wdq.T
            y = mod(x)
            assert ((y.double() - ref).norm() / ref.norm()).item() <= 4e-4      # one fp16 rounding: 2^-11 / sqrt(3)
            assert torch.equal(y, ops.w4a16_linear(x, mod.weight_packed, mod._scale_zero))
    torch.cuda.synchronize()
    ops.check_device_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("m", [17, 64, 96])
def test_parameters_the_stream_kernel_declines_for_their_alignment(m):
    """(scale, zero) pairs on a 4-byte boundary: the GEMM without scratch, the same bits with any buffer."""
    n, k = 4096, 4096
    mod = _module(n, k, 128)
    mod._ensure_prepared()
    sz = torch.empty(mod._scale_zero.numel() + 2, dtype=torch.float16, device="cuda")[2:].view(mod._scale_zero.shape)
    sz.copy_(mod._scale_zero)
    x = torch.randn(m, k, device="cuda").half()
    y = torch.empty(m, n, dtype=torch.float16, device="cuda")
    lib = _lib.load()
    got = []
    need = lib.mp_w4a16_linear_workspace_bytes(m, n, k, 128)
    for extra in (0, 6 << 20, 32 << 20):
        ws = torch.zeros(need + extra, dtype=torch.uint8, device="cuda")
        st = lib.mp_w4a16_linear(x.data_ptr(), mod.weight_packed.data_ptr(), sz.data_ptr(), None, y.data_ptr(), m, n, k, 128,
                                 ws.data_ptr(), ws.numel(), ops._error_word(x.device).data_ptr(),
                                 torch.cuda.current_stream().cuda_stream)
        assert st == 0
        got.append(y.clone())
    ref = x.double() @ mod.dequantize().double().T
    assert ((got[0].double() - ref).norm() / ref.norm()).item() <= 4e-4
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    ops.check_device_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,runs", [(128, 4096, 4096, False), (200, 1024, 1024, False), (512, 1024, 2048, False),
                                        (97, 1024, 28672, True)])
def test_only_equal_runs_ask_for_room(m, n, k, runs):
    """Whole tiles and clusters of pairs write no partial tiles: no scratch, and the bits of a call that has some."""
    mod = _module(n, k, 128)
    mod._ensure_prepared()
    x = torch.randn(m, k, device="cuda").half()
    need = _lib.load().mp_w4a16_linear_workspace_bytes(m, n, k, 128)
    assert (need > 0) == runs
    y = torch.empty(m, n, dtype=torch.float16, device="cuda")
    for nbytes in (need, need + (64 << 20)):
        ws = torch.zeros(nbytes, dtype=torch.uint8, device="cuda") if nbytes else None
        st = _lib.load().mp_w4a16_linear(x.data_ptr(), mod.weight_packed.data_ptr(), mod._scale_zero.data_ptr(), None,
                                         y.data_ptr(), m, n, k, 128, None if ws is None else ws.data_ptr(), nbytes,
                                         ops._error_word(x.device).data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert st == 0
        assert torch.equal(y, ops.w4a16_linear_prefill(x, mod.weight_packed, mod._scale_zero))
    ref = x.double() @ mod.dequantize().double().T
    assert ((y.double() - ref).norm() / ref.norm()).item() <= 4e-4
    ops.check_device_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,group", [(18, 260, 8256, 64), (101, 260, 12352, 64), (149, 1500, 20544, 64),
                                         (311, 260, 12416, 128)])
def test_equal_runs_at_ragged_edges(m, n, k, group):
    """Tiles cut between pairs, their partial tiles added by the second kernel: edges of M, N and K inside a tile."""
    mod = _module(n, k, group)
    mod._ensure_prepared()
    assert _lib.load().mp_w4a16_linear_workspace_bytes(m, n, k, group) > 0
    wdq = mod.dequantize().double()
    bias = torch.randn(n, device="cuda").half()
    x = torch.randn(m, k, device="cuda").half()
    for b in (None, bias):
        y = ops.w4a16_linear(x, mod.weight_packed, mod._scale_zero, b)
        ref = x.double() @ wdq.T + (0 if b is None else b.double())
        assert ((y.double() - ref).norm() / ref.norm()).item() <= 4e-4
        assert torch.equal(y, ops.w4a16_linear(x, mod.weight_packed, mod._scale_zero, b))
    ops.check_device_errors()
