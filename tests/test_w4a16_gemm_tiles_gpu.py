"""The many-token W4A16 product at row, column and K counts around its tiles and splits, against the expanded weights."""
import pytest
import torch

from mindpipe_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,group", [
    (1, 8, 64, 64), (31, 24, 192, 64), (33, 200, 320, 64), (97, 257, 384, 192), (129, 264, 4160, 64), (160, 4096, 4096, 128),
    (255, 512, 128, 128), (257, 19000, 256, 256), (333, 1000, 2048, 2048), (385, 4104, 1088, 64), (513, 12288, 512, 128),
    (1030, 2056, 640, 128), (2048, 520, 1152, 128)])
def test_against_expanded_weights(m, n, k, group):
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.02).half()
    packed, scale, zero, _ = ops.w4a16_quantize(w, group)
    sz = ops.w4a16_prepare(scale, zero, k)
    wdq = ops.w4a16_dequant(packed, scale, zero, n, k).float()
    x = torch.randn(m, k, generator=g, device="cuda").half()
    bias = torch.randn(n, generator=g, device="cuda").half()
    ref = x.double() @ wdq.double().T
    for b in (None, bias):
        want = ref if b is None else ref + b.double()
        whole = torch.empty(m, n, dtype=torch.float16, device="cuda")
        st = _lib.load().mp_w4a16_linear_prefill(x.data_ptr(), packed.data_ptr(), sz.data_ptr(),
                                                 0 if b is None else b.data_ptr(), whole.data_ptr(), m, n, k, group,
                                                 ops._error_word(x.device).data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert st == 0
        for y in (whole, ops.w4a16_linear_prefill(x, packed, sz, b)):
            ops.check_device_errors()
            err = (y.double() - want).abs().max() / want.abs().max()
            assert err.item() <= 1e-3
            assert ((y.double() - want).norm() / want.norm()).item() <= 4e-4


def test_large_scales():
    """Expanded weights near the top of fp16: the same products as the expanded matrix gives."""
    g = torch.Generator(device="cuda").manual_seed(5)
    w = (torch.randn(256, 256, generator=g, device="cuda") * 8000).half().clamp(-60000, 60000)
    packed, scale, zero, _ = ops.w4a16_quantize(w, 64)
    sz = ops.w4a16_prepare(scale, zero, 256)
    wdq = ops.w4a16_dequant(packed, scale, zero, 256, 256).double()
    x = (torch.randn(200, 256, generator=g, device="cuda") * 1e-3).half()
    y = ops.w4a16_linear_prefill(x, packed, sz)
    ops.check_device_errors()
    want = x.double() @ wdq.T
    assert ((y.double() - want).norm() / want.norm()).item() <= 4e-4
