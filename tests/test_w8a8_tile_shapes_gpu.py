"""The tiled W8A8 GEMM at row and column counts around its tile choices, against integer sums on the host."""
import numpy as np
import pytest
import torch

from mindpipe_b200 import ops

pytestmark = pytest.mark.gpu

SHAPES = [(129, 8, 128), (129, 40, 4112), (256, 200, 256), (257, 1000, 144), (333, 12288, 512), (385, 4104, 256),
          (777, 6160, 128), (1025, 520, 1024), (130, 4096, 14336)]


def _sums(qx, qw):
    return (qx.double() @ qw.double().T).round().to(torch.int64)


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_symmetric_and_raw_sums(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m)
    qx = torch.randint(-128, 128, (m, k), generator=g, device="cuda", dtype=torch.int8)
    qw = torch.randint(-128, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)
    sx, sw = torch.rand(m, generator=g, device="cuda"), torch.rand(n, generator=g, device="cuda") * 1e-4
    bias = torch.randn(n, generator=g, device="cuda").half()
    acc = _sums(qx, qw)
    assert torch.equal(ops.w8a8_gemm_i32(qx, qw).long(), acc)
    y = ops.w8a8_gemm(qx, sx, qw, sw, bias)
    want = ((acc.float() * sx[:, None]) * sw[None, :] + bias.float()).half()
    ops.check_device_errors()
    assert torch.equal(y, want)


@pytest.mark.parametrize("beyond", ["none", "rows", "channels"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_zero_points(m, n, k, beyond):
    """Zero points in [0, 255] take 32-bit products, others (a row or channel on one side of zero) 64-bit ones."""
    g = torch.Generator(device="cuda").manual_seed(n)
    qx = torch.randint(0, 256, (m, k), generator=g, device="cuda", dtype=torch.uint8)
    qw = torch.randint(0, 256, (n, k), generator=g, device="cuda", dtype=torch.uint8)
    sx, sw = torch.rand(m, generator=g, device="cuda"), torch.rand(n, generator=g, device="cuda") * 1e-4
    zx = torch.randint(0, 256, (m,), generator=g, device="cuda").float()
    zw = torch.randint(0, 256, (n,), generator=g, device="cuda").float()
    if beyond == "rows":
        zx[m // 2], zx[-1] = -70000.0, 1e6
    elif beyond == "channels":
        zw[n // 2], zw[-1] = 300.0, -200000.0
    rx, rw = qx.sum(1, dtype=torch.int32), qw.sum(1, dtype=torch.int32)
    zxl, zwl = zx.long()[:, None], zw.long()[None, :]
    t = _sums(qx, qw) - zwl * rx.long()[:, None] - zxl * rw.long()[None, :] + k * zxl * zwl
    want = (t.float() * sx[:, None]) * sw[None, :]
    y = ops.w8a8_affine_gemm(qx, sx, zx, rx, qw, sw, zw, rw)
    ops.check_device_errors()
    assert torch.equal(y, want.half())
