"""Per-token quantisation with few and many rows: the block shape follows the row count, the bits do not."""
import pytest
import torch

from mindpipe_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2056, 4096, 4104, 8192, 8200, 11008, 16384, 16392])
def test_same_bits_whatever_the_row_count(k):
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(149, k, generator=g, device="cuda").half()
    x[:, ::97] *= 20
    x[3], x[5] = 0, x[5].abs()
    q, s, fake = ops.act_quant_per_token(x, want_fake=True)
    parts = [ops.act_quant_per_token(x[i:i + 50].contiguous(), want_fake=True) for i in range(0, 149, 50)]
    for whole, j in ((q, 0), (s, 1), (fake, 2)):
        assert torch.equal(whole, torch.cat([p[j] for p in parts]))
    whole = ops.affine_quant_per_row(x)
    parts = [ops.affine_quant_per_row(x[i:i + 50].contiguous()) for i in range(0, 149, 50)]
    for j, t in enumerate(whole):
        if t is not None:
            assert torch.equal(t, torch.cat([p[j] for p in parts]))


@pytest.mark.parametrize("k", [8, 128, 1016, 1024, 1032, 2048, 2056, 4088, 4096, 4104, 8200, 11008])
def test_wide_blocks_give_the_bits_of_narrow_ones(k):
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(593, k, generator=g, device="cuda").half()
    x[:, -1] *= 20                                       # the last piece holds the largest value
    x[3], x[5], x[7] = 0, x[5].abs() * -1, 1e-5
    whole, affine = ops.act_quant_per_token(x, want_fake=True), ops.affine_quant_per_row(x)
    x[9, 0], x[11, k - 1], x[13] = float("inf"), float("nan"), float("nan")
    odd = ops.act_quant_per_token(x, want_fake=True)
    for rows in (1, 592):
        parts = [ops.affine_quant_per_row(p) for p in x[:9].split(rows)]
        assert all(torch.equal(torch.cat([p[j] for p in parts]), t[:9]) for j, t in enumerate(affine) if t is not None)
        for of, n in ((whole, 9), (odd, 593)):
            q, s, fake = (torch.cat(t) for t in zip(*(ops.act_quant_per_token(p, want_fake=True) for p in x[:n].split(rows))))
            assert torch.equal(q, of[0][:n]) and torch.equal(s, of[1][:n])
            assert torch.equal(fake.view(torch.int16), of[2][:n].view(torch.int16))


@pytest.mark.parametrize("rows", [64, 65, 160, 161, 200, 201, 256, 257, 296, 297, 592])
@pytest.mark.parametrize("k", [2048, 3072, 3080, 4096, 4104, 8192, 8200, 16384])
def test_either_side_of_the_lines_between_wide_and_narrow_blocks(k, rows):
    """The bits of the rows one at a time, at the row counts and widths where the block shape changes."""
    g = torch.Generator(device="cuda").manual_seed(k + rows)
    x = torch.randn(rows, k, generator=g, device="cuda").half()
    x[:, -1] *= 20
    few = torch.tensor([0, 1, rows // 2, rows - 1], device="cuda")
    whole, parts = ops.act_quant_per_token(x, want_fake=True), [ops.act_quant_per_token(x[i:i + 1], want_fake=True) for i in few]
    for j in range(3):
        assert torch.equal(whole[j][few], torch.cat([p[j] for p in parts]))
    whole, parts = ops.affine_quant_per_row(x), [ops.affine_quant_per_row(x[i:i + 1]) for i in few]
    for j, t in enumerate(whole):
        if t is not None:
            assert torch.equal(t[few], torch.cat([p[j] for p in parts]))
