"""The weight-streaming W8A8 product against the tiled GEMM: integer sums and the same output arithmetic, so the same
bits, at the row counts where its tiles change, ragged shapes and cuts of K over many blocks."""
import numpy as np
import pytest
import torch

from mindpipe_b200 import _lib, ops
from mindpipe_b200.modules import QuantLinear, SmoothQuantLinear, SmoothQuantPackedMoeExperts
from oracle import pseudo_quant as O

pytestmark = pytest.mark.gpu


def _linear(n, k, bias):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    lin = torch.nn.Linear(k, n, bias=bias, device="cuda", dtype=torch.float16)
    with torch.no_grad():
        lin.weight.normal_(0, 0.02, generator=g)
        lin.weight[0] = lin.weight[0].abs() + 0.01             # one-sided rows: zero points outside the codes
        lin.weight[n // 2] = -lin.weight[n // 2].abs() - 0.01
    return lin


@pytest.mark.parametrize("kind", [SmoothQuantLinear.from_float, QuantLinear], ids=["symmetric", "affine"])
@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65, 128, 129])
@pytest.mark.parametrize("n,k", [(40, 512), (384, 4112), (1026, 1024), (20480, 256), (256, 16384), (4096, 4096)])
def test_streamed_product_gives_the_tiled_gemm_s_bits(kind, m, n, k):
    mod = kind(_linear(n, k, bias=m % 2 == 0))
    x = torch.randn(m, k, device="cuda").half()
    x[:, ::97] *= 20
    x[m // 2] = x[m // 2].abs() + 1
    want = mod._forward_checked(x)
    assert mod._plan is not None
    for _ in range(3):
        assert torch.equal(mod(x), want)
    ops.check_device_errors()


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("n,k", [(40, 16), (8, 144), (384, 4112), (1026, 1024), (20480, 256), (256, 8192), (4096, 4096),
                                 (264, 28672), (24576, 2064)])
def test_rows_quantised_in_the_stream_give_the_quantiser_s_codes(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m * n + k)
    mod = SmoothQuantLinear.from_float(_linear(n, k, bias=m % 2 == 0))
    x = torch.randn(m, k, generator=g, device="cuda").half()
    x[:, ::97] *= 20
    x[:, -1] *= 30                                             # the last piece of a row holds its largest value
    if m > 2:
        x[1], x[2] = 0, x[2] * 1e-4                            # a scale below 2^-14
    q, s, _ = ops.act_quant_per_token(x)
    w_scale = mod.weight_scale.flatten().float()
    want = ops.w8a8_gemm(q, s, mod.weight, w_scale, mod.bias)
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    ws = torch.zeros(lib.mp_w8a8_linear_workspace_bytes(m, n, k), dtype=torch.uint8, device="cuda")
    for _ in range(3):
        q2, s2, y = torch.full_like(q, 85), torch.full_like(s, -1), torch.full_like(want, -1)
        assert lib.mp_w8a8_linear(x.data_ptr(), mod.weight.data_ptr(), w_scale.data_ptr(),
                                  mod.bias.data_ptr() if mod.bias is not None else None, y.data_ptr(), m, n, k,
                                  q2.data_ptr(), s2.data_ptr(), ws.data_ptr(), ws.numel(), None, st) == 0
        assert torch.equal(q2, q) and torch.equal(s2, s) and torch.equal(y, want)
        assert torch.equal(mod(x), want)
    if n == k:                                                 # results over the rows
        assert lib.mp_w8a8_linear(x.data_ptr(), mod.weight.data_ptr(), w_scale.data_ptr(),
                                  mod.bias.data_ptr() if mod.bias is not None else None, x.data_ptr(), m, n, k,
                                  q2.data_ptr(), s2.data_ptr(), ws.data_ptr(), ws.numel(), None, st) == 0
        assert torch.equal(x, want) and torch.equal(q2, q)


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("k", [8, 1024, 2056, 4096, 8192, 11008, 16392])
def test_affine_quantiser_bit_exact_at_every_row_length(k):
    rng = np.random.default_rng(k)
    x = rng.normal(0, 1, (12, k))
    x[0], x[1], x[2] = 0.0, 3.25, -np.abs(x[2]) - 5.0          # constant and one-sided rows
    x[3], x[4] = np.abs(x[3]) * 1e-3 + 50.0, x[4] * 1e-5       # far from zero; scale below 2^-14
    x[5], x[6, 0] = x[5] * 9000.0, 60000.0
    x[7] = np.arange(k) % 511 * 0.25
    x = x.astype(np.float16)
    q, s, z, rs, f = ops.affine_quant_per_row(torch.from_numpy(x).cuda(), want_fake=True)
    fake, codes, sc, zp = O.affine_quant_last_dim(x)
    assert np.array_equal(q.cpu().numpy(), codes)
    assert np.array_equal(s.cpu().numpy(), sc.astype(np.float32).reshape(-1))
    assert np.array_equal(z.cpu().numpy(), zp.astype(np.float32).reshape(-1))
    assert np.array_equal(rs.cpu().numpy(), codes.astype(np.int64).sum(axis=1).astype(np.int32))
    assert np.array_equal(f.cpu().numpy(), fake)


@pytest.mark.parametrize("t", [1, 16, 17, 33, 64, 65])
@pytest.mark.parametrize("e,h,i,k", [(4, 256, 384, 2), (8, 1024, 144, 2), (40, 512, 272, 4)])
@pytest.mark.parametrize("routing", ["random", "one expert", "twice the same"])
def test_expert_layer_of_few_tokens_gives_the_staged_layer_s_bits(t, e, h, i, k, routing):
    g = torch.Generator(device="cuda").manual_seed(t + e)
    mod = SmoothQuantPackedMoeExperts(torch.randn(e, 2 * i, h, generator=g, device="cuda").half() * 0.05,
                                      torch.randn(e, h, i, generator=g, device="cuda").half() * 0.05)
    x = torch.randn(t, h, generator=g, device="cuda").half()
    ids = torch.rand(t, e, generator=g, device="cuda").topk(k, dim=1).indices.int()
    if routing == "one expert":
        ids = torch.arange(k, device="cuda", dtype=torch.int32).expand(t, k).contiguous()
    elif routing == "twice the same":
        ids[:, 1] = ids[:, 0]
    w = torch.rand(t, k, generator=g, device="cuda").half()
    want = mod._forward_checked(x, ids, w)
    assert mod._plan is not None
    for _ in range(3):
        assert torch.equal(mod(x, ids, w), want)
    ops.check_device_errors()


@pytest.mark.parametrize("e", [4, 8, 12, 32, 40])
def test_router_matches_softmax_topk_at_every_width(e):
    logits = torch.randn(300, e, device="cuda") * 2
    logits[0] = 0.5                                            # all equal: lower indices first
    logits[1, 1], logits[1, 3] = 9.0, 9.0
    idx, w = ops.moe_router_topk(logits, 2)
    p = logits.softmax(dim=-1)
    top, ref = p.sort(dim=-1, descending=True, stable=True)
    assert torch.equal(idx.long(), ref[:, :2])
    want = top[:, :2] / top[:, :2].sum(dim=-1, keepdim=True)
    assert (w.float() - want).abs().max().item() <= 1e-3


@pytest.mark.parametrize("t,k,lo,hi", [(1, 1, 0, 4), (3, 2, 0, 16), (128, 2, 0, 8), (129, 2, 0, 8), (60, 4, 2, 6), (32, 8, 0, 256), (149, 2, 0, 8),
                                       (700, 3, 1, 6)])
def test_routing_plan_and_rows(t, k, lo, hi):
    """Routing of few entries makes its plan beside the gather, of many tokens goes token by token: counts, segments, tiles, scales and codes as the host
    lays them out, every entry on a row of its expert."""
    from mindpipe_b200 import _lib, ops
    lib = _lib.load()
    h, e = 256, hi - lo
    g = torch.Generator(device="cuda").manual_seed(t)
    x = torch.randn(t, h, generator=g, device="cuda").half()
    ids = torch.stack([torch.randperm(max(hi + 2, k), generator=g, device="cuda")[:k] for _ in range(t)]).int()
    padded = lib.mp_moe_padded_rows(e, t * k)
    plan = torch.full((lib.mp_moe_plan_ints(e, t * k),), -7, dtype=torch.int32, device="cuda")
    dest = torch.full((t * k,), -7, dtype=torch.int32, device="cuda")
    q = torch.full((padded, h), 99, dtype=torch.int8, device="cuda")
    s = torch.full((padded,), -1.0, device="cuda")
    assert lib.mp_moe_route_gather_quant(x.data_ptr(), ids.data_ptr(), t, h, k, lo, hi, plan.data_ptr(), dest.data_ptr(),
                                         q.data_ptr(), s.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    flat = ids.flatten().cpu().tolist()
    counts = [flat.count(x_) for x_ in range(lo, hi)]
    seg = [0]
    for c in counts:
        seg.append(seg[-1] + (c + 255) // 256 * 256)
    p, d = plan.cpu().tolist(), dest.cpu().tolist()
    assert p[:e] == counts and p[e:2 * e] == counts and p[2 * e:3 * e + 1] == seg and p[3 * e + 1] == seg[-1] // 128
    assert p[3 * e + 2:3 * e + 2 + seg[-1] // 128] == [i for i in range(e) for _ in range((seg[i + 1] - seg[i]) // 128)]
    want_q, want_s, _ = ops.act_quant_per_token(x)
    used = set()
    for i, x_ in enumerate(flat):
        if not lo <= x_ < hi:
            assert d[i] == -1
            continue
        assert seg[x_ - lo] <= d[i] < seg[x_ - lo] + counts[x_ - lo] and d[i] not in used
        used.add(d[i])
        assert torch.equal(q[d[i]], want_q[i // k]) and s[d[i]].item() == want_s.flatten()[i // k].item()
    rest = torch.ones(padded, dtype=torch.bool)
    rest[list(used)] = False
    assert (s.cpu()[rest] == 0).all()


@pytest.mark.parametrize("kind", [SmoothQuantLinear.from_float, QuantLinear], ids=["symmetric", "affine"])
@pytest.mark.parametrize("m,n,k", [(1, 24610, 4112), (8, 24610, 4112), (8, 6168, 16400)])
def test_long_streams_give_the_tiled_gemm_s_bits(kind, m, n, k):
    """Blocks of 40 stages and more, which take the longer ring."""
    mod = kind(_linear(n, k, bias=True))
    x = torch.randn(m, k, device="cuda").half()
    want = mod._forward_checked(x)
    for _ in range(3):
        assert torch.equal(mod(x), want)
    ops.check_device_errors()


@pytest.mark.parametrize("t", [5, 17, 33, 64])
def test_long_streams_of_experts_give_the_staged_layer_s_bits(t):
    g = torch.Generator(device="cuda").manual_seed(t)
    e, h, i = 8, 2064, 6400
    mod = SmoothQuantPackedMoeExperts(torch.randn(e, 2 * i, h, generator=g, device="cuda").half() * 0.05,
                                      torch.randn(e, h, i, generator=g, device="cuda").half() * 0.05)
    x = torch.randn(t, h, generator=g, device="cuda").half()
    ids = torch.rand(t, e, generator=g, device="cuda").topk(2, dim=1).indices.int()
    w = torch.rand(t, 2, generator=g, device="cuda").half()
    want = mod._forward_checked(x, ids, w)
    for _ in range(3):
        assert torch.equal(mod(x, ids, w), want)
    ops.check_device_errors()
