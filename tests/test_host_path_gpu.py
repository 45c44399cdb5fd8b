"""The native forward of the modules against their checked Python path: same bits, and never a stale plan."""
import copy

import pytest
import torch

from mindpipe_b200.modules import QuantLinear, SmoothQuantLinear, SmoothQuantPackedMoeExperts, VllmPackedInt4Linear

pytestmark = pytest.mark.gpu


def _linear(n, k, bias, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    lin = torch.nn.Linear(k, n, bias=bias, device="cuda", dtype=torch.float16)
    with torch.no_grad():
        lin.weight.normal_(0, 0.02, generator=g)
    return lin


MAKERS = {"w4": lambda lin: VllmPackedInt4Linear.from_float(lin, group_size=128), "w8": SmoothQuantLinear.from_float,
          "affine": QuantLinear}


@pytest.mark.parametrize("kind", sorted(MAKERS))
@pytest.mark.parametrize("lead", [(1,), (2, 3), (40,), (130,)])
@pytest.mark.parametrize("bias", [False, True])
def test_plan_gives_the_checked_path_s_bits(kind, lead, bias):
    mod = MAKERS[kind](_linear(384, 512, bias))
    x = torch.randn((*lead, 512), device="cuda").half()
    want = mod._forward_checked(x)
    assert mod._plan is not None
    got = mod(x)
    assert got.shape == want.shape == (*lead, 384) and torch.equal(got, want)
    assert torch.equal(mod(x.expand(2, *lead, 512).transpose(0, 1)[:, 0] if len(lead) == 1 else x), want)   # strided view


@pytest.mark.parametrize("kind", sorted(MAKERS))
def test_plan_follows_replaced_and_edited_weights(kind):
    mod, other = MAKERS[kind](_linear(256, 512, True)), MAKERS[kind](_linear(256, 512, True, seed=1))
    x = torch.randn((3, 512), device="cuda").half()
    first = mod(x).clone()
    twin = copy.deepcopy(mod)
    shallow = copy.copy(mod)
    assert torch.equal(mod(x), first)
    mod.load_state_dict(other.state_dict())                      # in place
    assert torch.equal(mod(x), other._forward_checked(x)) and not torch.equal(mod(x), first)
    assert torch.equal(twin(x), first)                           # a copy keeps its own weights
    assert torch.equal(shallow(x), mod(x))                       # a shallow one shares them
    mod.bias = torch.zeros_like(mod.bias)                        # replaced
    assert torch.equal(mod(x), mod._forward_checked(x)) and not torch.equal(mod(x), other(x))


def test_experts_plan_gives_the_checked_path_s_bits():
    e, h, i, t = 4, 256, 384, 21
    mod = SmoothQuantPackedMoeExperts(torch.randn(e, 2 * i, h, device="cuda").half() * 0.05,
                                      torch.randn(e, h, i, device="cuda").half() * 0.05)
    x = torch.randn(3, 7, h, device="cuda").half()
    ids = torch.rand(t, e, device="cuda").topk(2, dim=1).indices
    w = torch.rand(t, 2, device="cuda").half()
    want = mod._forward_checked(x, ids, w)
    assert torch.equal(mod(x, ids.int(), w), want)               # the plan's types
    assert torch.equal(mod(x, ids, w.float()), want)             # other types: converted by the checked path
