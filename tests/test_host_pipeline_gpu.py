"""``forward_host_many``: rows that come beside the first product and results that leave beside the later ones, for sets in
which a linear's kernel takes copies along, wherever it is given, and for ones in which none does; new rows at every call."""
import pytest
import torch

from mindpipe_b200 import ops
from mindpipe_b200.modules import VllmPackedInt4Linear, forward_host_many

pytestmark = pytest.mark.gpu

SETS = {"carried": [(12288, 4096), (4096, 11008), (4096, 4096), (1024, 4096)],
        "the smallest result given first": [(512, 2048), (22016, 4096), (4096, 11008)],
        "one linear": [(22016, 4096)],
        "everything in one copy each way": [(2048, 2048), (1024, 2048)],
        "a later one goes first": [(1024, 2048), (22016, 4096), (512, 11008)],
        "only the smallest result's kernel takes some": [(1536, 2048), (1536, 2048), (1024, 8192)],
        "no kernel takes any": [(512, 4096)] * 6,
        "no kernel takes any, results beside the products": [(2040, 3072)] * 9}


@pytest.mark.parametrize("shapes", list(SETS.values()), ids=list(SETS))
@pytest.mark.parametrize("rows", [1, 7, 16])
def test_results_are_those_of_the_single_forwards(shapes, rows):
    g = torch.Generator(device="cuda").manual_seed(rows)
    mods = []
    for n, k in shapes:
        lin = torch.nn.Linear(k, n, bias=False, device="meta", dtype=torch.float16)
        lin.weight = torch.nn.Parameter((torch.randn(n, k, generator=g, device="cuda") * 0.02).half(), requires_grad=False)
        mods.append(VllmPackedInt4Linear.from_float(lin, group_size=128))
        mods[-1].process_weights_after_loading()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    sets = [([torch.empty((rows, k), dtype=torch.float16).pin_memory() for _, k in shapes],
             [torch.empty((rows, n), dtype=torch.float16).pin_memory() for n, _ in shapes]) for _ in streams]
    for _ in range(4):
        want = []
        for (xs, ys), stream in zip(sets, streams):
            for x, y in zip(xs, ys):
                x.copy_(torch.randn(x.shape, generator=g, device="cuda"))
                y.fill_(float("nan"))
            want.append([m(x.cuda()).cpu() for m, x in zip(mods, xs)])
        torch.cuda.synchronize()
        for (xs, ys), stream in zip(sets, streams):
            forward_host_many(mods, xs, ys, stream=stream)
        for (xs, ys), stream, w in zip(sets, streams, want):
            stream.synchronize()
            for y, v in zip(ys, w):
                assert torch.equal(y, v)
    ops.check_device_errors()
