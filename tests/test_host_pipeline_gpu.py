"""``forward_host_many``: rows that come beside the first product and results that leave beside the later ones, for sets in
which a linear's kernel takes copies along, wherever it is given, and for ones in which none does; new rows at every call."""
import pytest
import torch

from mindpipe_b200 import _lib, ops
from mindpipe_b200.modules import VllmPackedInt4Linear, _HostPipeline, forward_host_many

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


def test_the_stream_waits_for_the_side_stream_after_an_error():
    """The second product is refused (a group that does not divide K) when the first one's result is on its way: whoever
    waits for the stream then may use the buffers again."""
    rows, bad, shapes = 16, 1, [(262144, 256), (4096, 4096), (1024, 4096)]
    g = torch.Generator(device="cuda").manual_seed(0)
    stream = torch.cuda.Stream()
    calls, keep = (_lib.HostLinear * len(shapes))(), []
    for c, (n, k) in zip(calls, shapes):
        lin = torch.nn.Linear(k, n, bias=False, device="meta", dtype=torch.float16)
        lin.weight = torch.nn.Parameter((torch.randn(n, k, generator=g, device="cuda") * 0.02).half(), requires_grad=False)
        mod = VllmPackedInt4Linear.from_float(lin, group_size=128)
        mod.process_weights_after_loading()
        x = torch.randn(rows, k, generator=g, device="cuda").half()
        x_host, y_host = x.cpu().pin_memory(), torch.full((rows, n), float("nan"), dtype=torch.float16).pin_memory()
        xs, ys = torch.empty_like(x), torch.empty((rows, n), dtype=torch.float16, device="cuda")
        ws = ops.new_workspace(16 << 20, "cuda")
        keep.append((mod, x, x_host, y_host, xs, ys, ws))
        c.x_host_f16, c.x_stage_f16, c.y_stage_f16, c.y_host_f16 = (t.data_ptr() for t in (x_host, xs, ys, y_host))
        c.packed_i32, c.sz_f16x2, c.bias_f16 = mod.weight_packed.data_ptr(), mod._scale_zero.data_ptr(), None
        c.M, c.N, c.K, c.group = rows, n, k, 128
        c.workspace, c.workspace_bytes = ws.data_ptr(), ws.numel()
    calls[bad].group = 96
    mod, x, _, y_host, *_ = keep[0]
    want = mod(x).cpu()
    pipeline = _HostPipeline(calls, len(shapes), stream.cuda_stream)
    assert pipeline.status == 0
    for _ in range(4):
        y_host.fill_(float("nan"))
        torch.cuda.synchronize()
        assert pipeline.run() != 0
        stream.synchronize()
        last = float(y_host[-1, -1])                        # the copy's end, before a look at the rest gives it time
        assert last == float(want[-1, -1]) and torch.equal(y_host, want)
    torch.cuda.synchronize()
    ops.check_device_errors()
