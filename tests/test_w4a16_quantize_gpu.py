"""Quantise / pack / expand kernels at every group size with its own kernel, ragged rows and extreme groups."""
import numpy as np
import pytest
import torch

from mindpipe_b200 import ops
from oracle import pseudo_quant as O

pytestmark = pytest.mark.gpu


def _weights(n, k, group, seed):
    rng = np.random.default_rng(seed)
    w = rng.normal(0, 0.02, (n, k // group, group))
    w[0, 0] = 0.0                                       # constant groups
    w[1, -1] = 0.75
    w[2, 0] = rng.normal(0, 1e-6, group)                # scale below 2^-14
    w[3, 0] = rng.normal(40.0, 0.01, group)             # far from zero: quotients beyond any code
    w[4, -1] = -rng.uniform(100, 101, group)
    w[5, 0] = rng.normal(0, 9000.0, group)              # large
    w[6, -1, :2] = (60000.0, -60000.0)                  # span overflows fp16
    w[7, 0] = np.arange(group) % 31 * 0.5               # ties
    w[8, 0] = rng.normal(1.0, 3e-4, group)
    return w.reshape(n, k).astype(np.float16)


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("group", [32, 64, 128, 256, 48, 8, 2048])
@pytest.mark.parametrize("groups_per_row", [1, 7, 8, 9, 24])
def test_codes_scales_zero_points_and_dequant_bit_exact(group, groups_per_row):
    n, k = 11, group * groups_per_row
    w = _weights(n, k, group, seed=group + groups_per_row)
    packed, scale, zero, g = ops.w4a16_quantize(torch.from_numpy(w).cuda(), group)
    assert g == group
    wdq, s, z, u = O.w4_group_asym_quantize(w, group)
    assert np.array_equal(scale.cpu().numpy().view(np.uint16), s.reshape(n, -1).view(np.uint16))
    assert np.array_equal(packed.cpu().numpy(), O.pack_int4_unsigned(u))
    zw = zero.cpu().numpy().view(np.uint32)
    zi = np.stack([(zw[:, i // 8] >> (4 * (i % 8))) & 15 for i in range(groups_per_row)], axis=1)
    assert np.array_equal(zi, z.reshape(n, -1).astype(np.uint32))
    out = ops.w4a16_dequant(packed, scale, zero, n, k).cpu().numpy()
    finite = np.isfinite(wdq)
    assert np.array_equal(out[finite].view(np.uint16), wdq[finite].view(np.uint16))
