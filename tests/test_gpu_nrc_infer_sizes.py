"""Radiance-cache inference at the edges of its tiles, warpgroups and grid,
from inputs on 16-byte boundaries and not: each row's answer is the one it has
in the largest batch, which follows the numpy emulation, and nothing past the
last row is written."""
import numpy as np
import pytest

from rs_illume_b200 import _lib
from rs_illume_b200.nrc import RadianceCache
from tests import nrc_reference as ref
from tests.test_gpu_nrc import BOUND, random_inputs

pytestmark = pytest.mark.gpu
TILE, SMS, GROUPS = 128, 148, 5


def test_sizes(ctx):
    import torch
    sizes = {1, 2, TILE - 1, TILE, TILE + 1, 2 * TILE, 3 * TILE + 5}
    for g in range(1, GROUPS + 1):
        sizes |= {g * SMS * TILE + k for k in (-1, 0, 1)}
    most = 2 * GROUPS * SMS * TILE + 77
    x, _ = random_inputs(most, 3)
    c = RadianceCache(ctx, BOUND, seed=11)
    d_x = torch.from_numpy(x).cuda()
    off = torch.zeros(most * 12 + 1, device="cuda")
    off[1:] = d_x.reshape(-1)

    def infer(inputs, n):
        out = torch.full((n + 1, 3), -7.0, device="cuda")
        torch.cuda.synchronize()
        ctx.check(ctx._lib.ilm_nrc_infer(ctx.handle, c.handle, inputs, n, out.data_ptr(), _lib.CUDA_STREAM_LEGACY),
                  "ilm_nrc_infer")
        assert torch.all(out[n] == -7.0)
        return out[:n]

    full = infer(d_x.data_ptr(), most)
    for n in sorted(sizes) + [most]:
        assert torch.equal(infer(d_x.data_ptr(), n), full[:n]), n
        assert torch.equal(infer(off.data_ptr() + 4, n), full[:n]), n
    pick = np.r_[0:300, most - 300:most]
    pred, _, _ = ref.forward_backward(c.encode(x[pick]), c.params(), np.zeros((len(pick), 3), np.float32))
    got = full.cpu().numpy()[pick]
    # the bars of test_inference_tile_pairs
    assert np.mean(np.abs(got - pred) <= 1e-4 + 1e-4 * np.abs(pred)) > 0.98
    assert np.linalg.norm(got - pred) <= 2e-2 * np.linalg.norm(pred)
    c.close()
