"""Radiance-cache gradients at the edges of the training kernels' tiles (128
rows), staging steps (64) and row chunks (256 and up), from inputs on 16-byte
boundaries and not, after a larger batch has left its rows behind: per layer
within 2% of the numpy emulation, as tests/test_gpu_nrc.py asks."""
import numpy as np
import pytest

from rs_illume_b200 import _lib
from rs_illume_b200.nrc import N_PARAMS, RadianceCache, split_params
from tests import nrc_reference as ref
from tests.test_gpu_nrc import BOUND, random_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 63, 64, 65, 127, 128, 129, 255, 257, 1000, 37889])
@pytest.mark.parametrize("word", [0, 1])
def test_gradients(ctx, rows, word):
    import ctypes

    import torch
    x, y = random_inputs(40000, 5)
    c = RadianceCache(ctx, BOUND, seed=9, ema=0.0, weight_decay=0.0)
    c.gradients(x, y)   # 40,000 rows stay behind in the buffers
    d_x = torch.zeros(40000 * 12 + 1, device="cuda")
    d_x[word:word + x.size] = torch.from_numpy(x.reshape(-1)).cuda()
    d_y = torch.from_numpy(y).cuda()
    torch.cuda.synchronize()
    g, loss = np.empty(N_PARAMS, np.float32), ctypes.c_float()
    ctx.check(ctx._lib.ilm_nrc_gradients(ctx.handle, c.handle, d_x.data_ptr() + 4 * word, d_y.data_ptr(), rows,
                                         g.ctypes.data, ctypes.byref(loss)), "ilm_nrc_gradients")
    _, want_loss, want = ref.forward_backward(c.encode(x[:rows]), c.params(), y[:rows])
    assert abs(loss.value - want_loss) <= 2e-2 * want_loss
    for got, w in zip(split_params(g), want):
        assert np.linalg.norm(got - w) <= 2e-2 * np.linalg.norm(w)
    c.close()
