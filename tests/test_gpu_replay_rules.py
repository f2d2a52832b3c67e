"""Renders on both sides of the rules that choose between CUDA graphs and
direct launches (four waves, four cache frames): images and ray counts agree."""
import numpy as np
import pytest

import rs_illume_b200 as rb
from rs_illume_b200 import workloads as wl
from rs_illume_b200.nrc import RadianceCache

pytestmark = pytest.mark.gpu
W = H = 64
SPP = 16


@pytest.fixture(scope="module")
def tracer():
    xyz, idx, mat, alb, emi = wl.cornell(6, 3)
    ctx = rb.Context(0)
    acc = rb.GpuBVHAccel(ctx, [rb.TriangleMesh(ctx, xyz, idx)], width=8)
    cam = wl.CORNELL_CAMERA
    yield rb.PathTracer(acc, mat, alb, emi, cam["eye"], cam["fov_deg"], W, H), acc.world_bound(), ctx
    ctx.close()


def wave_paths(waves):
    """Paths per wave that split a render into `waves` waves, the last one shorter."""
    return -(-W * H * SPP // waves) + (1 if W * H * SPP % waves == 0 else 0)


@pytest.mark.parametrize("waves", [1, 3, 4, 5, 9])
def test_replayed_bounces_equal_direct_ones(tracer, waves):
    pt, _, _ = tracer
    kw = {"seed": 9, "wave_paths": wave_paths(waves)} if waves > 1 else {"seed": 9}
    a, sa = pt.render(SPP, use_graphs=True, **kw)
    b, sb = pt.render(SPP, use_graphs=False, **kw)
    whole, _ = pt.render(SPP, seed=9, use_graphs=False)
    assert sa["waves"] == sb["waves"] == waves
    # same random numbers; only the order of the film's float atomics differs
    np.testing.assert_allclose(a, b, rtol=2e-5, atol=2e-6)
    np.testing.assert_allclose(a, whole, rtol=2e-5, atol=2e-6)
    assert sa["closest_rays"] == sb["closest_rays"] and sa["shadow_rays"] == sb["shadow_rays"]


def test_frames_on_both_sides_of_the_rule(tracer):
    """Without queries and training a render's frames are sums of non-negative
    path contributions, so what frame f adds to the first f of them is
    non-negative at each pixel, whichever way either render was launched."""
    pt, bound, ctx = tracer
    cache = RadianceCache(ctx, bound)
    total, rays = np.zeros((H, W, 3)), 0
    per_frame = []
    for frames in range(1, 8):
        img, st = pt.render_nrc(cache, frames=frames, spp_per_frame=4, seed=5, spread_c=1e30, train=False)
        assert st["frames"] == frames and st["queries"] == 0
        now = img.astype(np.float64) * frames
        # the sums' rounding: about a hundred float additions a pixel
        assert np.all(now - total >= -1e-4 * (1.0 + now)), frames
        per_frame.append(st["closest_rays"] + st["shadow_rays"] - rays)
        total, rays = now, st["closest_rays"] + st["shadow_rays"]
    assert max(per_frame) < 1.03 * min(per_frame)
    cache.close()


@pytest.mark.parametrize("frames", [3, 4])
def test_frames_with_the_cache(tracer, frames):
    pt, bound, ctx = tracer
    cache = RadianceCache(ctx, bound, seed=4)
    w0 = cache.params().copy()
    img, st = pt.render_nrc(cache, frames=frames, spp_per_frame=4, seed=7)
    assert st["frames"] == frames and st["queries"] > 0 and st["train_samples"] > 0
    assert np.all(np.isfinite(img)) and img.min() >= 0.0
    assert np.isfinite(st["last_loss"]) and not np.array_equal(cache.params(), w0)
    cache.close()
