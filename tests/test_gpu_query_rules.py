"""Query sizes on both sides of the rules that choose rays per warp, schedule
and build (148 SMs): the default, lane refill and the occupancy flag give the
records of the lone one-thread-per-ray traversal, and write nothing past them."""
import numpy as np
import pytest

import rs_illume_b200 as rb
from rs_illume_b200 import workloads as wl
from rs_illume_b200._lib import HIT_DTYPE
from tests.test_gpu_trace import compare_closest

pytestmark = pytest.mark.gpu

SMS = 148
WARPS = SMS * 7 * 4                                            # resident warps at 7 blocks per SM
EDGES = [WARPS * r * (16 - r) // 16 for r in (1, 2, 4, 8)] + [WARPS * 16, SMS * 5 * 128, WARPS * 32, WARPS * 32 * 3,
                                                              WARPS * 32 * 6]
FLAGS = ({}, {"lane_refill": True}, {"high_occupancy": True})


@pytest.fixture(scope="module")
def lone():
    """(mesh data, device rays, hits and flags by width) of the traversal without split tail."""
    import torch
    xyz, idx = wl.icosphere(5, 2)
    n = max(EDGES) + 1
    rays = np.ascontiguousarray(wl.ball_rays(5, 4, 2 * n, n)[n // 2: n // 2 + n])   # tmax infinite and finite
    d_rays = torch.from_numpy(rays.view(np.uint8)).cuda()
    ctx = rb.Context(0, grid_schedule=True, tail_split=False)
    want = {}
    for width in (4, 8):
        acc = rb.GpuBVHAccel(ctx, [rb.TriangleMesh(ctx, xyz, idx)], width=width)
        hits = torch.empty(n * 16, dtype=torch.uint8, device="cuda")
        occ = torch.empty(n, dtype=torch.int32, device="cuda")
        acc.intersect_batch(d_rays, hits)
        acc.intersect_p_batch(d_rays, occ)
        want[width] = hits.cpu().numpy().view(HIT_DTYPE), occ.cpu().numpy()
    ctx.close()
    return xyz, idx, d_rays, want


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("flags", FLAGS, ids=["default", "lane_refill", "high_occupancy"])
def test_sizes_around_the_rules(lone, flags, width):
    import torch
    xyz, idx, d_rays, both = lone
    want, flag = both[width]
    ctx = rb.Context(0, **flags)
    acc = rb.GpuBVHAccel(ctx, [rb.TriangleMesh(ctx, xyz, idx)], width=width)
    for n in sorted({e + k for e in EDGES for k in (-1, 0, 1)}):
        sub = d_rays[:32 * n]
        hits = torch.full((16 * n + 16,), 0xA5, dtype=torch.uint8, device="cuda")
        occ = torch.full((n + 1,), -7, dtype=torch.int32, device="cuda")
        acc.intersect_batch(sub, hits)
        acc.intersect_p_batch(sub, occ)
        g = hits.cpu().numpy()
        assert np.all(g[16 * n:] == 0xA5) and int(occ[n]) == -7
        assert np.array_equal(occ[:n].cpu().numpy(), flag[:n]), n
        # equal distances, where the split keeps the smaller primitive id, are the only difference
        assert compare_closest(g[:16 * n].view(HIT_DTYPE), want[:n], label=f"{n}") <= 16
    assert ctx.device_errors() == 0
    ctx.close()
