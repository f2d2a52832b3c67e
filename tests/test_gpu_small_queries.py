"""Queries of at most one wave, whose warps start with 1 to 32 rays: sizes on
both sides of each step against the oracle, for both widths and kinds."""
import numpy as np
import pytest

import oracle
import rs_illume_b200 as rb
from rs_illume_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def steps():
    """Ray counts around the multiples of the resident warps of 5 to 8 blocks per SM (148 SMs, 4 warps a block)."""
    out = {1, 2, 3, 31, 32, 33, 1000}
    for blocks in (5, 6, 7, 8):
        for rays in (1, 2, 4, 8, 16):
            out |= {148 * blocks * 4 * rays + k for k in (-1, 0, 1)}
    return sorted(out)


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("view", ["camera", "ball"])
def test_every_size_matches_the_oracle(ctx, width, view):
    import torch
    xyz, idx = wl.soup(31, 3000, 0.04)
    acc = rb.GpuBVHAccel(ctx, [rb.TriangleMesh(ctx, xyz, idx)], width=width)
    sc = oracle.Scene(xyz, idx)
    n = max(steps())
    if view == "camera":
        rays = wl.camera_rays(400, 400, (0.5, 0.5, -1.5), 45.0)[np.random.default_rng(1).permutation(160000)[:n]]
    else:
        rays = wl.ball_rays(9, 0, n, n, 1.0, 0.1, 4.0)
        rays["o"] += np.float32(0.5)
    rays = np.ascontiguousarray(rays)
    want = sc.intersect(rays)
    shadow = rays.copy()
    shadow["tmax"] = np.float32(1.2)
    occluded = sc.intersect_p(shadow)
    d_rays = torch.from_numpy(rays.view(np.uint8).reshape(-1, 32).copy()).cuda()
    d_shadow = torch.from_numpy(shadow.view(np.uint8).reshape(-1, 32).copy()).cuda()
    for k in steps():
        hits = torch.full((k + 1, 16), 0xA5, dtype=torch.uint8, device="cuda")
        acc.intersect_batch(d_rays[:k], hits)
        occ = torch.full((k + 1,), -7, dtype=torch.int32, device="cuda")
        acc.intersect_p_batch(d_shadow[:k], occ)
        g = hits.cpu().numpy()
        assert np.all(g[k] == 0xA5) and int(occ[k]) == -7
        g = g[:k].reshape(-1).view(rb.HIT_DTYPE)
        o = want[:k]
        differ = np.nonzero(g["prim"] != o["prim"])[0]
        assert np.all(np.abs(g["t"][differ] - o["t"][differ]) <= 1e-6 * o["t"][differ])
        same = g["prim"] == o["prim"]
        assert np.array_equal(g["t"][same], o["t"][same])
        assert np.array_equal(occ[:k].cpu().numpy().astype(np.uint8), occluded[:k])
    assert ctx.device_errors() == 0
