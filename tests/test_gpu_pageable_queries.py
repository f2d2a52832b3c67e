"""Queries on pageable host buffers, staged through the context's pinned block
once enough rays have come in: sizes around the rule's threshold, the chunks'
edges and the block's capacity, against the device path, byte for byte."""
import numpy as np
import pytest

import rs_illume_b200 as rb
from rs_illume_b200 import workloads as wl
from rs_illume_b200._lib import HIT_DTYPE

pytestmark = pytest.mark.gpu

RENT = 2 << 20                   # pageable rays after which the block is made
MOST = (8 << 20) // 4 // 48      # rays of the largest chunk


def sizes():
    out = {8191, 8192, 8193, 4096 * 4 + 1, MOST * 4 + 1, MOST * 8 - 1}
    for n in (8 * 4096, 8 * MOST // 1024 * 1024):
        out |= {n - 1, n, n + 1}
    return sorted(out) + [RENT + 77]


def aligned(n, dtype, fill):
    """n records and 64 bytes more, 16-byte aligned, all bytes `fill`."""
    raw = np.full(n * np.dtype(dtype).itemsize + 80, fill, np.uint8)
    at = -raw.ctypes.data % 16
    return raw[at: at + n * np.dtype(dtype).itemsize + 64]


@pytest.mark.parametrize("chunk", [1 << 19, 5000])
@pytest.mark.parametrize("layout", ["bvh8", "kd"])
def test_pageable_queries_match_the_device_path(layout, chunk):
    import torch
    ctx = rb.Context(0)
    ctx.check(ctx._lib.ilm_context_set_stage_chunk(ctx.handle, chunk), "ilm_context_set_stage_chunk")
    xyz, idx = wl.icosphere(5, 2)
    mesh = [rb.TriangleMesh(ctx, xyz, idx)]
    acc = rb.GpuBVHAccel(ctx, mesh, width=8) if layout == "bvh8" else rb.GpuKdTreeAccel(ctx, mesh)
    rays = np.ascontiguousarray(wl.ball_rays(2, 4, RENT + 77, 1 << 19))
    d_rays = torch.from_numpy(rays.view(np.uint8)).cuda()
    d_hits = torch.empty(len(rays) * 16, dtype=torch.uint8, device="cuda")
    d_occ = torch.empty(len(rays) * 4, dtype=torch.uint8, device="cuda")
    acc.intersect_batch(d_rays, d_hits)
    acc.intersect_p_batch(d_rays, d_occ)
    want_h, want_o = d_hits.cpu().numpy(), d_occ.cpu().numpy()
    for n in [10000] + [RENT] + sizes():        # the first before the block is there, the second makes it
        k0 = min(3, len(rays) - n)
        sub = rays[k0: k0 + n]
        h = aligned(n, HIT_DTYPE, 0xA5)
        acc.intersect_batch(sub, h[:16 * n].view(HIT_DTYPE))
        assert np.array_equal(h[:16 * n], want_h[16 * k0: 16 * (k0 + n)]) and np.all(h[16 * n:] == 0xA5)
        o = aligned(n, np.uint32, 0xA5)
        acc.intersect_p_batch(sub, o[:4 * n].view(np.uint32))
        assert np.array_equal(o[:4 * n], want_o[4 * k0: 4 * (k0 + n)]) and np.all(o[4 * n:] == 0xA5)
    # pinned rays into pageable results, and the other way round
    n = 100003
    pin_r = torch.from_numpy(rays[:n].view(np.uint8)).pin_memory()
    assert np.array_equal(acc.intersect_batch(pin_r.numpy().view(rays.dtype)).view(np.uint8), want_h[:16 * n])
    pin_h = torch.zeros(16 * n, dtype=torch.uint8).pin_memory()
    acc.intersect_batch(rays[:n], pin_h.numpy().view(HIT_DTYPE))
    assert np.array_equal(pin_h.numpy(), want_h[:16 * n])
    assert ctx.device_errors() == 0
    ctx.close()


def test_contexts_on_several_threads():
    import threading
    xyz, idx = wl.icosphere(4, 2)
    rays = np.ascontiguousarray(wl.ball_rays(2, 4, RENT, 1 << 19))
    ctx = rb.Context(0)
    want = rb.GpuBVHAccel(ctx, [rb.TriangleMesh(ctx, xyz, idx)], width=8).intersect_batch(rays[:40000]).tobytes()
    ctx.close()
    bad = []

    def work():
        c = rb.Context(0)
        acc = rb.GpuBVHAccel(c, [rb.TriangleMesh(c, xyz, idx)], width=8)
        acc.intersect_batch(rays)
        for _ in range(20):
            if acc.intersect_batch(rays[:40000]).tobytes() != want:
                bad.append(1)
        c.close()

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
