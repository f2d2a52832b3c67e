"""Surface-interaction records at the edges of a warp's block of 32 records,
from buffers on 16-byte boundaries and from buffers that are not: every field
equals the oracle's bit for bit, and no byte past the last record is written."""
import numpy as np
import pytest

import rs_illume_b200 as rb
from rs_illume_b200 import _lib
from tests.test_interaction import FIELDS, oracle_record, scene

pytestmark = pytest.mark.gpu
REC = 176


def at_word(data, word):
    """`data` on the device, `word` 4-byte words past a 16-byte boundary."""
    import torch
    raw = np.ascontiguousarray(data).view(np.uint8).reshape(-1)
    buf = torch.zeros(raw.size + 64, dtype=torch.uint8, device="cuda")
    buf[4 * word: 4 * word + raw.size] = torch.from_numpy(raw.copy()).cuda()
    return buf, buf.data_ptr() + 4 * word


@pytest.mark.parametrize("words", [(0, 0, 0), (1, 0, 0), (0, 2, 0), (0, 0, 3)])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 300])
def test_records_match_the_oracle(ctx, n, words):
    import torch
    xyz, idx, rays, extra = scene(22, True)
    acc = rb.GpuBVHAccel(ctx, [rb.TriangleMesh(ctx, xyz, idx, **extra)], width=8)
    hits = acc.intersect_batch(rays)
    pick = np.concatenate([np.nonzero(hits["prim"] != rb.ILM_MISS)[0][:n - n // 4],
                           np.nonzero(hits["prim"] == rb.ILM_MISS)[0][:n // 4]])
    pick = np.random.default_rng(n).permutation(pick)
    assert len(pick) == n
    rays, hits = np.ascontiguousarray(rays[pick]), np.ascontiguousarray(hits[pick])
    keep_r, p_rays = at_word(rays, words[0])
    keep_h, p_hits = at_word(hits, words[1])
    out = torch.full((n * REC + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    first = 4 * words[2]
    torch.cuda.synchronize()
    ctx.check(ctx._lib.ilm_surface_interactions(ctx.handle, acc.id, p_rays, p_hits, n, out.data_ptr() + first,
                                                _lib.CUDA_STREAM_LEGACY), "ilm_surface_interactions")
    raw = out.cpu().numpy()
    assert np.all(raw[:first] == 0xA5) and np.all(raw[first + n * REC:] == 0xA5)
    si = raw[first:first + n * REC].copy().view(_lib.SURFACE_INTERACTION_DTYPE)
    for i in range(n):
        assert si["prim"][i] == hits["prim"][i]
        if hits["prim"][i] == rb.ILM_MISS:
            assert si["kind"][i] == _lib.SI_MISS and not si["p"][i].any() and not si["shading_dndv"][i].any()
            continue
        want = oracle_record(xyz, idx, int(hits["prim"][i]), rays[i], extra)
        assert si["kind"][i] == _lib.SI_TRIANGLE
        for f in FIELDS:
            assert np.array_equal(si[f][i], want[f]), (i, f, si[f][i], want[f])


def test_meshes_with_and_without_attributes(ctx):
    """One accel of meshes with all attributes, some and none: every combination in one vertex table."""
    xyz, idx, rays, extra = scene(23, True)
    kinds = [{}, extra, {"n": extra["n"]}, {"uv": extra["uv"], "s": extra["s"]}]
    shift = [np.float32([k, 0, 0]) for k in range(len(kinds))]
    acc = rb.GpuBVHAccel(ctx, [rb.TriangleMesh(ctx, xyz + d, idx, **kw) for d, kw in zip(shift, kinds)], width=8)
    rays = np.concatenate([rays] * len(kinds))
    for k, d in enumerate(shift):
        rays["o"][k * len(rays) // len(kinds): (k + 1) * len(rays) // len(kinds)] += d
    hits = acc.intersect_batch(rays)
    si = acc.surface_interactions(rays, hits)
    picked = np.random.default_rng(3).permutation(np.nonzero(hits["prim"] != rb.ILM_MISS)[0])[:1200]
    seen = set()
    for i in picked:
        mesh, prim = divmod(int(hits["prim"][i]), len(idx))
        seen.add(mesh)
        want = oracle_record(xyz + shift[mesh], idx, prim, rays[i], kinds[mesh])
        assert si["kind"][i] == _lib.SI_TRIANGLE
        for f in FIELDS:
            assert np.array_equal(si[f][i], want[f]), (i, mesh, f, si[f][i], want[f])
    assert seen == {0, 1, 2, 3}
