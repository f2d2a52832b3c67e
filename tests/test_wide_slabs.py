"""Child slab tests of the wide layouts (csrc/wide_tracer.cuh, axis_slab).

CPU: the kernel's arithmetic, restated in numpy with one float32 rounding per
operation, accepts every child whose exact box the ray meets (in float64), for
nodes of scenes of several sizes and places and rays with zero, tiny and
ordinary direction components.
GPU: closest and any hit on such rays against the oracle: the same rays hit,
no hit is farther than the oracle's by more than a near-tie (1e-6 of t), equal
primitives have equal t and u, and occlusion is the oracle's."""
import numpy as np
import pytest

import oracle
import rs_illume_b200 as rb
from rs_illume_b200 import workloads as wl
from tests.layout_utils import host_layout

F = np.float32
PLACES = {"unit": (1.0, 0.0), "far": (1.0, 1000.0), "tiny": (2.0 ** -30, 0.0), "huge": (2.0 ** 30, 0.0),
          "tiny_far": (2.0 ** -12, 1.0)}


def fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def placed(place, kind):
    scale, shift = PLACES[place]
    xyz, idx = wl.icosphere(3, 2, 0.05, 1.0) if kind == "ico" else wl.soup(3, 1500, 0.05)
    return (xyz * F(scale) + F(shift)).astype(F), idx


def odd_rays(xyz, n, seed):
    """Rays around the scene: all directions, directions with zero components, with components of 1e-6 and 1e-30 of
    the others, and origins on coordinates of the scene's own vertices."""
    rng = np.random.default_rng(seed)
    lo, hi = xyz.min(0).astype(np.float64), xyz.max(0).astype(np.float64)
    r = np.zeros(n, rb.RAY_DTYPE)
    o = lo + (hi - lo) * (rng.random((n, 3)) * 3 - 1)
    on = rng.random((n, 3)) < 0.3
    r["o"] = np.where(on, xyz[rng.integers(0, len(xyz), n)], o.astype(F))
    d = rng.normal(size=(n, 3))
    pick = rng.integers(0, 4, n)[:, None]
    weak = rng.random((n, 3)) < 0.5
    weak[np.arange(n), rng.integers(0, 3, n)] = False
    d = np.where(weak & (pick == 1), 0.0, np.where(weak & (pick == 2), d * 1e-6, np.where(weak & (pick == 3),
                                                                                          d * 1e-30, d)))
    r["d"] = d.astype(F)
    r["tmax"] = np.inf
    return r


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("place", sorted(PLACES))
@pytest.mark.parametrize("kind", ["ico", "soup"])
def test_every_met_child_is_accepted(width, place, kind):
    xyz, idx = placed(place, kind)
    lay = host_layout(xyz, idx, width)
    nodes, recs = lay["nodes"], lay["records"]
    rays = odd_rays(xyz, 3000, 5)
    tri = np.stack([recs["p0"], recs["p1"], recs["p2"]], 1)
    bounds = {}

    def bound(k):
        if k not in bounds:
            nd, got = nodes[k], []
            for c in range(width):
                m = int(nd["meta"][c])
                if m == 0:
                    got.append(None)
                elif (int(nd["packed"]) >> (24 + c)) & 1:
                    b = [x for x in bound(int(nd["child_base"]) + (m & 31)) if x is not None]
                    got.append((np.min([x[0] for x in b], 0), np.max([x[1] for x in b], 0)))
                else:
                    t = tri[int(nd["prim_base"]) + (m & 31):][:m >> 5].reshape(-1, 3)
                    got.append((t.min(0), t.max(0)))
            bounds[k] = got
        return bounds[k]

    bound(0)
    with np.errstate(all="ignore"):
        inv = np.clip(F(1) / rays["d"], F(-2.0 ** 80), F(2.0 ** 80))
        met_all = 0
        for k in np.random.default_rng(1).permutation(len(nodes))[:60]:
            nd = nodes[k]
            near, far, tn64, tf64 = [], [], [], []
            for a in range(3):
                s = F(2.0 ** (((int(nd["packed"]) >> (8 * a)) & 0xFF) - 127))
                start = fma(F(8388608.0), s, nd["origin"][a])
                slope = s * inv[:, a]
                b = fma(F(-32768.0), slope, (start - rays["o"][:, a]) * inv[:, a])
                margin = fma(np.abs(start), F(2.0 ** -22), s * F(2.0 ** -6))
                nb, fb = fma(-margin, np.abs(inv[:, a]), b), fma(margin, np.abs(inv[:, a]), b)
                neg = (inv[:, a] < 0)[:, None]
                qn = np.where(neg, nd["qhi"][a], nd["qlo"][a]).astype(F) + F(32768)
                qf = np.where(neg, nd["qlo"][a], nd["qhi"][a]).astype(F) + F(32768)
                near.append(fma(qn, slope[:, None], nb[:, None]))
                far.append(fma(qf, slope[:, None], fb[:, None]))
                box = np.array([(0, 0) if x is None else (x[0][a], x[1][a]) for x in bound(k)], np.float64)
                o, d = rays["o"][:, a, None].astype(np.float64), rays["d"][:, a, None].astype(np.float64)
                t0, t1 = (box[None, :, 0] - o) / d, (box[None, :, 1] - o) / d
                inside = (box[None, :, 0] <= o) & (o <= box[None, :, 1])
                tn64.append(np.where(d == 0, np.where(inside, -np.inf, np.inf), np.minimum(t0, t1)))
                tf64.append(np.where(d == 0, np.where(inside, np.inf, -np.inf), np.maximum(t0, t1)))
            tn = np.fmax(np.fmax(np.fmax(near[0], near[1]), near[2]), F(0))
            tf = np.fmin(np.fmin(far[0], far[1]), far[2]) * F(1 + 2.0 ** -20)
            there = np.array([x is not None for x in bound(k)])
            met = (np.maximum(np.max(tn64, 0), 0.0) <= np.min(tf64, 0)) & there[None, :]
            met_all += int(met.sum())
            assert np.all(tn[met] <= tf[met])
            # and the entry distance, which orders and culls children, is not beyond the exact one
            exact = np.maximum(np.max(tn64, 0), 0.0)
            assert np.all(tn[met] <= exact[met] * (1 + 1e-6) + 1e-30)
    assert met_all > 100


@pytest.mark.gpu
@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("place", sorted(PLACES))
def test_gpu_matches_the_oracle(ctx, width, place):
    xyz, idx = placed(place, "ico")
    acc = rb.GpuBVHAccel(ctx, [rb.TriangleMesh(ctx, xyz, idx)], width=width)
    sc = oracle.Scene(xyz, idx)
    rays = odd_rays(xyz, 20000, 7)
    g, o = acc.intersect_batch(rays), sc.intersect(rays)
    hit = o["prim"] != rb.ILM_MISS
    assert hit.sum() > 1000
    assert np.array_equal(g["prim"] != rb.ILM_MISS, hit)
    # never farther than the oracle's hit, up to a near-tie; where nearer, the triangle is met there in float64 (a
    # hit on an edge that lies in its box's face, which the exact boxes can lose and the wide layouts' boxes keep)
    assert np.all(g["t"][hit] <= o["t"][hit] * F(1 + 1e-6))
    near = np.nonzero(hit & (g["t"] < o["t"] * F(1 - 1e-6)))[0]
    v = xyz[idx[g["prim"][near]]].astype(np.float64)
    e1, e2, d = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0], rays["d"][near].astype(np.float64)
    s, p = rays["o"][near].astype(np.float64) - v[:, 0], np.cross(d, e2)
    q, det = np.cross(s, e1), np.sum(p * e1, 1)
    b1, b2, t = np.sum(s * p, 1) / det, np.sum(d * q, 1) / det, np.sum(e2 * q, 1) / det
    assert np.all((b1 > -1e-6) & (b2 > -1e-6) & (b1 + b2 < 1 + 1e-6) & (np.abs(t - g["t"][near]) <= 1e-5 * t))
    same = hit & (g["prim"] == o["prim"])
    assert np.array_equal(g["t"][same], o["t"][same]) and np.array_equal(g["u"][same], o["u"][same])
    r = rays.copy()
    r["tmax"] = np.where(hit, np.nan_to_num(o["t"], posinf=1.0), F(1.0)) * np.random.default_rng(3).choice(
        np.array([0.5, 0.999, 1.001, 2.0], F), len(r))
    r = np.delete(r, near)   # their nearer hits are the oracle's misses
    assert np.array_equal(acc.intersect_p_batch(r).astype(np.uint8), sc.intersect_p(r))
    assert ctx.device_errors() == 0
