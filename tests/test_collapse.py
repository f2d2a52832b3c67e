"""Collapse of the binary tree into wide nodes (csrc/builder.cpp,
CollapsePlan): every primitive in one leaf, children inside their boxes, and
the emitted tree's cost equal to the optimum of an independent recursion."""
import functools

import numpy as np
import pytest

from rs_illume_b200 import workloads as wl
from tests.layout_utils import host_layout

PRIM_COST, MAX_LEAF = 1.5, 4


def line():
    """Degenerate: all triangles on one line, boxes without area."""
    x = np.arange(90, dtype=np.float32)
    return np.stack([x, 0 * x, 0 * x], 1), np.arange(90, dtype=np.uint32).reshape(-1, 3)


def copies():
    """Forty copies of one triangle: binary leaves of more primitives than a leaf child holds."""
    return np.tile(np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32), (40, 1)), \
        np.arange(120, dtype=np.uint32).reshape(-1, 3)


def far_apart():
    """Coordinates near the float range: areas overflow."""
    xyz, idx = wl.soup(4, 60, 0.1)
    return ((xyz - np.float32(0.5)) * np.float32(3e29)).astype(np.float32), idx


SCENES = {"soup": lambda: wl.soup(2, 700, 0.05), "ico": lambda: wl.icosphere(3, 2), "one": lambda: wl.soup(2, 1, 0.1),
          "five": lambda: wl.soup(2, 5, 0.1), "line": line, "copies": copies, "far_apart": far_apart}


def area(lo, hi):
    d = (hi - lo).astype(np.float64)
    return d[0] * d[1] + d[1] * d[2] + d[2] * d[0]


@pytest.mark.parametrize("max_prims", [1, 4, 9])
@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_collapse(name, width, max_prims):
    xyz, idx = SCENES[name]()
    lay = host_layout(xyz, idx, width, max_prims)
    nodes, recs, bin_nodes = lay["nodes"], lay["records"], lay["bin"]
    tri = np.stack([recs["p0"], recs["p1"], recs["p2"]], 1)
    used = np.zeros(len(recs), int)
    fills = []

    def walk(k):
        """(cost, lower corner, upper corner) of wide node k."""
        nd, cost, los, his = nodes[k], 0.0, [], []
        fill = 0
        for c in range(width):
            m = int(nd["meta"][c])
            if m == 0:
                continue
            fill += 1
            if (int(nd["packed"]) >> (24 + c)) & 1:
                cc, lo, hi = walk(int(nd["child_base"]) + (m & 31))
            else:
                n, first = m >> 5, int(nd["prim_base"]) + (m & 31)
                assert 1 <= n <= MAX_LEAF
                used[first:first + n] += 1
                t = tri[first:first + n].reshape(-1, 3)
                lo, hi = t.min(0), t.max(0)
                cc = area(lo, hi) * PRIM_COST * n
            cost += cc
            los.append(lo)
            his.append(hi)
        fills.append(fill)
        lo, hi = np.min(los, 0), np.max(his, 0)
        return cost + area(lo, hi), lo, hi

    cost = walk(0)[0]
    assert np.all(used == 1)
    assert sorted(recs["prim"].tolist()) == list(range(len(idx)))
    if name in ("line", "copies", "far_apart") or np.any(bin_nodes["n_prims"] > MAX_LEAF) or len(bin_nodes) == 1:
        return   # every split costs the same, or leaves are halved beyond the plan

    def children(i):
        return i + 1, int(bin_nodes[i]["offset"])

    @functools.lru_cache(maxsize=None)
    def count(i):
        return int(bin_nodes[i]["n_prims"]) or sum(map(count, children(i)))

    @functools.lru_cache(maxsize=None)
    def best(i, k):
        nd = bin_nodes[i]
        a = area(nd["bmin"], nd["bmax"])
        leaf = a * PRIM_COST * count(i) if count(i) <= MAX_LEAF else np.inf
        if nd["n_prims"]:
            return leaf
        left, right = children(i)

        def split(n):
            return min(best(left, j) + best(right, n - j) for j in range(1, n))
        if k == 1:
            return min(leaf, a + split(width))
        return min(best(i, k - 1), split(k))

    root = bin_nodes[0]
    want = best(0, 1)
    if count(0) <= MAX_LEAF:   # a root leaf still sits in a node
        want = min(want, best(0, 1)) + (0 if want != area(root["bmin"], root["bmax"]) * PRIM_COST * count(0)
                                        else area(root["bmin"], root["bmax"]))
    assert cost == pytest.approx(want, rel=1e-5)   # float32 sums in the plan: a few ulps per level
    assert fills[-1] >= 1
