"""The tuner on a sample for which the occupancy flag selects nothing: it is
never reported as a choice, whatever the timings."""
import pytest

import rs_illume_b200 as rb
from rs_illume_b200 import batch as bt
from rs_illume_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("any_hit", [False, True])
def test_idle_flag_is_not_a_choice(ctx, any_hit):
    xyz, idx = wl.icosphere(5, 2)
    rays = wl.ball_rays(2, 4, 1 << 20, 1 << 19)
    mesh = rb.TriangleMesh(ctx, xyz, idx)
    for _ in range(5):
        r = bt.autotune(ctx, [mesh], rays, any_hit, force=True)
        assert not r["high_occupancy"] and r["n_tried"] == 13
