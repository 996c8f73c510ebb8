"""Frames queued without waits into tables that their leaf bounds nearly fill or overrun: nothing is
lost, the table grows where a frame's bound asks for it, and the map equals one made frame by frame
with a wait after each."""
import numpy as np
import pytest

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from tests.workloads import compare_maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity", [1024, 4096, 1 << 14, 1 << 16])
@pytest.mark.parametrize("records", [False, True])
def test_queue_of_frames(ctx, capacity, records):
    import torch
    w, h = 48, 36
    desc = A.sensor_desc(hres=w, vres=h, hfov_deg=90.0, vfov_deg=70.0, max_range=6.0,
                         explicit_log_odds=1, log_odds_hit=0.85, log_odds_miss=-0.4)
    sensor = A.Sensor(ctx, desc)
    g = torch.Generator(device="cuda").manual_seed(capacity)
    a = A.Map(ctx, A.map_desc(res=0.1, initial_leaf_capacity=capacity))
    b = A.Map(ctx, A.map_desc(res=0.1, initial_leaf_capacity=1 << 18))
    x = torch.rand(40, h * w, 3, generator=g, device="cuda") * 6.0 - 3.0 if records else \
        torch.rand(40, h, w, generator=g, device="cuda") * 5.5 + 0.2
    for k in range(40):  # through new ground all the time
        pose = A.Pose((0.9 * k, 0.5 * (k % 3), 0.0), (0.9, 0.0, 0.4, 0.1 * (k % 5)))
        for m, flags in ((a, 0), (b, N.NM_SYNC)):
            if records:
                m.insert_points(sensor, pose, x[k], w, h, 12, flags=flags)
            else:
                m.insert_ranges(sensor, pose, x[k], flags=flags)
    sa, sb = a.stats(), b.stats()
    assert sa["error_flags"] == 0 and sa["leaf_count"] == sb["leaf_count"]
    assert sa["leaf_count"] <= sa["leaf_capacity"] * 7 // 8
    for k in ("visits", "rays", "unique_voxels", "touched_leaves"):
        assert sa[k] == sb[k]
    errs = compare_maps(a.export(), b.export())
    assert not errs, "; ".join(errs[:4])
