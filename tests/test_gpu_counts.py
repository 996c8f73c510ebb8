"""Accumulate mode (a voxel's hits and misses of a frame all count) against the CPU oracle, map and
counters bit-identical: one pixel, partial tiles, a beam so narrow that every ray of a tile crosses
the same voxels, tiles with more leaves than the shared table has entries, and a reach past the
leaf codes'."""
import numpy as np
import pytest
import torch

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from nanomap_b200 import scenes as S
from oracle import oracle as O
from tests.workloads import compare_maps, oracle_frame

pytestmark = pytest.mark.gpu

FRAMES = {  # width, height, horizontal and vertical field of view (degrees), range (m), voxel (m)
    "pixel": (1, 1, 60.0, 40.0, 6.0, 0.05),
    "beam": (16, 8, 0.4, 0.2, 6.0, 0.05),
    "partial": (75, 50, 60.0, 40.0, 5.0, 0.05),
    "spread": (17, 9, 100.0, 80.0, 30.0, 0.05),
    "fine": (40, 8, 90.0, 20.0, 4.0, 0.01),
    "wide": (5, 3, 30.0, 20.0, 9.0, 0.002),
}


@pytest.mark.parametrize("frame", sorted(FRAMES))
@pytest.mark.parametrize("rounding", [N.NM_ROUND_DOWN, N.NM_ROUND_NEAREST])
@pytest.mark.parametrize("eye", [(0.137, -0.218, 0.391), (1.0, -0.05, 2.0), (-211.37, 93.21, 17.77)])
def test_counts(ctx, frame, rounding, eye):
    w, h, hfov, vfov, rng_m, res = FRAMES[frame]
    desc = A.sensor_desc(hres=w, vres=h, hfov_deg=hfov, vfov_deg=vfov, max_range=rng_m,
                         explicit_log_odds=1, log_odds_hit=0.85, log_odds_miss=-0.4,
                         frame_transform=S.OPTICAL_TO_BODY)
    sensor, osen = A.Sensor(ctx, desc), O.Sensor.from_desc(desc)
    m = A.Map(ctx, A.map_desc(res=res, rounding=rounding, update_mode=N.NM_UPDATE_ACCUMULATE))
    om = O.Map(res, rounding=rounding, update_mode=1)
    for k in range(2):
        rng = np.random.default_rng(k)
        r = rng.uniform(0.3 * rng_m, rng_m, (h, w)).astype(np.float32) if k else \
            np.full((h, w), 0.9 * rng_m, np.float32)
        if h * w > 1:
            r[rng.uniform(size=r.shape) < 0.05] = 0.0
            r[rng.uniform(size=r.shape) < 0.05] = np.float32(rng_m)             # dropped
            r[rng.uniform(size=r.shape) < 0.05] = np.float32(rng_m - 1.2 * res)  # ends near the range
        q = rng.normal(size=4)
        pose = A.Pose(eye, tuple(q / np.linalg.norm(q)))
        m.insert_ranges(sensor, pose, torch.from_numpy(r).cuda())
        R, e, mt = oracle_frame(desc, pose, res, rounding)
        om.insert(R, e, mt, desc.log_odds_hit, desc.log_odds_miss, osen.points(r))
    errs = compare_maps(m.export(), om.export())
    assert not errs, "; ".join(errs[:4])
    st, ost = m.stats(), om.stats()
    for k in ("visits", "rays", "unique_voxels"):
        assert st[k] == ost[k], k
