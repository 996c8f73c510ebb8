"""Tick plans of one to the most sensors, some of a single tile: every sensor's rendered ranges and
the shared map equal solo renders and inserts (a tile finds its sensor among all of them)."""
import numpy as np
import pytest
import torch

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from nanomap_b200 import scenes as S
from tests.workloads import compare_maps

pytestmark = pytest.mark.gpu

SIZES = [(7, 5), (33, 17), (16, 16), (48, 8), (1, 1), (64, 48)]


@pytest.mark.parametrize("n", [1, 2, 5, 31, 32])
def test_every_slot(ctx, n):
    scene = S.make_scene(S.SCENES["plain_small"], 1)
    sim = A.SimMap(ctx, 0.05, boxes=scene.boxes, cylinders=scene.cylinders, vox_min=(0, 0, 0),
                   vox_max=(400, 400, 100))
    sensors, bufs, poses = [], [], []
    for i in range(n):
        w, h = SIZES[i % len(SIZES)]
        d = A.sensor_desc(hres=w, vres=h, hfov_deg=87, vfov_deg=58, max_range=4.0 + i % 3,
                          explicit_log_odds=1, log_odds_hit=0.85, log_odds_miss=-0.4,
                          frame_transform=S.OPTICAL_TO_BODY)
        sensors.append(A.Sensor(ctx, d))
        bufs.append(torch.zeros(h, w, device="cuda"))
        poses.append([A.Pose(p, q) for p, q in S.trajectory(scene, 2, seed=3 + i)])
    m = A.Map(ctx, A.map_desc(res=0.05, max_agents=n))
    solo = A.Map(ctx, A.map_desc(res=0.05))
    plan = A.TickPlan(m, [(sensors[i], bufs[i], i) for i in range(n)], sim=sim)
    for t in range(2):
        for i in range(n):
            plan.set_pose(i, poses[i][t])
        plan.run()
        torch.cuda.synchronize()
        for i in range(n):
            r = torch.zeros_like(bufs[i])
            sim.render(sensors[i], poses[i][t], r)
            solo.insert_ranges(sensors[i], poses[i][t], r)
            torch.cuda.synchronize()
            assert np.array_equal(r.cpu().numpy().view(np.uint32), bufs[i].cpu().numpy().view(np.uint32)), i
    errs = compare_maps(m.export(), solo.export())
    assert not errs, "; ".join(errs[:4])
