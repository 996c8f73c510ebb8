"""Accumulate mode on each of its routes -- counted in shared memory, table-free in a tile whose rays fan
out, table-free for large images and for reaches past the leaf codes' -- against the CPU oracle, the map,
its leaves and the counters bit-identical."""
import numpy as np
import pytest
import torch

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from oracle import oracle as O
from tests.workloads import compare_maps, oracle_frame

pytestmark = pytest.mark.gpu

IDENTITY = np.eye(3, dtype=np.float32).reshape(-1)
# width, height, horizontal and vertical spread of the directions, lengths (voxels), range (voxels)
FRAMES = {
    "table": (40, 20, 0.3, 0.2, (10.0, 60.0), 70.0),
    "table_full": (33, 17, 1.2, 0.8, (30.0, 60.0), 70.0),       # fans of about the limit
    "fan": (33, 17, 3.0, 2.0, (100.0, 400.0), 500.0),
    "mixed": (64, 32, 1.0, 1.0, (2.0, 400.0), 500.0),           # short on the left, long on the right
    "tiles_4096": (1024, 512, 0.6, 0.4, (2.0, 6.0), 9.0),       # the most tiles that keep the table
    "tiles_4160": (1040, 512, 0.6, 0.4, (2.0, 6.0), 9.0),
    "ragged_large": (1041, 523, 0.6, 0.4, (2.0, 6.0), 9.0),
    "beyond": (5, 3, 0.5, 0.3, (100.0, 4400.0), 4500.0),
}


def _points(name, res, seed):
    w, h, a, b, (near, far), _ = FRAMES[name]
    u, v = np.meshgrid(np.linspace(-a, a, w), np.linspace(-b, b, h))
    d = np.stack([np.ones_like(u), u, v], -1)
    rng = np.random.default_rng(seed)
    t = np.linspace(0.0, 1.0, w)[None, :, None] ** 3 if name == "mixed" else rng.uniform(size=(h, 1, 1))
    r = near + (far - near) * np.clip(t + 0.05 * rng.uniform(size=(h, w, 1)), 0.0, 1.0)
    p = d / np.linalg.norm(d, axis=2, keepdims=True) * r * res
    p[rng.uniform(size=(h, w)) < 0.02] = np.nan
    return p.astype(np.float32)


@pytest.mark.parametrize("frame", sorted(FRAMES))
@pytest.mark.parametrize("rounding", [N.NM_ROUND_DOWN, N.NM_ROUND_NEAREST])
@pytest.mark.parametrize("filtered", [False, True])
def test_routes(ctx, frame, rounding, filtered):
    if filtered and frame == "beyond":
        pytest.skip("the voxel filter does not take this range")
    w, h, _, _, _, reach = FRAMES[frame]
    res = 0.05
    desc = A.sensor_desc(hres=w, vres=h, max_range=reach * res, explicit_log_odds=1, log_odds_hit=0.85,
                         log_odds_miss=-0.4)
    sensor = A.Sensor(ctx, desc)
    m = A.Map(ctx, A.map_desc(res=res, rounding=rounding, update_mode=N.NM_UPDATE_ACCUMULATE))
    om = O.Map(res, rounding=rounding, update_mode=1)
    for k in range(2):
        pts = _points(frame, res, k)
        rec = np.zeros((h, w, 4), np.float32)
        rec[..., :3] = pts
        pose = A.Pose((0.137 + 0.3 * k, -0.218, 0.391), (0.9, 0.1, -0.3, 0.2))
        m.insert_points(sensor, pose, torch.from_numpy(rec).cuda(), w, h, 16,
                        flags=N.NM_FILTER_MEAN if filtered else 0)
        R, eye, mt = oracle_frame(desc, pose, res, rounding)
        pts = pts.reshape(-1, 3)
        if filtered:
            pts, R = O.voxel_filter(R, eye, res, mt, rounding, pts)[0], IDENTITY
        om.insert(R, eye, mt, desc.log_odds_hit, desc.log_odds_miss, pts)
    ours, ref = m.export(), om.export()
    assert {tuple(o) for o in ours[0]} == {tuple(o) for o in ref[0]}
    errs = compare_maps(ours, ref)
    assert not errs, "; ".join(errs[:4])
    st, ost = m.stats(), om.stats()
    assert st["leaf_count"] == ost["leaves"]
    for k in ("visits", "rays", "unique_voxels"):
        assert st[k] == ost[k], k
