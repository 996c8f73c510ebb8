"""Long rays in few tiles (the traversal takes such tiles apart and marches over lattice planes)
against the CPU oracle: labels, map and counters bit-identical, at the places where the exact line
comes close to a tie (eye on lattice planes, edges and corners, axis-aligned and diagonal rays),
for narrow and wide beams, partial tiles, both signs, both roundings and every input kind.
"""
import numpy as np
import pytest

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from nanomap_b200 import scenes as S
from oracle import oracle as O
from tests.workloads import compare_labels, compare_maps, oracle_frame

pytestmark = pytest.mark.gpu

RES = 0.05
EYES = {
    "inside": (0.137, -0.218, 0.391),
    "plane": (0.137, -0.218, 0.05),
    "edge": (0.05, -0.2, 0.391),
    "corner": (1.0, -0.05, 2.0),
    "origin": (0.0, 0.0, 0.0),
    "near_corner": (1.0 + 4e-8, -0.05 + 1e-9, 2.0),
    "far": (-211.37, 93.21, 17.77),
}


def _quat(k):
    q = np.random.default_rng(100 + k).normal(size=4)
    return (1.0, 0.0, 0.0, 0.0) if k == 0 else tuple(q / np.linalg.norm(q))


def _check(ctx, sensor, desc, frames, rounding, insert):
    """frames: [(pose, points for the oracle, argument of insert)]"""
    m = A.Map(ctx, A.map_desc(res=RES, rounding=rounding))
    om = O.Map(RES, rounding=rounding)
    for pose, pts, arg in frames:
        insert(m, pose, arg)
        R, eye, mt = oracle_frame(desc, pose, RES, rounding)
        om.insert(R, eye, mt, desc.log_odds_hit, desc.log_odds_miss, pts, keep_labels=True)
        errs = compare_labels(m.export_labels(), om.labels())
        assert not errs, "; ".join(errs[:4])
        m.integrate()
    errs = compare_maps(m.export(), om.export())
    assert not errs, "; ".join(errs[:4])
    st, ost = m.stats(), om.stats()
    for k in ("visits", "rays", "unique_voxels"):
        assert st[k] == ost[k], k


@pytest.mark.parametrize("eye", sorted(EYES))
@pytest.mark.parametrize("rounding", [N.NM_ROUND_DOWN, N.NM_ROUND_NEAREST])
@pytest.mark.parametrize("kind", ["camera", "wide_camera", "laser"])
def test_range_images(ctx, eye, rounding, kind):
    w, h, rng_m = {"camera": (67, 45, 12.0), "wide_camera": (17, 33, 30.0), "laser": (128, 19, 14.0)}[kind]
    kw = (dict(type=1, hfov_deg=360.0, vfov_deg=30.0) if kind == "laser" else
          dict(type=0, hfov_deg=20.0 if kind == "camera" else 100.0, vfov_deg=15.0 if kind == "camera" else 80.0))
    desc = A.sensor_desc(hres=w, vres=h, max_range=rng_m, explicit_log_odds=1, log_odds_hit=0.85,
                         log_odds_miss=-0.4, frame_transform=S.OPTICAL_TO_BODY, **kw)
    sensor, osen = A.Sensor(ctx, desc), O.Sensor.from_desc(desc)
    import torch
    frames = []
    for k in range(3):
        rng = np.random.default_rng(10 * k + 1)
        r = rng.uniform(0.0, rng_m, (h, w)).astype(np.float32) if k else np.full((h, w), 0.97 * rng_m, np.float32)
        r[rng.uniform(size=r.shape) < 0.05] = 0.0
        r[rng.uniform(size=r.shape) < 0.02] = np.float32(rng_m)          # dropped at max range
        r[rng.uniform(size=r.shape) < 0.02] = np.float32(rng_m - 0.06)   # ends near max range
        frames.append((A.Pose(EYES[eye], _quat(k)), osen.points(r), torch.from_numpy(r).cuda()))
    _check(ctx, sensor, desc, frames, rounding,
           lambda m, pose, x: m.insert_ranges(sensor, pose, x, flags=N.NM_DEFER_INTEGRATE))


@pytest.mark.parametrize("eye", sorted(EYES))
@pytest.mark.parametrize("rounding", [N.NM_ROUND_DOWN, N.NM_ROUND_NEAREST])
@pytest.mark.parametrize("step", [12, 16, 20])
def test_records(ctx, eye, rounding, step):
    """Records of any directions in one cloud: axis-aligned, diagonal (exact ties), lattice
    points as ends, parallel beams' worth of spread, NaN and Inf."""
    w, h = 37, 21
    desc = A.sensor_desc(hres=w, vres=h, max_range=9.0, explicit_log_odds=1, log_odds_hit=0.85,
                         log_odds_miss=-0.4)
    sensor = A.Sensor(ctx, desc)
    rng = np.random.default_rng(step)
    d = rng.normal(size=(h * w, 3))
    d[:200] = np.array([0.8, 0.5, -0.3]) + 0.02 * rng.normal(size=(200, 3))
    d[200:230] = np.sign(rng.normal(size=(30, 3)))
    d[230:260] = np.eye(3)[rng.integers(0, 3, 30)] * rng.choice([-1, 1], (30, 1))
    d[260:290, 2] = 0.0
    d[290:320, 0] = d[290:320, 1]
    p = (d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.2, 8.9, (h * w, 1))).astype(np.float32)
    p[320:350] = (np.round(p[320:350] / RES) * RES).astype(np.float32)
    p[350], p[351], p[352] = np.nan, np.inf, 0.0
    rec = np.zeros((h * w, step // 4), np.float32)
    rec[:, :3] = p
    import torch
    frames = [(A.Pose(EYES[eye], _quat(k)), p, torch.from_numpy(rec).cuda()) for k in range(2)]
    _check(ctx, sensor, desc, frames, rounding,
           lambda m, pose, x: m.insert_points(sensor, pose, x, w, h, step, flags=N.NM_DEFER_INTEGRATE))


@pytest.mark.parametrize("tile", [(16, 8, 64), (32, 32, 512), (16, 16, 16), (48, 16, 128), (64, 24, 256),
                                  (64, 64, 256)])
def test_launch_shapes(ctx, tile):
    """Quarters of 32 to 1024 rays (several rounds), tables too small for a unit, tiles not square
    and tiles whose quarters are no whole number of rounds."""
    desc = A.sensor_desc(hres=75, vres=50, hfov_deg=60.0, vfov_deg=40.0, max_range=20.0,
                         explicit_log_odds=1, log_odds_hit=0.85, log_odds_miss=-0.4,
                         frame_transform=S.OPTICAL_TO_BODY)
    sensor, osen = A.Sensor(ctx, desc), O.Sensor.from_desc(desc)
    import torch
    rng = np.random.default_rng(3)
    r = rng.uniform(1.0, 19.8, (50, 75)).astype(np.float32)
    pose = A.Pose(EYES["inside"], _quat(2))

    def insert(m, pose, x):
        m.set_launch(*tile)
        m.insert_ranges(sensor, pose, x, flags=N.NM_DEFER_INTEGRATE)

    _check(ctx, sensor, desc, [(pose, osen.points(r), torch.from_numpy(r).cuda())], N.NM_ROUND_DOWN, insert)
