"""Labels of single frames against the CPU oracle, bit-identical, where a ray's first and last voxels are
hard to tell: first planes almost at the eye, and ends almost at the maximum range.
"""
import numpy as np
import pytest
import torch

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from oracle import oracle as O
from tests.workloads import compare_labels, compare_maps, oracle_frame

pytestmark = pytest.mark.gpu

ROUNDINGS = [N.NM_ROUND_DOWN, N.NM_ROUND_NEAREST]


def _check(ctx, pts, eye, res, rng_m, rounding):
    """Inserts the records `pts` (h, w, 3), world offsets from the eye."""
    h, w, _ = pts.shape
    desc = A.sensor_desc(hres=w, vres=h, max_range=rng_m, explicit_log_odds=1, log_odds_hit=0.85,
                         log_odds_miss=-0.4)
    m, om = A.Map(ctx, A.map_desc(res=res, rounding=rounding)), O.Map(res, rounding=rounding)
    rec = np.zeros((h, w, 4), np.float32)
    rec[..., :3] = pts
    pose = A.Pose(eye, (1.0, 0.0, 0.0, 0.0))
    m.insert_points(A.Sensor(ctx, desc), pose, torch.from_numpy(rec).cuda(), w, h, 16,
                    flags=N.NM_DEFER_INTEGRATE)
    R, e, mt = oracle_frame(desc, pose, res, rounding)
    om.insert(R, e, mt, desc.log_odds_hit, desc.log_odds_miss, rec[..., :3].reshape(-1, 3), keep_labels=True)
    errs = compare_labels(m.export_labels(), om.labels())
    assert not errs, "; ".join(errs[:4])
    m.integrate()
    errs = compare_maps(m.export(), om.export())
    assert not errs, "; ".join(errs[:4])
    st, ost = m.stats(), om.stats()
    for k in ("visits", "rays", "unique_voxels"):
        assert st[k] == ost[k], k
    return e


@pytest.mark.parametrize("rounding", ROUNDINGS)
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_first_plane_at_the_near_limit(ctx, rounding, axis):
    """An eye whose distance to a plane is below the limit of close planes (1e-4f), by so little that
    it rounds to it as a float."""
    res, limit = 0.05, np.float32(1e-4)
    p = np.float32(limit * np.float32(res))
    for _ in range(40):
        d = float(p) * (1.0 / float(np.float32(res)))
        if d < float(limit) and np.float32(d) == limit:
            break
        p = np.nextafter(p, np.float32(0.0)) if d >= float(limit) else np.nextafter(p, np.float32(1.0))
    else:
        pytest.fail("no such eye")
    eye = [0.137, -0.218, 0.391]
    eye[axis] = float(p)
    rng = np.random.default_rng(axis)
    v = rng.normal(size=(16, 32, 3))
    v[..., axis] = -np.abs(v[..., axis])
    v *= rng.uniform(4.0, 9.5, (16, 32, 1)) / np.linalg.norm(v, axis=2, keepdims=True)
    e = _check(ctx, v, tuple(eye), res, 10.0, rounding)
    assert e[axis] < float(limit) and np.float32(e[axis]) == limit


@pytest.mark.parametrize("rounding", ROUNDINGS)
@pytest.mark.parametrize("units", [(1, 7), (7, 1), (11, 4)])
def test_denormal_eye(ctx, rounding, units):
    """An eye a few denormal floats from a lattice edge.  In voxels of 0.3 m its distances to the two planes
    are no whole number of them: all rays run between the direction that crosses both planes at once and
    the one that seems to when the distances are rounded to floats."""
    res, unit = 0.3, float(np.float32(1.4e-45))
    e = [units[i] * unit / float(np.float32(res)) for i in range(2)]
    true, rounded = e[1] / e[0], float(np.float32(e[1])) / float(np.float32(e[0]))
    rng = np.random.default_rng(units[0])
    v = -np.ones((16, 32, 3))
    v[..., 1] = -(true + (rounded - true) * rng.uniform(0.2, 0.8, (16, 32)))
    v[..., 2] = rng.normal(size=(16, 32)) * true
    v *= rng.uniform(40.0, 58.0, (16, 32, 1)) / np.linalg.norm(v, axis=2, keepdims=True)
    e = _check(ctx, v, (units[0] * unit, units[1] * unit, 0.391), res, 60.0, rounding)
    assert 0.0 < e[0] < 1e-42 and 0.0 < e[1] < 1e-42


@pytest.mark.parametrize("rounding", ROUNDINGS)
@pytest.mark.parametrize("eye", [(0.137, -0.218, 0.391), (0.05, -0.2, 1.0), (0.0, 0.0, 0.0)])
@pytest.mark.parametrize("reach", [9.0, 50.0, 80.0, 130.0, 400.0])
def test_ends_near_the_range(ctx, rounding, eye, reach):
    """Rays that end within three voxels of the range, or leave their end voxel there (a hit only when that
    crossing comes before the range): walked tiles up to 80 voxels, marched ones from 130 on; axis-aligned
    and diagonal rays among them, and ends up to 1e-6 voxels from the range."""
    res = 0.05
    rng = np.random.default_rng(int(reach))
    d = rng.normal(size=(32, 32, 3))
    d[:4] = np.eye(3)[rng.integers(0, 3, (4, 32))] * rng.choice([-1.0, 1.0], (4, 32, 1))
    d[4:6] = np.sign(rng.normal(size=(2, 32, 3)))
    d[6, :, 2] = 0.0
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    r = reach - rng.uniform(0.0, 3.0, (32, 32, 1))
    r[::5] = reach - 10.0 ** rng.uniform(-6.0, 0.0, (7, 32, 1))
    r[1::5] = rng.uniform(1.0, reach, (7, 32, 1))
    _check(ctx, d * r * res, eye, res, reach * res, rounding)


@pytest.mark.parametrize("rounding", ROUNDINGS)
@pytest.mark.parametrize("spread", [2e-4, 2e-2, 1.0])
@pytest.mark.parametrize("reach", [1000.0, 2500.0, 3900.0])
def test_long_reach(ctx, rounding, spread, reach):
    """Up to 3900 voxels of reach: past the 2032 planes of a window (a beam narrow enough to stay in it, one
    that leaves it early, and rays of all directions)."""
    res = 0.005
    rng = np.random.default_rng(int(reach))
    d = np.array([0.7, -0.5, 0.51]) + spread * rng.normal(size=(8, 32, 3))
    d[0, :6] = np.concatenate([np.eye(3), -np.eye(3)])
    d[0, 6:9] = [[1, 1, 1], [1, -1, 0], [0, 1, -1]]
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    r = rng.uniform(0.5 * reach, reach, (8, 32, 1))
    _check(ctx, d * r * res, (0.0137, -0.0218, 0.391), res, reach * res, rounding)
