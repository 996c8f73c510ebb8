"""Accumulate mode: the map holds the leaves that some ray counted a voxel in, and no others.  Rays that
end in their first voxel of a leaf and leave it past the maximum range count nothing there."""
import numpy as np
import pytest
import torch

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from oracle import oracle as O
from tests.workloads import compare_maps, oracle_frame

pytestmark = pytest.mark.gpu


def _check(ctx, pts, eye, res, rng_m, rounding):
    """One frame of records `pts` (h, w, 3): leaves, their number and the touched ones, and the map."""
    h, w, _ = pts.shape
    desc = A.sensor_desc(hres=w, vres=h, max_range=rng_m, explicit_log_odds=1, log_odds_hit=0.85,
                         log_odds_miss=-0.4)
    m = A.Map(ctx, A.map_desc(res=res, rounding=rounding, update_mode=N.NM_UPDATE_ACCUMULATE))
    om = O.Map(res, rounding=rounding, update_mode=1)
    rec = np.zeros((h, w, 4), np.float32)
    rec[..., :3] = pts
    pose = A.Pose(eye, (1.0, 0.0, 0.0, 0.0))
    m.insert_points(A.Sensor(ctx, desc), pose, torch.from_numpy(rec).cuda(), w, h, 16)
    R, e, mt = oracle_frame(desc, pose, res, rounding)
    om.insert(R, e, mt, desc.log_odds_hit, desc.log_odds_miss, pts.reshape(-1, 3).astype(np.float32))
    ours, ref = m.export(), om.export()
    assert {tuple(o) for o in ours[0]} == {tuple(o) for o in ref[0]}
    errs = compare_maps(ours, ref)
    assert not errs, "; ".join(errs[:4])
    st, ost = m.stats(), om.stats()
    assert st["leaf_count"] == st["touched_leaves"] == ost["leaves"]
    for k in ("visits", "rays", "unique_voxels"):
        assert st[k] == ost[k], k


@pytest.mark.parametrize("rounding", [N.NM_ROUND_DOWN, N.NM_ROUND_NEAREST])
@pytest.mark.parametrize("x", [7.3, 7.45, 7.55, 7.7, 7.95])
def test_one_ray(ctx, rounding, x):
    """From x = 0.5 along +x at a range of 8 voxels: from 7.5 on the ray ends in voxel 8, the first of
    the next leaf, and would leave it at 8.5, past the range."""
    _check(ctx, np.array([[[x, 0.0, 0.0]]]), (0.5, 0.5, 0.5), 1.0, 8.0, rounding)


@pytest.mark.parametrize("rounding", [N.NM_ROUND_DOWN, N.NM_ROUND_NEAREST])
@pytest.mark.parametrize("rng_vox", [9.0, 40.0, 250.0])
def test_rays_ending_near_the_range(ctx, rounding, rng_vox):
    """Ends within two voxels of the range in all directions; at 250 voxels with more leaves a tile than
    the shared table has entries, where the others are counted in the device table."""
    res = 0.05
    rng = np.random.default_rng(int(rng_vox))
    d = rng.normal(size=(24, 32, 3))
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    r = rng.uniform(rng_vox - 2.0, rng_vox, (24, 32, 1)) * res
    _check(ctx, (d * r).astype(np.float32), (0.137, -0.218, 0.391), res, rng_vox * res, rounding)
