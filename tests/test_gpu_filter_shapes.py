"""Voxel filter at the shapes its binning and packing turn on: images made of 8 x 4 patches and not,
of 64 x 64 super-tiles and not, packing blocks full, partial and empty, and points at both length
limits -- filtered points, labels and map bit-identical to the oracle's.
"""
import numpy as np
import pytest

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from oracle import oracle as O
from tests.workloads import compare_labels, compare_maps, oracle_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (7, 5), (8, 4), (9, 4), (8, 5), (1000, 1), (64, 63), (64, 64),
                                  (65, 64), (72, 68), (128, 100), (200, 129)])
@pytest.mark.parametrize("rounding", [N.NM_ROUND_DOWN, N.NM_ROUND_NEAREST])
def test_shapes(ctx, size, rounding):
    import torch
    w, h = size
    res, reach = 0.1, 6.0
    desc = A.sensor_desc(hres=w, vres=h, max_range=reach, explicit_log_odds=1, log_odds_hit=0.85,
                         log_odds_miss=-0.4)
    sensor = A.Sensor(ctx, desc)
    m, om = A.Map(ctx, A.map_desc(res=res, rounding=rounding)), O.Map(res, rounding=rounding)
    rng = np.random.default_rng(w * 1000 + h)
    for k in range(2):
        # a wall seen by a camera: neighbours share voxels
        u, v = np.meshgrid(np.linspace(-0.6, 0.6, w), np.linspace(-0.4, 0.4, h))
        d = np.stack([u, v, np.ones_like(u)], -1).reshape(-1, 3)
        p = (d * rng.uniform(2.0, 2.3, (w * h, 1))).astype(np.float32)
        far = rng.uniform(size=w * h)
        p[far < 0.1] *= np.float32(10.0)                       # out of range
        edge = (far > 0.1) & (far < 0.2)                       # round the maximum range
        n = np.linalg.norm(p[edge].astype(np.float64), axis=1, keepdims=True)
        p[edge] = (p[edge] / n * (reach * (1.0 + rng.choice([-1e-7, 0.0, 1e-7, -1e-4, 1e-4], (len(n), 1))))).astype(np.float32)
        p[(far > 0.2) & (far < 0.25)] = np.nan
        tiny = (far > 0.25) & (far < 0.3)
        p[tiny] = (d[tiny] * rng.choice([0.0, 1e-9, 9e-8, 1.1e-7, 4e-7], (int(tiny.sum()), 1))).astype(np.float32)
        pose = A.Pose((0.31 + k, -0.17, 0.05), (0.9, 0.1, -0.3, 0.2))
        dev = torch.from_numpy(p).cuda()
        R, eye, mt = oracle_frame(desc, pose, res, rounding)
        op, oc = O.voxel_filter(R, eye, res, mt, rounding, p)
        gp, gc = m.filter_points(sensor, pose, dev, w, h, 12)
        assert np.array_equal(gc, oc) and np.array_equal(gp.view(np.uint32), op.view(np.uint32))
        m.insert_points(sensor, pose, dev, w, h, 12, flags=N.NM_FILTER_MEAN | N.NM_DEFER_INTEGRATE)
        om.insert(np.eye(3, dtype=np.float32).reshape(-1), eye, mt, desc.log_odds_hit, desc.log_odds_miss,
                  op, keep_labels=True)
        errs = compare_labels(m.export_labels(), om.labels())
        assert not errs, "; ".join(errs[:4])
        m.integrate()
    errs = compare_maps(m.export(), om.export())
    assert not errs, "; ".join(errs[:4])
