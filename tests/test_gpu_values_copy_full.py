"""nm_map_values_copy of tables that hold few leaves to almost their limit (copied leaf by leaf or whole)."""
import numpy as np
import pytest
import torch

from nanomap_b200 import _native as N
from nanomap_b200 import api as A

pytestmark = pytest.mark.gpu

CAPACITY = 1 << 16


@pytest.mark.parametrize("load", [0.05, 0.15, 0.18, 0.44])
def test_every_slot(ctx, load):
    desc = A.sensor_desc(hres=48, vres=1, max_range=6.0, explicit_log_odds=1, log_odds_hit=0.85,
                         log_odds_miss=-0.4)
    sensor = A.Sensor(ctx, desc)
    m = A.Map(ctx, A.map_desc(res=0.05, initial_leaf_capacity=CAPACITY))
    rng = np.random.default_rng(7)
    for k in range(200):
        v = rng.normal(size=(48, 3))
        rec = np.zeros((48, 4), np.float32)
        rec[:, :3] = v / np.linalg.norm(v, axis=1, keepdims=True) * 5.9
        m.insert_points(sensor, A.Pose((13.0 * k, 0.0, 0.0), (1, 0, 0, 0)), torch.from_numpy(rec).cuda(), 48, 1,
                        16, flags=N.NM_SYNC)
        if m.stats()["leaf_count"] >= load * CAPACITY:
            break
    assert m.stats()["leaf_capacity"] == CAPACITY and m.stats()["leaf_count"] >= load * CAPACITY
    got = m.values_copy().cpu().numpy()
    so = m.slot_origins()
    used = so[:, 0] != np.iinfo(np.int32).min
    assert not got[~used].any()
    org, val, _ = m.export()
    want = {tuple(o): v for o, v in zip(org, val)}
    assert used.sum() == len(want)
    for o, v in zip(so[used], got[used]):
        assert np.array_equal(v, want[tuple(o)])
