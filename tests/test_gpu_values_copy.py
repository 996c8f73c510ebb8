"""nm_map_values_copy: whole tables and tables copied leaf by leaf, device memory at every
alignment, with leaves in the first and last slots' warps, into dirty memory."""
import ctypes as C

import numpy as np
import pytest

from nanomap_b200 import _native as N
from nanomap_b200 import api as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity", [1024, 1 << 15, 1 << 16, 1 << 17])
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_every_slot(ctx, capacity, offset):
    import torch
    desc = A.sensor_desc(hres=40, vres=30, hfov_deg=80.0, vfov_deg=60.0, max_range=4.0,
                         explicit_log_odds=1, log_odds_hit=0.85, log_odds_miss=-0.4)
    sensor = A.Sensor(ctx, desc)
    m = A.Map(ctx, A.map_desc(res=0.1, initial_leaf_capacity=capacity))
    r = torch.rand(30, 40, device="cuda") * 3.0 + 0.5
    for k in range(4):
        m.insert_ranges(sensor, A.Pose((0.3 * k, 0.0, 0.0), (1, 0, 0, 0)), r)
    n = C.c_uint64()
    N.call("nm_map_values_copy", m.h, None, 0, C.byref(n), None)
    buf = torch.full((n.value + offset,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    N.call("nm_map_values_copy", m.h, C.c_void_p(buf.data_ptr() + 4 * offset), n.value, C.byref(n), None)
    got = buf[offset:].cpu().numpy().reshape(-1, 512)
    so = m.slot_origins()
    used = so[:, 0] != np.iinfo(np.int32).min
    assert len(got) == len(so) and not got[~used].any() and not np.isnan(got).any()
    org, val, _ = m.export()
    want = {tuple(o): v for o, v in zip(org, val)}
    assert used.sum() == len(want)
    for o, v in zip(so[used], got[used]):
        assert np.array_equal(v, want[tuple(o)])
    assert torch.isnan(buf[:offset]).all()
