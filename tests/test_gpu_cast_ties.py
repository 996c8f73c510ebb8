"""Ray casts against the CPU oracle, bit for bit, where a skip over empty leaves lands on or beside a
voxel plane: origins on the lattice and a hair off it, directions along axes and diagonals and at a
hair from them, worlds near the origin, far from it, and past the coordinates where a position alone
may decide on the voxel."""
import numpy as np
import pytest

from nanomap_b200 import api as A
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, -3000, 60000, 600000])
@pytest.mark.parametrize("n", [300, 40000])
def test_casts_match_oracle(ctx, shift, n):
    res = np.float32(0.125)  # (origins on the lattice are exact)
    rng = np.random.default_rng(abs(shift) + n)
    vox = rng.integers(-150, 150, size=(1500, 3))
    vox = np.concatenate([vox, np.stack(np.meshgrid(range(-60, 60), range(-60, 60), [-97]), -1).reshape(-1, 3)])
    vox = (vox + shift).astype(np.int32)
    g, o = A.SimMap(ctx, float(res), voxels=vox), O.SimMap(float(res), voxels=vox)
    e = rng.uniform(-170.0, 170.0, (n, 3))
    d = rng.normal(size=(n, 3))
    k = n // 6
    e[:2 * k] = np.round(e[:2 * k])                                   # corners
    e[2 * k:3 * k] = np.round(e[2 * k:3 * k] / 8) * 8 + rng.choice([-1e-4, 1e-4], (k, 3))
    d[::3] = np.sign(d[::3])                                          # diagonals
    d[1::6] = np.eye(3)[rng.integers(0, 3, len(d[1::6]))] * rng.choice([-1.0, 1.0], (len(d[1::6]), 1))
    d[2::6, 1] = 0.0
    d[::4] += 1e-5 * rng.normal(size=d[::4].shape)
    e, d = ((e + shift) * res).astype(np.float32), d.astype(np.float32)
    for max_range in (10.0, 60.0):
        got, want = g.cast_rays(e, d, max_range), o.cast(e, d, max_range)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), int((got != want).sum())
