"""Ray casts through the sim map: few rays (each walked in parts by several lanes) against the same
rays among many (one lane each) and against rays cast alone, bit for bit, at the places where a
part's start could land beside the whole walk's voxel.
"""
import numpy as np
import pytest

from nanomap_b200 import api as A
from nanomap_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0.05, 0.1])
def world(ctx, request):
    spec = S.SceneSpec(**{**S.SCENES["plain_small"].__dict__, "sim_res": request.param})
    scene = S.make_scene(spec, 2)
    return A.SimMap(ctx, request.param, boxes=scene.boxes, cylinders=scene.cylinders,
                    vox_min=scene.vox_min, vox_max=scene.vox_max)


def _rays(n, seed, res=0.1):
    rng = np.random.default_rng(seed)
    o = rng.uniform([-3.0, -3.0, -2.0], [23.0, 23.0, 7.0], (n, 3))
    d = rng.normal(size=(n, 3))
    k = n // 8
    d[:k] = np.eye(3)[rng.integers(0, 3, k)] * rng.choice([-1.0, 1.0], (k, 1))     # axis-aligned
    d[k:2 * k] = np.sign(d[k:2 * k])                                              # exact ties
    d[2 * k:3 * k, 2] = 0.0
    o[k // 2:2 * k] = np.round(o[k // 2:2 * k] / res) * res                       # lattice corners
    o[3 * k:4 * k, 0] = np.round(o[3 * k:4 * k, 0] / (8 * res)) * 8 * res         # leaf faces
    d[4 * k:5 * k] *= 10.0 ** rng.uniform(-6, 6, (k, 1))                          # any length
    d[0], d[1], d[2], d[3] = 0.0, np.nan, np.inf, (1e-30, 1.0, 0.0)
    return o.astype(np.float32), d.astype(np.float32)


@pytest.mark.parametrize("n", [8, 33, 511, 4736, 4737, 9472])
@pytest.mark.parametrize("max_range", [0.0, 0.4, 5.0, 200.0, 3e5])
def test_parts_equal_whole(world, n, max_range):
    import torch
    o, d = _rays(n, n)
    few = world.cast_rays(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda(), max_range)
    reps = 20000 // n + 1
    to = torch.from_numpy(np.tile(o, (reps, 1))).cuda()
    td = torch.from_numpy(np.tile(d, (reps, 1))).cuda()
    many = world.cast_rays(to, td, max_range).view(reps, n)
    assert torch.equal(few.view(torch.int32), many[0].view(torch.int32))
    assert torch.equal(many[0].view(torch.int32), many[-1].view(torch.int32))


@pytest.mark.parametrize("n", [9473, 18945, 75777, 160000])
def test_rays_do_not_depend_on_their_number(world, n):
    import torch
    o, d = _rays(n, 5)
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    got = world.cast_rays(to, td, 8.0)
    for lo in range(0, n, n // 3):
        part = world.cast_rays(to[lo:lo + 4000].contiguous(), td[lo:lo + 4000].contiguous(), 8.0)
        assert torch.equal(part.view(torch.int32), got[lo:lo + 4000].view(torch.int32))
