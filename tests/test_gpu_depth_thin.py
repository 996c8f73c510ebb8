"""Expected depth and its gradients where the density is too thin for a reciprocal: denormal and
vanishing densities everywhere, and observed free space that thin beside dense unknown space.
"""
import numpy as np
import pytest

from nanomap_b200 import api as A
from nanomap_b200 import scenes as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RES = 0.1
SIZE = (64, 48)


@pytest.fixture(scope="module")
def world(ctx):
    import torch
    spec = S.SCENES["plain_small"]
    scene = S.make_scene(spec, 3)
    pos, q = S.trajectory(scene, 1, seed=5)[0]
    pose = A.Pose(pos, q)
    desc = A.sensor_desc(**{**S.sensor_desc_kwargs(spec), "hres": SIZE[0], "vres": SIZE[1]})
    cam = A.Sensor(ctx, desc)
    sim = A.SimMap(ctx, RES, boxes=scene.boxes, cylinders=scene.cylinders, vox_min=scene.vox_min,
                   vox_max=scene.vox_max)
    r = torch.zeros(SIZE[1], SIZE[0], device="cuda")
    sim.render(cam, pose, r)
    m = A.Map(ctx, A.map_desc(res=RES))
    for _ in range(12):  # observed free space reaches the lower clamp
        m.insert_ranges(cam, pose, r)
    p, R = A.Map.ray_pose(cam, pose)
    org, val, _ = m.export()
    return dict(m=m, cam=cam, osen=O.Sensor.from_desc(desc), p=p, R=R, org=org, val=val)


@pytest.mark.parametrize("scale,bias", [(0.5, -70.0), (0.5, -88.0), (0.5, -89.0), (0.5, -95.0), (0.5, -103.0),
                                        (0.5, -110.0), (1.0, -90.0), (45.0, 0.0), (50.0, 0.0)])
def test_thin(world, scale, bias):
    """Depth within 1e-5 of the FP64 definition (relative to the largest).  Log-odds gradients within
    1e-4 of the largest, and 1e-33: a density of at most 1.2e-38 may count as zero in FP32, which
    moves a voxel's gradient by res * scale * 1.2e-38 * (segment x range in voxels, < 350) for each of
    3072 rays."""
    import torch
    w = world
    D = w["m"].depth_render(w["cam"], w["p"], w["R"], scale=scale, bias=bias)
    gd = np.random.default_rng(1).choice([-1.0, 1.0], SIZE[0] * SIZE[1]).astype(np.float32)
    vals = w["m"].values_copy()
    gv = torch.zeros_like(vals)
    g6 = w["m"].depth_backward(w["cam"], w["p"], w["R"], torch.from_numpy(gd).cuda().view(SIZE[1], SIZE[0]),
                               values=vals, grad_values=gv, scale=scale, bias=bias, depth=D)
    ref, _, _, ogv = O.depth(w["osen"], w["p"], w["R"], float(np.float32(RES)), w["org"], w["val"],
                             scale=scale, bias=bias, grad_depth=gd.astype(np.float64))
    D = D.cpu().numpy().reshape(-1)
    assert np.isfinite(D).all() and np.isfinite(g6).all() and bool(torch.isfinite(gv).all())
    assert np.abs(D - ref).max() <= 1e-5 + 1e-5 * ref.max()
    so = w["m"].slot_origins()
    used = so[:, 0] != np.iinfo(np.int32).min
    G = {tuple(o): x for o, x in zip(so[used], gv.cpu().numpy()[used])}
    worst = max(float(np.abs(G[tuple(o)] - ogv[i]).max()) for i, o in enumerate(w["org"]))
    assert worst <= 1e-4 * np.abs(ogv).max() + 1e-33 * max(scale, 1.0)
