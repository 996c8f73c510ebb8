"""Expected depth where the walk's short cuts begin and end: densities on both sides of the
series' limit and near zero (thin media, the ray reaching its range), and the fixed-order sums of
the adjoint's and the refinement's partials at image sizes round their strides.
"""
import numpy as np
import pytest

from nanomap_b200 import api as A
from nanomap_b200 import scenes as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RES = 0.1


@pytest.fixture(scope="module")
def world(ctx):
    import torch
    spec = S.SCENES["plain_small"]
    scene = S.make_scene(spec, 3)
    pos, q = S.trajectory(scene, 1, seed=5)[0]
    pose = A.Pose(pos, q)
    desc = A.sensor_desc(**{**S.sensor_desc_kwargs(spec), "hres": 64, "vres": 48})
    sensor = A.Sensor(ctx, desc)
    sim = A.SimMap(ctx, RES, boxes=scene.boxes, cylinders=scene.cylinders, vox_min=scene.vox_min,
                   vox_max=scene.vox_max)
    r = torch.zeros(48, 64, device="cuda")
    sim.render(sensor, pose, r)
    m = A.Map(ctx, A.map_desc(res=RES))
    for _ in range(3):
        m.insert_ranges(sensor, pose, r)
    p, R = A.Map.ray_pose(sensor, pose)
    org, val, _ = m.export()
    return dict(ctx=ctx, spec=spec, m=m, p=p, R=R, org=org, val=val, sim=sim, pose=pose)


def _camera(w, width, height):
    desc = A.sensor_desc(**{**S.sensor_desc_kwargs(w["spec"]), "hres": width, "vres": height})
    return A.Sensor(w["ctx"], desc), O.Sensor.from_desc(desc)


@pytest.mark.parametrize("bias", [-30.0, -14.0, -6.95, -6.9, -6.85, -3.0, 0.0])
@pytest.mark.parametrize("size", [(13, 9), (64, 48)])
def test_thin_and_dense_media(world, bias, size):
    """Unknown space has the density softplus(bias), which crosses the series' limit (2^-10 per
    segment) between the biases here.  Depth within 1e-5 of the FP64 definition (relative to the
    largest), log-odds gradient within 1e-4."""
    import torch
    w = world
    cam, osen = _camera(w, *size)
    res = float(np.float32(RES))
    D = w["m"].depth_render(cam, w["p"], w["R"], scale=0.5, bias=bias)
    gd = np.random.default_rng(1).choice([-1.0, 1.0], size[0] * size[1]).astype(np.float32)
    vals = w["m"].values_copy()
    gv = torch.zeros_like(vals)
    w["m"].depth_backward(cam, w["p"], w["R"], torch.from_numpy(gd).cuda().view(size[1], size[0]),
                              values=vals, grad_values=gv, scale=0.5, bias=bias, depth=D)
    ref, _, _, ogv = O.depth(osen, w["p"], w["R"], res, w["org"], w["val"], scale=0.5, bias=bias,
                                 grad_depth=gd.astype(np.float64))
    assert np.abs(D.cpu().numpy().reshape(-1) - ref).max() <= 1e-5 + 1e-5 * ref.max()
    so = w["m"].slot_origins()
    used = so[:, 0] != np.iinfo(np.int32).min
    G = {tuple(o): x for o, x in zip(so[used], gv.cpu().numpy()[used])}
    worst = max(float(np.abs(G[tuple(o)] - ogv[i]).max()) for i, o in enumerate(w["org"]))
    assert worst <= 1e-4 * np.abs(ogv).max()


@pytest.mark.parametrize("size", [(1, 1), (8, 8), (9, 8), (1016, 8), (1024, 8), (1032, 8), (1024, 32),
                                  (1024, 33), (257, 129), (640, 480)])
def test_sums_of_partials(world, size):
    """The pose gradient of an image is the sum of its parts' (linear in grad_depth): 1 to 4800
    blocks of partials, round the 128 rows a pass adds and the four passes in flight."""
    import torch
    w = world
    cam, _ = _camera(w, *size)
    W, H = size
    gd = torch.from_numpy(np.random.default_rng(2).normal(size=(H, W)).astype(np.float32)).cuda()
    full = w["m"].depth_backward(cam, w["p"], w["R"], gd, scale=2.0)
    parts, mag = np.zeros(6), np.zeros(6)
    mask = torch.from_numpy(np.random.default_rng(3).integers(0, 3, (H, W))).cuda()
    for k in range(3):
        x = w["m"].depth_backward(cam, w["p"], w["R"], gd * (mask == k), scale=2.0)
        parts += x
        mag += np.abs(x)
    assert (np.abs(full - parts) <= 1e-12 * W * H * (mag + 1e-6)).all()


@pytest.mark.parametrize("size", [(8, 8), (65, 47), (1024, 33)])
def test_refinement_sums(world, size):
    """The first loss of a refinement is the mean of |prediction - target| over the target's
    pixels with a return."""
    import torch
    w = world
    cam, _ = _camera(w, *size)
    t = torch.zeros(size[1], size[0], device="cuda")
    w["sim"].render(cam, w["pose"], t)
    D = w["m"].depth_render(cam, w["p"], w["R"], scale=3.0)
    ok = t > 0
    assert bool(ok.any())
    want = float((D - t).abs()[ok].double().mean())
    _, _, losses = w["m"].pose_refine(cam, w["p"], w["R"], t, steps=2, scale=3.0)
    assert abs(losses[0] - want) <= 1e-5 * want + 1e-6
    assert np.isfinite(losses).all()
