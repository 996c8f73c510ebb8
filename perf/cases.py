"""What this framework's users have it do, as cases that can be timed and compared.

Every case goes through the Python view of the C ABI (nanomap_b200.api, nanomap_b200.diff) the
way a mapping or simulation program does: handles (context, sensor, map, sim map, tick plan) and
buffers are made once, frames arrive as device or page-locked host buffers, calls are queued on
the current stream.  Worlds, cameras, ranges and resolutions are those of nanomap_b200.scenes;
drawn cases vary them over the same span.

A mapping case inserts a stretch of a trajectory through ground the map already covers and reads
back the log-odds of a box of leaves round the middle of the stretch (the window a planner
keeps), leaf by leaf in (x, y, z) order.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from nanomap_b200 import _native as N
from nanomap_b200 import api as A
from nanomap_b200 import diff
from nanomap_b200 import scenes as S

CAMERA = dict(type=0, hfov_deg=87.0, vfov_deg=58.0)
LASER = dict(type=1, hfov_deg=360.0, vfov_deg=30.0)


# ---- the cases -----------------------------------------------------------------------------

def listed():
    return [
        # a simulated agent's observation / collision rays: the smallest call
        dict(name="observe", kind="cast", world="plain_small", res=0.1, rays=512, range=5.0),
        # one frame of a small depth camera on a coarse map: launch latency
        dict(name="insert_small", kind="insert", world="plain_small", sensor="camera", width=320,
             height=240, range=5.0, res=0.1, frames=1, input="ranges", host=False, filter=False,
             rounding="down", mode="label"),
        # the headline: 640x480 PointCloud2-style records already on the device
        dict(name="insert_points", kind="insert", world="sim_headline", sensor="camera", width=640,
             height=480, range=10.0, res=0.05, frames=16, input="points", host=False, filter=False,
             rounding="down", mode="label"),
        # the same stream from page-locked host memory (a driver's message buffers)
        dict(name="insert_host", kind="insert", world="sim_headline", sensor="camera", width=640,
             height=480, range=10.0, res=0.05, frames=16, input="points", host=True, filter=False,
             rounding="down", mode="label"),
        # with the voxel filter in front (FilterType 1, the reference's usual setting)
        dict(name="insert_filtered", kind="insert", world="sim_headline", sensor="camera",
             width=640, height=480, range=10.0, res=0.05, frames=16, input="points", host=False,
             filter=True, rounding="down", mode="label"),
        # a spinning 64-beam sensor, 20 m: long rays far apart
        dict(name="insert_laser", kind="insert", world="sim_headline", sensor="laser", width=1024,
             height=64, range=20.0, res=0.05, frames=8, input="ranges", host=False, filter=False,
             rounding="down", mode="label"),
        # exact visit counts instead of labels (the reference's device path), odd image size
        dict(name="insert_counts", kind="insert", world="plain_small", sensor="camera", width=317,
             height=239, range=5.0, res=0.05, frames=4, input="ranges", host=False, filter=False,
             rounding="nearest", mode="counts"),
        # simulation in the loop: render a noisy frame, insert it
        dict(name="sim_frames", kind="sim", world="sim_headline", width=640, height=480,
             range=10.0, res=0.05, frames=16),
        # the 16-agent tick (cameras of three sizes and a spinning sensor in one map)
        dict(name="tick", kind="tick", world="plain_small", res=0.05, agents=16, ticks=4),
        # fine resolution, large image: map a frame, render the expected depth over the map
        dict(name="fine_map_render", kind="render", world="large_fine", width=1280, height=720,
             range=15.0, res=0.02),
        # gradients of the expected depth with respect to log-odds and pose
        dict(name="depth_gradients", kind="gradients", world="sim_headline", width=640,
             height=480, range=10.0, res=0.05),
        # scan-to-map pose refinement
        dict(name="refine", kind="refine", world="sim_headline", width=640, height=480,
             range=10.0, res=0.05, steps=30),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cast", "insert", "insert", "insert", "insert", "sim", "tick", "render",
                       "gradients", "refine"])
    if kind == "cast":
        return dict(kind=kind, world=rng.choice(["plain_small", "sim_headline"]),
                    res=rng.choice([0.05, 0.1]), rays=_log_int(rng, 50, 100000),
                    range=round(rng.uniform(3.0, 15.0), 2))
    if kind == "tick":
        return dict(kind=kind, world="plain_small", res=rng.choice([0.05, 0.1]),
                    agents=rng.randint(2, 16), ticks=rng.randint(1, 4))
    width = _log_int(rng, 100, 800)
    height = max(60, int(width * rng.uniform(0.5, 0.8)))
    world = rng.choice(["plain_small", "sim_headline"])
    res = rng.choice([0.05, 0.1]) if world == "plain_small" else rng.choice([0.04, 0.05, 0.1])
    rng_m = round(rng.uniform(3.0, 10.0), 2)
    c = dict(kind=kind, world=world, width=width, height=height, range=rng_m, res=res)
    if kind == "insert":
        laser = rng.random() < 0.2
        mode = "counts" if rng.random() < 0.15 else "label"
        c.update(sensor="laser" if laser else "camera", frames=rng.randint(1, 12),
                 input=rng.choice(["ranges", "points"]), host=rng.random() < 0.25,
                 filter=rng.random() < 0.25, rounding=rng.choice(["down", "down", "nearest"]),
                 mode=mode)
        if laser:
            c.update(width=_log_int(rng, 360, 1100), height=rng.choice([16, 32, 33, 64]),
                     range=round(rng.uniform(6.0, 20.0), 2))
        if mode == "counts":
            c.update(frames=min(c["frames"], 4), width=min(c["width"], 400),
                     height=min(c["height"], 300), range=min(c["range"], 6.0))
    elif kind == "sim":
        c.update(frames=rng.randint(1, 12))
    elif kind == "refine":  # a view that shows something: the dense world, a long range
        c.update(steps=rng.randint(5, 30), width=min(width, 640), height=min(height, 480),
                 world="sim_headline", range=round(rng.uniform(7.0, 10.0), 2))
    return c


# ---- worlds, poses, frames -----------------------------------------------------------------

@functools.lru_cache(maxsize=16)
def _world(name, res, seed):
    """The scene of a seed with `res` as its sim resolution (the voxel box follows)."""
    spec = S.SceneSpec(**{**S.SCENES[name].__dict__, "sim_res": res, "map_res": res})
    return S.make_scene(spec, seed % 100003 + 1)


@functools.lru_cache(maxsize=64)
def _poses(name, res, seed, n, which=0):
    return S.trajectory(_world(name, res, seed), n, seed=seed % 9973 + 7 + 31 * which)


def _sim_map(ctx, scene):
    return A.SimMap(ctx, scene.spec.sim_res, boxes=scene.boxes, cylinders=scene.cylinders,
                    vox_min=scene.vox_min, vox_max=scene.vox_max)


def _desc(case):
    base = LASER if case.get("sensor") == "laser" else CAMERA
    return A.sensor_desc(**base, hres=case["width"], vres=case["height"], max_range=case["range"],
                         explicit_log_odds=1, log_odds_hit=0.85, log_odds_miss=-0.4,
                         frame_transform=S.OPTICAL_TO_BODY)


def _pixel_dirs(case):
    """Sensor-frame unit directions (h, w, 3), float64: the pixel model of the sensor docs."""
    W, H = case["width"], case["height"]
    if case.get("sensor") == "laser":
        u = torch.arange(W, dtype=torch.float64, device="cuda") * (360.0 / W) - 180.0
        v = torch.arange(H, dtype=torch.float64, device="cuda") * (30.0 / H) - 15.0
        su, cu = torch.sin(u.deg2rad()), torch.cos(u.deg2rad())
        sv, cv = torch.sin(v.deg2rad()), torch.cos(v.deg2rad())
        return torch.stack([su[None] * cv[:, None], sv[:, None].expand(H, W),
                            cu[None] * cv[:, None]], -1)
    hw, hh = (math.tan(math.radians(a) / 2) for a in (87.0, 58.0))
    x = torch.arange(W, dtype=torch.float64, device="cuda") / W * 2 * hw - hw
    y = torch.arange(H, dtype=torch.float64, device="cuda") / H * 2 * hh - hh
    d = torch.stack([x[None].expand(H, W), y[:, None].expand(H, W), torch.ones_like(x[None]).expand(H, W)], -1)
    return d / d.norm(dim=-1, keepdim=True)


def _rotation(q):
    return torch.as_tensor(S.rotation_matrix(q), dtype=torch.float64, device="cuda")


def _scene_ranges(case, scene, pos, q, noise_seed):
    """(h, w) float32 ranges against the world's boxes and cylinders (0 = no return), with the
    range noise and dropped pixels of a real sensor."""
    d = (_pixel_dirs(case).reshape(-1, 3) @ _rotation(q).T).float()
    p = torch.tensor(pos, dtype=torch.float32, device="cuda")
    far = case["range"]
    best = torch.full((d.shape[0],), float("inf"), device="cuda")
    lo = torch.as_tensor(scene.boxes[:, :3], dtype=torch.float32, device="cuda")
    hi = torch.as_tensor(scene.boxes[:, 3:], dtype=torch.float32, device="cuda")
    near = torch.clamp(torch.maximum(lo - p, p - hi), min=0).norm(dim=1) <= far
    lo, hi = lo[near], hi[near]
    inv = 1.0 / torch.where(d.abs() < 1e-12, torch.full_like(d, 1e-12), d)
    for c in range(0, lo.shape[0], 64):
        ta = (lo[None, c:c + 64] - p) * inv[:, None]
        tb = (hi[None, c:c + 64] - p) * inv[:, None]
        t0 = torch.minimum(ta, tb).amax(-1)
        t1 = torch.maximum(ta, tb).amin(-1)
        best = torch.minimum(best, torch.where((t0 <= t1) & (t0 > 0), t0, float("inf")).amin(1))
    cyl = torch.as_tensor(scene.cylinders, dtype=torch.float32, device="cuda")
    if len(cyl):
        cyl = cyl[(cyl[:, :2] - p[:2]).norm(dim=1) - cyl[:, 2] <= far]
    a = d[:, 0] ** 2 + d[:, 1] ** 2
    for c in range(0, len(cyl), 32):
        cx, cy, r, z0, z1 = cyl[c:c + 32].T
        ox, oy = p[0] - cx, p[1] - cy
        b = d[:, :1] * ox + d[:, 1:2] * oy
        disc = b * b - a[:, None] * (ox * ox + oy * oy - r * r)
        t = (-b - disc.clamp(min=0).sqrt()) / a[:, None]
        z = p[2] + t * d[:, 2:]
        ok = (disc >= 0) & (t > 0) & (z >= z0) & (z <= z1)
        best = torch.minimum(best, torch.where(ok, t, float("inf")).amin(1))
    g = torch.Generator(device="cuda").manual_seed(noise_seed)
    r = best + torch.randn(best.shape, generator=g, device="cuda") * 0.005 * best.clamp(max=far) ** 2
    drop = torch.rand(best.shape, generator=g, device="cuda") < 0.02
    ok = (best <= far) & (r > 0.0) & (r < far) & ~drop
    return torch.where(ok, r, 0.0).float().reshape(case["height"], case["width"])


def _records(case, ranges):
    """PointCloud2-style records (x, y, z, 0), NaN where there is no return."""
    xyz = (_pixel_dirs(case) * ranges.double()[..., None]).float()
    xyz = torch.where(ranges[..., None] > 0, xyz, float("nan"))
    return torch.cat([xyz, torch.zeros_like(xyz[..., :1])], -1).contiguous()


def _frames(case, seed):
    """[(position, quaternion, range image, records or None)] of an insert case."""
    scene = _world(case["world"], case["res"], seed)
    out = []
    for k, (pos, q) in enumerate(_poses(case["world"], case["res"], seed, case["frames"])):
        r = _scene_ranges(case, scene, pos, q, (seed * 1009 + k) % (1 << 31))
        out.append((pos, q, r, _records(case, r) if case["input"] == "points" else None))
    return out


def _capacity(case, box_leaves):
    """A leaf table with room for the map and the frames in flight."""
    return 1 << max(14, math.ceil(math.log2(3.0 * box_leaves)))


def _reach_leaves(case):
    side = 2 * case["range"] / case["res"] / 8 + 2
    return min(side ** 3, 150000.0)


def _window(case, pos):
    """Leaf box (lo, n) of the read-back window: 3 m round `pos` (1.5 m up and down)."""
    v = np.asarray(pos, np.float64) / case["res"] / 8
    half = np.array([3.0, 3.0, 1.5]) / case["res"] / 8
    return np.floor(v - half).astype(np.int64), np.ceil(2 * half).astype(np.int64) + 1


def _window_slots(m, case, pos):
    """Table slot of every leaf of the window, (x, y, z) order; an empty (all zero) slot where
    the map holds no leaf."""
    lo, n = _window(case, pos)
    o = torch.from_numpy(m.slot_origins()).cuda().long()
    empty = int((o[:, 0] == -2 ** 31).nonzero()[0])
    leaf = (o >> 3) - torch.as_tensor(lo, device="cuda")
    dims = torch.as_tensor(n, device="cuda")
    inside = ((leaf >= 0) & (leaf < dims)).all(1) & (o[:, 0] != -2 ** 31)
    at = (leaf[:, 0] * n[1] + leaf[:, 1]) * n[2] + leaf[:, 2]
    slots = torch.full((int(n.prod()),), empty, dtype=torch.int64, device="cuda")
    slots[at[inside]] = inside.nonzero().flatten()
    return slots


def _map(ctx, case, leaves, agents=1):
    return A.Map(ctx, A.map_desc(
        res=case["res"], max_agents=agents, initial_leaf_capacity=_capacity(case, leaves),
        update_mode=N.NM_UPDATE_ACCUMULATE if case.get("mode") == "counts" else N.NM_UPDATE_LABEL,
        rounding=N.NM_ROUND_NEAREST if case.get("rounding") == "nearest" else N.NM_ROUND_DOWN))


# ---- preparation ---------------------------------------------------------------------------

def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _cast_rays(case, seed):
    pos = _poses(case["world"], case["res"], seed, 16)
    n = case["rays"]
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    o = np.array([pos[i % 16][0] for i in range(n)], np.float32)
    return o, d


def _prepare_cast(case, seed):
    ctx = A.Context(0)
    o, d = _cast_rays(case, seed)
    return dict(case=case, ctx=ctx, sim=_sim_map(ctx, _world(case["world"], case["res"], seed)),
                o=torch.from_numpy(o).cuda(), d=torch.from_numpy(d).cuda())


def _run_cast(s):
    return s["sim"].cast_rays(s["o"], s["d"], s["case"]["range"])


def _prepare_insert(case, seed):
    ctx = A.Context(0)
    sensor = A.Sensor(ctx, _desc(case))
    m = _map(ctx, case, _reach_leaves(case))
    frames = []
    for pos, q, r, rec in _frames(case, seed):
        x = rec if rec is not None else r
        frames.append((A.Pose(pos, q), x.cpu().pin_memory() if case["host"] else x))
    s = dict(case=case, ctx=ctx, sensor=sensor, map=m, frames=frames,
             flags=N.NM_FILTER_MEAN if case["filter"] else 0)
    _insert_all(s)
    s["slots"] = _window_slots(m, case, frames[len(frames) // 2][0].position)
    return s


def _insert_all(s):
    c, m, sensor = s["case"], s["map"], s["sensor"]
    for pose, x in s["frames"]:
        if c["input"] == "points":
            m.insert_points(sensor, pose, x, c["width"], c["height"], 16, flags=s["flags"])
        else:
            m.insert_ranges(sensor, pose, x, flags=s["flags"])


def _run_insert(s):
    _insert_all(s)
    return s["map"].values_copy()[s["slots"]]


def _prepare_sim(case, seed):
    ctx = A.Context(0)
    scene = _world(case["world"], case["res"], seed)
    s = dict(case=case, ctx=ctx, sensor=A.Sensor(ctx, _desc(case)), sim=_sim_map(ctx, scene),
             map=_map(ctx, case, _reach_leaves(case)), seed=seed % (1 << 31),
             poses=[A.Pose(p, q) for p, q in _poses(case["world"], case["res"], seed, case["frames"])],
             ranges=[torch.zeros(case["height"], case["width"], device="cuda") for _ in range(case["frames"])])
    _sim_frames(s)
    s["slots"] = _window_slots(s["map"], case, s["poses"][len(s["poses"]) // 2].position)
    return s


def _sim_frames(s):
    for k, (pose, r) in enumerate(zip(s["poses"], s["ranges"])):
        s["sim"].render_noisy(s["sensor"], pose, r, 0.005, 0.02, s["seed"] + k)
        s["map"].insert_ranges(s["sensor"], pose, r)


def _run_sim(s):
    _sim_frames(s)
    return dict(ranges=s["ranges"][-1], values=s["map"].values_copy()[s["slots"]])


def _prepare_tick(case, seed):
    ctx = A.Context(0)
    scene = _world(case["world"], case["res"], seed)
    sim = _sim_map(ctx, scene)
    # spread over the agents so that every count has sensors of each kind
    agents = [S.TICK_AGENTS[(i * 16) // case["agents"] if case["agents"] < 16 else i]
              for i in range(case["agents"])]
    sensors = [A.Sensor(ctx, A.sensor_desc(**S.tick_agent_desc_kwargs(a))) for a in agents]
    bufs = [torch.zeros(a[2], a[1], device="cuda") for a in agents]
    trajs = [[A.Pose(p, q) for p, q in _poses(case["world"], case["res"], seed, case["ticks"], which=1 + i)]
             for i in range(case["agents"])]
    m = _map(ctx, case, 300000.0 if case["res"] < 0.08 else 60000.0, agents=case["agents"])
    plan = A.TickPlan(m, [(sensors[i], bufs[i], i) for i in range(len(agents))], sim=sim)
    s = dict(case=case, ctx=ctx, sim=sim, sensors=sensors, ranges=bufs, trajs=trajs, map=m, plan=plan)
    _ticks(s)
    s["slots"] = _window_slots(m, case, trajs[0][-1].position)
    return s


def _ticks(s):
    for t in range(s["case"]["ticks"]):
        for i, traj in enumerate(s["trajs"]):
            s["plan"].set_pose(i, traj[t])
        s["plan"].run()


def _run_tick(s):
    _ticks(s)
    return dict(ranges=list(s["ranges"]), values=s["map"].values_copy()[s["slots"]])


def _prepare_render(case, seed):
    ctx = A.Context(0)
    scene = _world(case["world"], case["res"], seed)
    (pos, q), = _poses(case["world"], case["res"], seed, 1)
    sensor = A.Sensor(ctx, _desc(case))
    m = _map(ctx, case, 60000.0)
    pose = A.Pose(pos, q)
    r = _scene_ranges(case, scene, pos, q, seed % (1 << 31))
    m.insert_ranges(sensor, pose, r)
    p, R = A.Map.ray_pose(sensor, pose)
    return dict(case=case, ctx=ctx, sensor=sensor, map=m, pose=pose, ranges=r, position=p, rotation=R)


def _run_render(s):
    s["map"].insert_ranges(s["sensor"], s["pose"], s["ranges"])
    return s["map"].depth_render(s["sensor"], s["position"], s["rotation"], scale=4.0)


def _mapped(case, seed, n=4):
    """A map built from a few frames, and the pose of the last one."""
    s = _prepare_insert(dict(case, sensor="camera", frames=n, input="ranges", host=False,
                             filter=False, mode="label"), seed)
    pose, r = s["frames"][-1]
    p, R = A.Map.ray_pose(s["sensor"], pose)
    return s, r, p, R


def _prepare_gradients(case, seed):
    s, r, p, R = _mapped(case, seed)
    m = s["map"]
    s["case"] = case
    s.update(target=r, position=p, rotation=R, values=m.values_copy().requires_grad_(),
             xi=torch.zeros(6, requires_grad=True), scale=4.0)
    return s


def _run_gradients(s):
    s["values"].grad = None
    s["xi"].grad = None
    depth = diff.expected_depth(s["values"], s["xi"], s["map"], s["sensor"], s["position"],
                                s["rotation"], s["scale"], 0.0)
    seen = s["target"] > 0
    loss = ((depth - s["target"]) * seen).square().sum() / seen.sum()
    loss.backward()
    return dict(depth=depth.detach(), values_grad=s["values"].grad[s["slots"]],
                pose_grad=s["xi"].grad)


def _prepare_refine(case, seed):
    s, r, p, R = _mapped(case, seed)
    s["case"] = case
    rng = np.random.default_rng(seed)
    off = rng.uniform(-0.05, 0.05, 3)
    tilt = np.radians(rng.uniform(-2.0, 2.0, 3))
    s.update(target=r, position=p + off, rotation=diff.so3_exp(tilt) @ R)
    return s


def _run_refine(s):
    """The refined pose goes back into the mapping calls, which take 32-bit poses."""
    pos, R, losses = s["map"].pose_refine(s["sensor"], s["position"], s["rotation"], s["target"],
                                          steps=s["case"]["steps"], scale=12.0, max_residual=0.5,
                                          surface_offset=0.5, edge_threshold=0.2)
    return dict(position=pos.astype(np.float32), rotation=R.astype(np.float32), losses=losses)


# ---- work ----------------------------------------------------------------------------------

def _mean_visits(case):
    """Voxels a ray passes, about: a quarter of the range, 1.6 voxels per voxel length."""
    return 0.25 * case["range"] / case["res"] * 1.6


def work(case):
    k = case["kind"]
    if k == "cast":
        return dict(bytes=28.0 * case["rays"], flops=40.0 * case["rays"])
    if k == "tick":
        sensors = [S.TICK_AGENTS[(i * 16) // case["agents"] if case["agents"] < 16 else i]
                   for i in range(case["agents"])]
        px = sum(a[1] * a[2] for a in sensors)
        fl = sum(a[1] * a[2] * 0.25 * a[5] / case["res"] * 1.6 * 4 for a in sensors)
        return dict(bytes=case["ticks"] * 8.0 * px, flops=case["ticks"] * fl)
    px = case["width"] * case["height"]
    walk = px * _mean_visits(case)
    lo, n = _window(case, (0.0, 0.0, 0.0))
    window = 2048.0 * float(n.prod())
    if k == "insert":
        rec = 16.0 if case["input"] == "points" else 4.0
        return dict(bytes=case["frames"] * px * rec + window, flops=case["frames"] * walk * 4)
    if k == "sim":
        return dict(bytes=case["frames"] * px * 8.0 + window, flops=case["frames"] * walk * 5)
    if k == "render":
        return dict(bytes=px * 8.0, flops=walk * 16)
    if k == "gradients":
        return dict(bytes=px * 16.0 + 2 * window, flops=walk * 40)
    return dict(bytes=px * 4.0 * case["steps"], flops=walk * 30 * (case["steps"] + 1))


# ---- values in 64 bits ---------------------------------------------------------------------

def _crossings(eye, d, length):
    """Every lattice-plane crossing with t <= length along the rays eye + t d (unit d), in
    order: (ray, t, axis, voxel left (m, 3), voxel entered (m, 3))."""
    n = d.shape[0]
    v0 = torch.floor(eye).long()
    step = torch.sign(d).long()
    first = torch.where(step > 0, v0 + 1, v0).double() - eye
    inv = torch.where(step != 0, 1.0 / d, torch.zeros_like(d))
    t0 = first * inv
    cnt = torch.where(step != 0, torch.floor((length[:, None] - t0) * d.abs()).long() + 1, 0).clamp(min=0)
    rays, ts, axes = [], [], []
    ar = torch.arange(n, device=d.device)
    for a in (2, 1, 0):  # ties go to the higher axis: it comes first in a stable sort
        r = torch.repeat_interleave(ar, cnt[:, a])
        k = torch.arange(r.numel(), device=d.device) - torch.repeat_interleave(cnt[:, a].cumsum(0) - cnt[:, a], cnt[:, a])
        rays.append(r)
        ts.append(t0[r, a] + k.double() * inv[r, a].abs())
        axes.append(torch.full_like(r, a))
    ray, t, axis = torch.cat(rays), torch.cat(ts), torch.cat(axes)
    o = torch.sort(t, stable=True).indices
    o = o[torch.sort(ray[o], stable=True).indices]
    ray, t, axis = ray[o], t[o], axis[o]
    total = cnt.sum(1)
    start = total.cumsum(0) - total
    moves = torch.zeros(ray.numel(), 3, dtype=torch.int32, device=d.device)
    moves[torch.arange(ray.numel(), device=d.device), axis] = step[ray, axis].int()
    after = moves.cumsum(0)
    after = after - torch.where(start > 0, 1, 0).unsqueeze(1)[ray] * after[(start - 1).clamp(min=0)][ray] \
        if ray.numel() else after
    entered = v0.long() + after
    return ray, t, axis, entered - moves, entered, total, start


_KEY = 1 << 20


def _key(v):
    v = v.long() + (_KEY >> 1)
    return (v[:, 0] * _KEY + v[:, 1]) * _KEY + v[:, 2]


def _frame_labels(case, pos, q, points):
    """(keys of missed voxels, keys of hit voxels) of one frame, and their counts per voxel."""
    res = float(np.float32(case["res"]))
    mt = float(np.float32(case["range"])) / res
    eye = torch.tensor([float(np.float32(p)) for p in pos], dtype=torch.float64, device="cuda") / res
    d = points.double() @ _rotation(q).float().double().T
    ln = d.norm(dim=1) / res
    ok = (ln < mt) & (ln > 1e-7)
    d, ln = d[ok], ln[ok]
    d = d / d.norm(dim=1, keepdim=True)
    ray, t, axis, left, entered, total, start = _crossings(eye, d, ln)
    v0 = torch.floor(eye).long()
    end = v0.expand(d.shape[0], 3).clone()
    has = total > 0
    end[has] = entered[(start + total - 1)[has]]
    # the crossing that leaves the end voxel
    nxt = torch.where(d > 0, end + 1, end).double() - eye
    tn = torch.where(d != 0, nxt / d, float("inf")).amin(1)
    return _key(left), _key(end[tn < mt])


def _exact_points(case, r, rec):
    if rec is not None:
        x = rec.reshape(-1, 4)[:, :3]
        return x[~torch.isnan(x[:, 0])]
    return (_pixel_dirs(case) * r.double()[..., None]).reshape(-1, 3)[r.reshape(-1) > 0]


def _filtered(case, pos, q, points):
    """The voxel filter: one point per occupied voxel, the mean of its points (sensor frame)."""
    res = float(np.float32(case["res"]))
    eye = torch.tensor([float(np.float32(p)) for p in pos], dtype=torch.float64, device="cuda") / res
    R = _rotation(q)
    d = points.double() @ R.T
    ln = d.norm(dim=1) / res
    d = d[(ln < case["range"] / res) & (ln > 1e-7)]
    at = eye + d / res
    key, inv = torch.unique(_key(torch.floor(at)), return_inverse=True)
    mean = torch.zeros(key.numel(), 3, dtype=torch.float64, device="cuda").index_add_(0, inv, d)
    cnt = torch.zeros(key.numel(), dtype=torch.float64, device="cuda").index_add_(0, inv, torch.ones_like(d[:, 0]))
    return (mean / cnt[:, None]) @ R


def _exact_map(case, seed, passes=2):
    """{voxel key: log-odds} after `passes` passes over the frames, as sorted (keys, values)."""
    per_frame = []
    for pos, q, r, rec in _frames(case, seed):
        p = _exact_points(case, r, rec)
        if case["filter"]:
            p = _filtered(case, pos, q, p)
        miss, hit = _frame_labels(case, pos, q, p)
        if case["mode"] == "counts":
            k, inv = torch.unique(torch.cat([miss, hit]), return_inverse=True)
            w = torch.cat([torch.full_like(miss, -0.4, dtype=torch.float64), torch.full_like(hit, 0.85, dtype=torch.float64)])
            per_frame.append((k, torch.zeros(k.numel(), dtype=torch.float64, device="cuda").index_add_(0, inv, w)))
        else:
            miss, hit = torch.unique(miss), torch.unique(hit)
            k = torch.unique(torch.cat([miss, hit]))
            up = torch.isin(k, hit)
            per_frame.append((k, torch.where(up, 0.85, -0.4).double()))
    keys = torch.unique(torch.cat([k for k, _ in per_frame]))
    val = torch.zeros(keys.numel(), dtype=torch.float64, device="cuda")
    for _ in range(passes):
        for k, w in per_frame:
            i = torch.searchsorted(keys, k)
            val[i] = (val[i] + w).clamp(-2.0, 3.5)
    return keys, val


def _exact_window(case, pos, keys, val):
    lo, n = _window(case, pos)
    ax = [torch.arange(int(n[a]) * 8, device="cuda") + int(lo[a]) * 8 for a in range(3)]
    g = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    k = _key(g)
    i = torch.searchsorted(keys, k).clamp(max=keys.numel() - 1)
    v = torch.where(keys[i] == k, val[i], 0.0)
    v = v.reshape(int(n[0]), 8, int(n[1]), 8, int(n[2]), 8).permute(0, 2, 4, 1, 3, 5)
    return v.reshape(-1, 512)


def _voxel_grid(case, seed):
    """The world's occupied voxels as a dense grid: a voxel is on when its centre lies in a box
    or a cylinder."""
    scene = _world(case["world"], case["res"], seed)
    res = float(np.float32(case["res"]))
    grid = torch.zeros(*scene.vox_max, dtype=torch.bool, device="cuda")
    ax = [(torch.arange(k, dtype=torch.float64, device="cuda") + 0.5) * res for k in scene.vox_max]
    for b in scene.boxes:
        sl = [(int(torch.searchsorted(ax[a], float(b[a]))), int(torch.searchsorted(ax[a], float(b[3 + a]), right=True)))
              for a in range(3)]
        grid[sl[0][0]:sl[0][1], sl[1][0]:sl[1][1], sl[2][0]:sl[2][1]] = True
    for cx, cy, r, z0, z1 in scene.cylinders:
        on = ((ax[0] - cx)[:, None] ** 2 + (ax[1] - cy)[None] ** 2) <= r * r
        grid |= on[:, :, None] & ((ax[2] >= z0) & (ax[2] <= z1))[None, None]
    return grid


def _exact_cast(case, seed):
    grid = _voxel_grid(case, seed)
    res = float(np.float32(case["res"]))
    o, d = (torch.from_numpy(x).cuda().double() for x in _cast_rays(case, seed))
    d = d / d.norm(dim=1, keepdim=True)
    out = torch.zeros(d.shape[0], dtype=torch.float64, device="cuda")
    mt = float(np.float32(case["range"])) / res
    dims = torch.tensor(grid.shape, device="cuda")
    for k in range(16):  # rays of one origin at a time
        at = torch.arange(k, d.shape[0], 16, device="cuda")
        if not at.numel():
            continue
        eye = o[k] / res
        L = torch.full((at.numel(),), mt, dtype=torch.float64, device="cuda")
        ray, t, _, _, v, total, start = _crossings(eye, d[at], L)
        ins = ((v >= 0) & (v < dims)).all(1)
        w = v.clamp(min=0).minimum(dims - 1)
        hit = ins & grid[w[:, 0], w[:, 1], w[:, 2]]
        best = torch.full((at.numel(),), float("inf"), dtype=torch.float64, device="cuda")
        best = best.scatter_reduce(0, ray[hit], t[hit], "amin")
        out[at] = torch.where(torch.isinf(best), 0.0, best * res)
    return out


def _exact_gradients(case, seed):
    case4 = dict(case, sensor="camera", frames=4, input="ranges", host=False, filter=False, mode="label")
    keys, val = _exact_map(case4, seed, passes=1)
    frames = _frames(case4, seed)
    pos, q, r, _ = frames[-1]
    res = float(np.float32(case["res"]))
    t_max = float(np.float32(case["range"])) / res
    R = _rotation(q)
    p = torch.tensor([float(np.float32(x)) for x in pos], dtype=torch.float64, device="cuda")
    dirs = _pixel_dirs(case).reshape(-1, 3)
    n = dirs.shape[0]
    seen = r.reshape(-1) > 0
    target = r.reshape(-1).double()
    val = val.requires_grad_()
    depth = torch.zeros(n, dtype=torch.float64, device="cuda")
    gv = torch.zeros_like(val)
    gx = torch.zeros(6, dtype=torch.float64, device="cuda")
    for c in range(0, n, 40000):
        xi = torch.zeros(6, dtype=torch.float64, device="cuda", requires_grad=True)
        d0 = dirs[c:c + 40000] @ R.T
        with torch.no_grad():
            ray, t, axis, left, v, total, start = _crossings(p / res, d0, torch.full((d0.shape[0],), t_max, dtype=torch.float64, device="cuda"))
            plane = torch.maximum(v, left).gather(1, axis[:, None]).squeeze(1).double()
            i = torch.searchsorted(keys, _key(v)).clamp(max=keys.numel() - 1)
            known = keys[i] == _key(v)
            last = torch.zeros_like(ray, dtype=torch.bool)
            last[(start + total - 1)[total > 0]] = True
        e = (p + xi[:3]) / res
        d = d0 + torch.cross(xi[3:].expand_as(d0), d0, dim=1)
        te = (plane - e[axis]) / d[ray, axis]
        tout = torch.where(last, torch.full_like(te, t_max), torch.roll(te, -1))
        L = torch.where(known, val[i], torch.zeros((), dtype=torch.float64, device="cuda"))
        sg = torch.nn.functional.softplus(4.0 * L, threshold=1e9)
        u = sg * (tout - te)
        cum = u.cumsum(0)
        off = torch.where(start > 0, cum[(start - 1).clamp(min=0)], torch.zeros((), dtype=torch.float64, device="cuda"))
        T = torch.exp(-(cum - u - off[ray]).clamp(min=0))
        seg = T * (-torch.expm1(-u)) / sg
        D = torch.zeros(d0.shape[0], dtype=torch.float64, device="cuda").index_add(0, ray, seg)
        has = total > 0
        D = D + torch.where(has, te[start.clamp(max=max(te.numel() - 1, 0))], torch.full_like(D, t_max))
        D = D * res
        loss = (((D - target[c:c + 40000]) * seen[c:c + 40000]) ** 2).sum() / seen.sum()
        g = torch.autograd.grad(loss, [val, xi])
        gv += g[0]
        gx += g[1]
        depth[c:c + 40000] = D.detach()
    return dict(depth=depth.reshape(case["height"], case["width"]),
                values_grad=_exact_window(case, frames[2][0], keys, gv), pose_grad=gx.cpu())


def exact(case, seed):
    k = case["kind"]
    if k == "cast":
        return _exact_cast(case, seed)
    if k == "insert":
        keys, val = _exact_map(case, seed)
        frames = _poses(case["world"], case["res"], seed, case["frames"])
        return _exact_window(case, frames[case["frames"] // 2][0], keys, val)
    if k == "gradients":
        return _exact_gradients(case, seed)
    # simulated ranges end exactly on voxel faces, where 32-bit and 64-bit walks label different
    # voxels; a refinement's path and the large map's walk take too long in plain torch
    return None
