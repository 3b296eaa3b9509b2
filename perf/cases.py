"""Performance cases: the calls a program that maps with this package makes, one pass at a time.

Every case is a dict of plain values with a "kind":

  preprocess  what each camera frame goes through before the tracker: downsample_depth and
              bilateral_filter
  query       a planner's batch of field values and gradients on a TSDF map
  track       one blocking Tracker.track of a depth frame against a raycast of the map
  map         mapping at known poses: integrateDepth, then raycast_volume at the same pose
  frame       the tracked frame loop: FramePipeline.run from a pinned host frame (bilateral
              filter, track, integrate, raycast) and the asynchronous pose read
  occupancy   a depth camera's occupancy map: integrateDepth, then raycast_volume
  lidar       one step of a fleet of LiDAR occupancy maps (OccupancyBatch.integrate and its
              counters), and a view of one of the maps
  rays        a Leica scan integrated ray by ray (integrate_ray_batch), and a view of the map
  render      one step of gradient pose and map refinement: render_depth forward, a Huber loss's
              gradient, raycast_adjoint backward into the twist and the voxels

The sensors, scenes, resolutions and options are those of the repository's tests and benchmark
(room of 6 x 5 x 3 m seen by a depth camera, outdoor scene driven through by 64-beam LiDARs) and
sizes around them. Maps hold some frames already when a pass begins, and successive passes go back
and forth along a short trajectory, so that the first passes allocate blocks and all of them
update old ones.
"""
import math

import numpy as np
import torch

import supereight2_gb300 as se
from supereight2_gb300 import synthetic as syn

DIM = 10.24           # side of the room's map in metres
FRAMES = 6            # frames of a trajectory that the passes go back and forth on
HALF = 3              # frames that the map holds before the first pass
LAP = 12              # frames of the tracked loop's trajectory
TRACKED_NOISE = 0.003  # depth noise of the tracked frames (m per m^2): a structured-light camera's


# ------------------------------------------------------------------------------ the cases --

def listed():
    return [
        # the sensor's full frame halved and filtered: the smallest calls, two launches
        dict(name="preprocess_640", kind="preprocess", width=640, height=480, ratio=2, radius=2),
        # a planner checks the clearance and its gradient along sampled trajectories
        dict(name="query_50k", kind="query", points=50_000, res=0.02, storage="f32"),
        # the tracker's blocking call at the usual camera size
        dict(name="track_640", kind="track", width=640, height=480, res=0.01),
        # mapping from a half-size camera at 2 cm with ground-truth poses
        dict(name="map_320", kind="map", width=320, height=240, res=0.02, storage="f32", multi=False),
        # full camera at 1 cm, compact voxels
        dict(name="map_640_f16", kind="map", width=640, height=480, res=0.01, storage="f16", multi=False),
        # a megapixel depth camera into a multi-resolution map: the largest integration
        dict(name="map_1280_multi", kind="map", width=1280, height=960, res=0.01, storage="f32", multi=True),
        # the whole tracked loop, the headline configuration
        dict(name="frame_640", kind="frame", width=640, height=480, res=0.01, storage="f32", multi=False),
        # the same loop on the multi-resolution map with compact voxels
        dict(name="frame_640_multi_f16", kind="frame", width=640, height=480, res=0.01, storage="f16", multi=True),
        # occupancy mapping for exploration from a depth camera
        dict(name="occupancy_320", kind="occupancy", width=320, height=240, res=0.02),
        # eight vehicles' maps fed together
        dict(name="lidar_8", kind="lidar", maps=8, columns=1024, beams=64),
        # a terrestrial scanner's sweep: rays in scan order, all from one place
        dict(name="rays_8k", kind="rays", columns=160, beams=96),
        # refinement of a pose and of the voxels against a held-out frame
        dict(name="render_640", kind="render", width=640, height=480, res=0.01),
    ]


def _between(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _camera_size(rng, lo, hi):
    w = _between(rng, lo, hi)
    return w, max(96, int(w * rng.uniform(0.55, 0.8)))


def draw(rng):
    kind = rng.choice(["preprocess", "query", "track", "map", "map", "frame", "frame", "occupancy", "lidar", "rays",
                       "render"])
    if kind == "preprocess":
        ratio = rng.choice([1, 2, 2, 3, 4])
        w, h = _camera_size(rng, 160, 960)
        return dict(kind=kind, width=w * ratio, height=h * ratio, ratio=ratio, radius=rng.choice([1, 2, 2, 3, 5]))
    if kind == "query":
        return dict(kind=kind, points=_between(rng, 1_000, 2_000_000), res=rng.choice([0.02, 0.04]),
                    storage=rng.choice(["f32", "f16"]))
    if kind == "track":
        w, h = _camera_size(rng, 160, 560)
        return dict(kind=kind, width=w, height=h, res=rng.choice([0.01, 0.02]))
    if kind in ("map", "frame"):
        w, h = _camera_size(rng, 160, 1024 if kind == "map" else 560)
        return dict(kind=kind, width=w, height=h, res=rng.choice([0.01, 0.02, 0.04]),
                    storage=rng.choice(["f32", "f16"]), multi=rng.random() < 0.4)
    if kind == "occupancy":
        w, h = _camera_size(rng, 160, 480)
        return dict(kind=kind, width=w, height=h, res=rng.choice([0.02, 0.04]))
    if kind == "lidar":
        return dict(kind=kind, maps=rng.choice([1, 2, 3, 4, 6, 8]), columns=_between(rng, 360, 1024),
                    beams=_between(rng, 16, 64))
    if kind == "rays":
        return dict(kind=kind, columns=_between(rng, 40, 150), beams=_between(rng, 16, 90))
    w, h = _camera_size(rng, 160, 800)
    return dict(kind=kind, width=w, height=h, res=rng.choice([0.01, 0.02]))


# ---------------------------------------------------------------------------- the inputs --

def _spec(w, h):
    f = 525.0 * w / 640.0
    return syn.PinholeSpec(w, h, f, f, (w - 1) / 2.0, (h - 1) / 2.0, 0.4, 6.0)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _depth(scene, spec, T, gen, noise):
    """A depth frame on the GPU: the scene traced, noise that grows with the squared range, 2 % missing."""
    z = torch.from_numpy(syn.render_depth(scene, spec, T, 0, device="cuda", noise=False)).cuda()
    z = z + torch.randn(z.shape, generator=gen, device="cuda") * (noise * z * z)
    drop = torch.rand(z.shape, generator=gen, device="cuda") < 0.02
    return torch.where(drop, torch.zeros_like(z), z).contiguous()


def _room(spec, seed, frames=FRAMES, noise=0.0015):
    scene = syn.make_scene(int(seed) % (1 << 31))
    # a camera carried by hand, 30 frames a second: about a centimetre and half a degree a frame
    walk = syn.random_walk_trajectory(frames, seed=int(seed) % (1 << 31) + 1, sigma_m=0.005, sigma_deg=0.3)
    poses = [T.astype(np.float32) for T in walk]
    gen = _generator(seed)
    return poses, [_depth(scene, spec, T, gen, noise) for T in poses]


def _to_and_fro(k, n=FRAMES):
    """0, 1, ..., n - 1, n - 2, ..., 1, 0, 1, ..."""
    k %= 2 * n - 2
    return k if k < n else 2 * n - 2 - k


def _tsdf_map(case, seed, camera, poses, depths, held=HALF):
    m = se.Map(DIM, case["res"], max_blocks=1 << 17 if case["res"] < 0.015 else 1 << 15,
               storage=case.get("storage", "f32"), res_type="multi" if case.get("multi") else "single")
    integrator = se.MapIntegrator(m)
    for k in range(held):
        integrator.integrateDepth(k, depths[k], camera, poses[k])
    m.check()
    return m, integrator


def _images(h, w):
    pts = torch.zeros((h, w, 3), device="cuda")
    return pts, torch.zeros_like(pts), torch.zeros((h, w), dtype=torch.int8, device="cuda")


def _forward_view(T):
    """The pose of a camera (z forward, y down) that looks along x of a vehicle (x forward, z up)."""
    C = np.eye(4, dtype=np.float32)
    C[:3, :3] = [[0, 0, 1], [-1, 0, 0], [0, -1, 0]]
    return (np.asarray(T, np.float32) @ C).astype(np.float32)


# An analytic field for the query cases: the room's walls and the scene's spheres, in voxels' centres.
def _room_sdf(scene, p):
    half = torch.as_tensor(scene.room_half, dtype=p.dtype, device=p.device)
    d = (half - p.abs()).amin(-1)
    for c, r in zip(scene.sphere_c, scene.sphere_r):
        d = torch.minimum(d, (p - torch.as_tensor(c, dtype=p.dtype, device=p.device)).norm(dim=-1) - float(r))
    return d


def _query_field(case, seed):
    """(blocks' coordinates [N, 3] in voxels, tsdf [N, 512], map size in voxels, points [P, 3])."""
    res = case["res"]
    scene = syn.make_scene(int(seed) % (1 << 31))
    size = 1 << max(4, math.ceil(math.log2(DIM / res)))
    side = size // 8
    b = torch.arange(side, device="cuda")
    blocks = torch.stack(torch.meshgrid(b, b, b, indexing="ij"), -1).reshape(-1, 3) * 8
    centre = (blocks.double() + 4.0) * res - DIM / 2
    trunc = 8 * res
    blocks = blocks[_room_sdf(scene, centre).abs() < trunc + 8 * res]
    v = torch.arange(512, device="cuda")
    local = torch.stack([v % 8, v // 8 % 8, v // 64], -1)
    centres = ((blocks[:, None, :] + local[None]).double() + 0.5) * res - DIM / 2
    tsdf = (_room_sdf(scene, centres) / trunc).clamp(-1, 1).float()
    # points near the surfaces, where a planner asks
    gen = _generator(seed)
    n = case["points"]
    at = torch.randint(0, blocks.shape[0], (n,), generator=gen, device="cuda")
    pts = (blocks[at].double() + 8 * torch.rand((n, 3), generator=gen, device="cuda").double()) * res - DIM / 2
    return blocks, tsdf, size, pts.float().contiguous()


def _block_keys(blocks):
    code = np.zeros(len(blocks), np.uint64)
    for bit in range(19):
        for a in range(3):
            code |= ((blocks[:, a].astype(np.uint64) >> np.uint64(bit)) & np.uint64(1)) << np.uint64(3 * bit + a)
    return (code << np.uint64(5)) | np.uint64(3)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------------- preprocess --

def _prepare_preprocess(case, seed):
    spec = _spec(case["width"], case["height"])
    _, depths = _room(spec, seed, 1)
    h, w = case["height"] // case["ratio"], case["width"] // case["ratio"]
    return dict(kind="preprocess", depth=depths[0], small=torch.zeros((h, w), device="cuda"),
                map=torch.zeros((h, w), dtype=torch.int64, device="cuda"), out=torch.zeros((h, w), device="cuda"),
                radius=case["radius"])


def _run_preprocess(s):
    se.downsample_depth(s["depth"], s["small"], s["map"])
    se.bilateral_filter(s["small"], s["out"], radius=s["radius"])
    return {"small": s["small"], "map": s["map"], "filtered": s["out"]}


def _exact_preprocess(case, seed):
    d = _prepare_preprocess(case, seed)["depth"].double()
    r, R = case["ratio"], case["radius"]
    h, w = d.shape[0] // r, d.shape[1] // r
    win = d.reshape(h, r, w, r).permute(0, 2, 1, 3).reshape(h, w, r * r)
    ok = win >= np.float32(1e-5).item()
    n = ok.sum(-1)
    srt = torch.where(ok, win, torch.full_like(win, math.inf)).sort(-1).values
    small = srt.gather(-1, (n // 2).clamp(max=r * r - 1)[..., None])[..., 0]
    small = torch.where(n > 0, small, torch.zeros_like(small))
    pad = torch.nn.functional.pad(small[None, None], (R, R, R, R))[0, 0]
    num, den = torch.zeros_like(small), torch.zeros_like(small)
    for dy in range(-R, R + 1):
        for dx in range(-R, R + 1):
            tap = pad[R + dy:R + dy + h, R + dx:R + dx + w]
            wgt = math.exp(-(dx * dx + dy * dy) / (2 * 4.0 ** 2)) * torch.exp(-(tap - small) ** 2 / (2 * 0.03 ** 2))
            wgt = torch.where(tap > 0, wgt, torch.zeros_like(wgt))
            num, den = num + wgt * tap, den + wgt
    out = torch.where(small > 0, num / den.clamp(min=1e-300), torch.zeros_like(small))
    return {"small": small, "map": None, "filtered": out}


# --------------------------------------------------------------------------------- query --

def _prepare_query(case, seed):
    blocks, tsdf, _, pts = _query_field(case, seed)
    m = se.Map(DIM, case["res"], storage=case["storage"], max_blocks=1 << 17)
    keys = _block_keys(blocks.cpu().numpy())
    m.upload_blocks(keys, tsdf.cpu().numpy(), np.ones((len(keys), 1), np.float32))
    m.check()
    return dict(kind="query", map=m, points=pts)


def _run_query(s):
    value, has_value = s["map"].getFieldInterp(s["points"])
    grad, has_grad = s["map"].getFieldGrad(s["points"])
    return {"value": value, "has_value": has_value, "grad": grad, "has_grad": has_grad}


def _exact_query(case, seed):
    blocks, tsdf, size, pts = _query_field(case, seed)
    grid = torch.full((size, size, size), math.nan, dtype=torch.float64, device="cuda")   # [z, y, x]
    v = torch.arange(512, device="cuda")
    x = blocks[:, 0, None] + v % 8
    y = blocks[:, 1, None] + v // 8 % 8
    z = blocks[:, 2, None] + v // 64
    grid[z, y, x] = tsdf.double()
    # voxel coordinates less half a voxel; the cell's lower corner
    b = (pts.double() + DIM / 2) / case["res"] - 0.5
    lo = b.floor().long()
    t = b - lo

    def at(ox, oy, oz):
        c = [(lo[:, a] + o).clamp(0, size - 1) for a, o in enumerate((ox, oy, oz))]
        return grid[c[2], c[1], c[0]]

    value = torch.zeros(len(pts), dtype=torch.float64, device="cuda")
    grad = torch.zeros((len(pts), 3), dtype=torch.float64, device="cuda")
    for i in range(2):
        for j in range(2):
            for k in range(2):
                w = (t[:, 0] if i else 1 - t[:, 0]) * (t[:, 1] if j else 1 - t[:, 1]) * (t[:, 2] if k else 1 - t[:, 2])
                value += w * at(i, j, k)
                for a, e in enumerate(((1, 0, 0), (0, 1, 0), (0, 0, 1))):
                    up, dn = at(i + e[0], j + e[1], k + e[2]), at(i - e[0], j - e[1], k - e[2])
                    grad[:, a] += w * 0.5 * (up - dn) / case["res"]
    grad = torch.where(grad.isnan().any(-1, keepdim=True), torch.zeros_like(grad), grad)
    return {"value": torch.nan_to_num(value), "has_value": None, "grad": grad, "has_grad": None}


# --------------------------------------------------------------------------------- track --

def _prepare_track(case, seed):
    spec = _spec(case["width"], case["height"])
    camera = se.PinholeCamera.from_spec(spec)
    poses, depths = _room(spec, seed, noise=TRACKED_NOISE)
    m, _ = _tsdf_map(case, seed, camera, poses, depths)
    pts, nrm, scale = _images(spec.height, spec.width)
    se.raycast_volume(m, camera, poses[HALF - 1], pts, nrm, scale)
    return dict(kind="track", tracker=se.Tracker(m, camera), depth=se.bilateral_filter(depths[HALF]), pts=pts, nrm=nrm,
                T=poses[HALF - 1])


def _run_track(s):
    T = s["T"].copy()
    accepted = s["tracker"].track(s["depth"], T, s["pts"], s["nrm"])
    return {"T_WS": T, "accepted": accepted}


# ----------------------------------------------------------------------------------- map --

def _prepare_map(case, seed):
    spec = _spec(case["width"], case["height"])
    camera = se.PinholeCamera.from_spec(spec)
    poses, depths = _room(spec, seed)
    m, integrator = _tsdf_map(case, seed, camera, poses, depths)
    pts, nrm, scale = _images(spec.height, spec.width)
    return dict(kind="map", map=m, integrator=integrator, camera=camera, poses=poses, depths=depths, pts=pts, nrm=nrm,
                scale=scale, k=HALF)


def _run_map(s):
    k = s["k"]
    s["k"] = k + 1
    i = _to_and_fro(k)
    s["integrator"].integrateDepth(k, s["depths"][i], s["camera"], s["poses"][i])
    se.raycast_volume(s["map"], s["camera"], s["poses"][i], s["pts"], s["nrm"], s["scale"])
    return {"points": s["pts"], "normals": s["nrm"], "scale": s["scale"]}


# --------------------------------------------------------------------------------- frame --

def _prepare_frame(case, seed):
    spec = _spec(case["width"], case["height"])
    camera = se.PinholeCamera.from_spec(spec)
    poses, depths = _room(spec, seed, LAP, TRACKED_NOISE)
    m, _ = _tsdf_map(case, seed, camera, poses, depths, held=0)
    tracker = se.Tracker(m, camera)
    pipe = se.FramePipeline(m, camera, tracker)
    pipe.set_bilateral(**se.BILATERAL_DEFAULTS)
    host = [d.cpu().pin_memory() for d in depths]
    pipe.set_pose(poses[0])
    pipe.run(track=False, depth=host[0])
    for k in range(1, HALF):
        pipe.run(track=True, depth=host[k])
    m.check()
    return dict(kind="frame", pipe=pipe, host=host, T0=poses[0], pose=torch.zeros(12, pin_memory=True),
                accepted=torch.zeros(1, dtype=torch.int32, pin_memory=True), k=HALF)


def _run_frame(s):
    k = s["k"]
    s["k"] = k + 1
    i, pipe = _to_and_fro(k, LAP), s["pipe"]
    if i == 0:   # a lap is closed: its first frame at the known start, so that no drift builds up
        pipe.set_pose(s["T0"], k)
    pipe.run(track=i > 0, depth=s["host"][i])
    pipe.pose_async(s["pose"], s["accepted"])
    return {"points": pipe.points_W, "normals": pipe.normals_W, "pose": s["pose"], "accepted": s["accepted"]}


# ----------------------------------------------------------------------------- occupancy --

def _prepare_occupancy(case, seed):
    spec = _spec(case["width"], case["height"])
    camera = se.PinholeCamera.from_spec(spec)
    poses, depths = _room(spec, seed)
    m = se.Map(DIM, case["res"], res_type="multi", field="occupancy",
               max_blocks=1 << 17 if case["res"] < 0.03 else 1 << 15)
    integrator = se.MapIntegrator(m)
    for k in range(HALF):
        integrator.integrateDepth(k, depths[k], camera, poses[k])
    m.check()
    pts, nrm, scale = _images(spec.height, spec.width)
    return dict(kind="map", map=m, integrator=integrator, camera=camera, poses=poses, depths=depths, pts=pts, nrm=nrm,
                scale=scale, k=HALF)


# --------------------------------------------------------------------------------- lidar --

LIDAR_T_MW = np.eye(4, dtype=np.float32)
LIDAR_T_MW[:3, 3] = (51.2, 51.2, 12.8)


def _scan(scene, spec, T, keep, gen):
    r = torch.from_numpy(syn.render_range(scene, spec, T, 0, device="cuda", noise=False)).cuda()
    r = torch.where(r > 0, r + 0.01 * torch.randn(r.shape, generator=gen, device="cuda"), r)
    return torch.where(torch.rand(r.shape, generator=gen, device="cuda") < keep, r, torch.zeros_like(r))


def _prepare_lidar(case, seed):
    n = case["maps"]
    spec = syn.LidarSpec(width=case["columns"], height=case["beams"])
    sensor = se.OusterLidar.from_spec(spec)
    scene = syn.make_outdoor_scene(int(seed) % (1 << 31))
    gen = _generator(seed)
    poses = [syn.road_trajectory(k, 4, phase=0.7 * k) for k in range(n)]
    keep = [0.40 + 0.55 * k / max(n - 1, 1) for k in range(n)]
    scans = [torch.stack([_scan(scene, spec, poses[k][i], keep[k], gen) for k in range(n)]) for i in range(4)]
    T = [np.stack([poses[k][i] for k in range(n)]).astype(np.float32) for i in range(4)]
    maps = [se.Map(102.4, 0.4, res_type="multi", field="occupancy", T_MW=LIDAR_T_MW, max_blocks=1 << 14)
            for _ in range(n)]
    batch = se.OccupancyBatch(maps, sensor, graph=True)
    for i in range(2):
        batch.integrate(scans[i], T[i], i)
    for m in maps:
        m.check()
    view = se.PinholeCamera(160, 120, 131.25, 131.25, 79.5, 59.5, 0.4, 40.0)
    pts, nrm, scale = _images(120, 160)
    return dict(kind="lidar", batch=batch, maps=maps, scans=scans, T=T, view=view, pts=pts, nrm=nrm, scale=scale,
                stats=torch.zeros((n, 4), dtype=torch.int32, pin_memory=True), k=2)


def _run_lidar(s):
    k = s["k"]
    s["k"] = k + 1
    i = _to_and_fro(k, 4)
    s["batch"].integrate(s["scans"][i], s["T"][i], k)
    s["batch"].stats_async(s["stats"])
    at = k % len(s["maps"])
    se.raycast_volume(s["maps"][at], s["view"], _forward_view(s["T"][i][at]), s["pts"], s["nrm"], s["scale"])
    return {"stats": s["stats"], "points": s["pts"], "normals": s["nrm"], "scale": s["scale"]}


# ---------------------------------------------------------------------------------- rays --

def _prepare_rays(case, seed):
    # a terrestrial scanner: columns in scan order, its beams up each column
    spec = syn.LidarSpec(width=case["columns"], height=case["beams"], far_plane=30.0)
    scene = syn.make_outdoor_scene(int(seed) % (1 << 31))
    gen = _generator(seed)
    T = syn.road_trajectory(int(seed) % 8, 1)[0].astype(np.float32)
    r = _scan(scene, spec, T, 0.95, gen)
    d = torch.as_tensor(syn.lidar_directions(spec), device="cuda")
    rays = (d * r[..., None].double()).permute(1, 0, 2).reshape(-1, 3).float()
    rays = rays[(r.T.reshape(-1) > 0)].contiguous()
    poses = torch.from_numpy(T).cuda()[None].expand(len(rays), 4, 4).contiguous()
    m = se.Map(102.4, 0.2, res_type="multi", field="occupancy", T_MW=LIDAR_T_MW, max_blocks=1 << 16)
    view = se.PinholeCamera(160, 120, 131.25, 131.25, 79.5, 59.5, 0.4, 30.0)
    pts, nrm, scale = _images(120, 160)
    return dict(kind="rays", map=m, rays=rays, poses=poses, sensor=se.LeicaLidar(), view=view, T=_forward_view(T),
                pts=pts, nrm=nrm, scale=scale, k=0)


def _run_rays(s):
    k = s["k"]
    s["k"] = k + 1
    n = se.integrate_ray_batch(s["map"], k, s["poses"], s["rays"], s["sensor"], with_octants=False)
    se.raycast_volume(s["map"], s["view"], s["T"], s["pts"], s["nrm"], s["scale"])
    return {"octants": n, "points": s["pts"], "normals": s["nrm"], "scale": s["scale"]}


# -------------------------------------------------------------------------------- render --

def _prepare_render(case, seed):
    spec = _spec(case["width"], case["height"])
    camera = se.PinholeCamera.from_spec(spec)
    poses, depths = _room(spec, seed)
    m = se.Map(DIM, case["res"], max_blocks=1 << 15 if case["res"] < 0.015 else 1 << 13)
    integrator = se.MapIntegrator(m)
    for k in range(FRAMES - 1):
        integrator.integrateDepth(k, depths[k], camera, poses[k])
    m.check()
    # the pool's blocks by key, so that the gradients' rows are in an order that programs can name
    keys = m.download_blocks(voxels=False)[0]
    order = torch.from_numpy(np.concatenate([np.argsort(keys), np.arange(len(keys), m.max_blocks)])).cuda()
    rng = np.random.default_rng(int(seed) % (1 << 31))
    T = poses[FRAMES - 1].copy()
    T[:3, 3] += rng.normal(0.0, 0.01, 3).astype(np.float32)
    return dict(kind="render", map=m, camera=camera, T=T, target=depths[FRAMES - 1], order=order,
                depth=torch.zeros((spec.height, spec.width), device="cuda"),
                twist=torch.zeros(6, dtype=torch.float64, device="cuda"),
                voxels=torch.zeros((m.max_blocks, 512), device="cuda"))


def _run_render(s):
    d = se.render_depth(s["map"], s["camera"], s["T"], out=s["depth"])
    # Huber (0.02 m) on the pixels that both have, averaged
    g = ((d - s["target"]) * 50.0).clamp_(-1.0, 1.0) * ((d > 0) & (s["target"] > 0)) / d.numel()
    s["twist"].zero_()
    s["voxels"].zero_()
    se.raycast_adjoint(s["map"], s["camera"], s["T"], g, s["twist"], s["voxels"])
    return {"depth": d, "twist": s["twist"], "voxels": s["voxels"].index_select(0, s["order"])}


_PREPARE = dict(preprocess=_prepare_preprocess, query=_prepare_query, track=_prepare_track, map=_prepare_map,
                frame=_prepare_frame, occupancy=_prepare_occupancy, lidar=_prepare_lidar, rays=_prepare_rays,
                render=_prepare_render)
_RUN = dict(preprocess=_run_preprocess, query=_run_query, track=_run_track, map=_run_map, frame=_run_frame,
            lidar=_run_lidar, rays=_run_rays, render=_run_render)


def exact(case, seed):
    """The outputs in 64 bits where they are formulas of the inputs. The raycasts, the tracker and the
    maps take discrete decisions on float values (a voxel's pixel, an outlier gate, the sample that
    crosses the surface), which another precision takes otherwise: no value for those."""
    if case["kind"] == "preprocess":
        return _exact_preprocess(case, seed)
    if case["kind"] == "query":
        return _exact_query(case, seed)
    return None


# ------------------------------------------------------------------------- the least work --

# The room as the camera sees it: the mean depth of a frame, and so the surface a frame covers.
MEAN_DEPTH = 2.2


def _surface_voxels(case):
    """Voxel faces of the surface that a frame covers: its area over the area of one face."""
    f = 525.0 * case["width"] / 640.0
    return case["width"] * case["height"] * (MEAN_DEPTH / f) ** 2 / case["res"] ** 2


def _voxel_bytes(case):
    return (4 if case.get("storage") == "f16" else 8) * (2 if case.get("multi") else 1)


def _integrate_work(case):
    # the band of 2 x 8 voxels about the surface, read and written once; the frame read once
    v = 16 * _surface_voxels(case)
    return {"bytes": 2 * v * _voxel_bytes(case) + 4 * case["width"] * case["height"], "flops": 40 * v}


def _raycast_work(case):
    # points, normals and scales written; the voxels beside the surface that the gradient reads
    px = case["width"] * case["height"]
    return {"bytes": 25 * px + 4 * _surface_voxels(case) * _voxel_bytes(case), "flops": 200 * px}


def _track_work(case):
    # the frame and the raycast read once by each of the pyramid's levels; 60 operations a pixel and iteration
    px = case["width"] * case["height"]
    return {"bytes": px * (4 + 24), "flops": 60 * px * (4 + 5 / 4 + 10 / 16)}


def work(case):
    kind = case["kind"]
    parts = []
    if kind == "preprocess":
        out = case["width"] * case["height"] // case["ratio"] ** 2
        parts = [{"bytes": 4 * case["width"] * case["height"] + (4 + 8 + 4 + 4) * out,
                  "flops": 20 * out * (2 * case["radius"] + 1) ** 2}]
    elif kind == "query":
        n = case["points"]
        cells = min(32 * n, 512 * 16_000)   # voxels read: each point's 32, or the field's
        parts = [{"bytes": n * (12 + 4 + 1 + 12 + 1) + cells * (4 if case["storage"] == "f16" else 8), "flops": 120 * n}]
    elif kind == "track":
        parts = [_track_work(case)]
    elif kind == "map":
        parts = [_integrate_work(case), _raycast_work(case)]
    elif kind == "frame":
        px = case["width"] * case["height"]
        parts = [{"bytes": 8 * px, "flops": 20 * 25 * px}, _track_work(case), _integrate_work(case), _raycast_work(case)]
    elif kind == "occupancy":
        # 12-byte voxels; the band behind and before the surface
        v = 16 * _surface_voxels(case)
        px = case["width"] * case["height"]
        parts = [{"bytes": 2 * 12 * v + (4 + 25) * px, "flops": 60 * v + 400 * px}]
    elif kind == "lidar":
        px = case["columns"] * case["beams"]
        view = 160 * 120
        parts = [{"bytes": case["maps"] * (4 * px + 2 * 12 * 8 * px) + 25 * view, "flops": case["maps"] * 400 * px + 400 * view}]
    elif kind == "rays":
        n = case["columns"] * case["beams"] // 2     # about half of the beams return
        steps = 10.0 / 0.2                           # voxels that a ray of 10 m crosses
        parts = [{"bytes": n * (12 + 64) + 2 * 12 * n * steps + 25 * 160 * 120, "flops": 60 * n * steps}]
    elif kind == "render":
        px = case["width"] * case["height"]
        blocks = 16 * _surface_voxels(case)          # voxels of the blocks that get gradients, written
        parts = [{"bytes": (4 + 4 + 4) * px + 4 * _surface_voxels(case) * 8 + 4 * blocks, "flops": 500 * px}]
    return {"bytes": float(sum(p["bytes"] for p in parts)), "flops": float(sum(p["flops"] for p in parts))}
