"""The work whose speed is watched: what a user's program has the library do.

A case is a dict of plain values.  Its "kind" says which call sequence it
stands for:

  query    query_states of n points of a built map (a planner's collision
           checks), points and states in host memory;
  scan     one LiDAR scan integrated as the reference's driver does it:
           update, recenter on the sensor, then the planner's point checks;
  driver   the driver's whole cycle from a sensor-frame cloud and a pose:
           update_pose, recenter, the visualisation cloud of the OCCUPIED
           voxels around the robot (the display's limit of points);
  depth    a depth image and a pose: update_depth, recenter, point checks;
  batch    one scan into each of several robots' maps: Batch.update,
           Batch.recenter, point checks in every map;
  served   several robots' scans and fetches submitted to a Server, waited
           for, and their results read;
  fetch    fetch_batch around many centres of a built map;
  noalloc  cublox_integrate_noalloc on map buffers and points that the
           program holds on the device.

Inputs are made on the GPU from the seed alone: LiDAR scans of a scene of a
ground plane and boxes (the recipe of cublox_b200.synth), a few poses along
a line, used in turn from pass to pass.  Scans reach the library from where
a program has them ("source"): pageable numpy arrays (a ROS message),
page-locked memory, or the device.
"""
import ctypes

import numpy as np
import torch

import cublox_b200 as C

POSES = 4  # scans a program's state holds, used in turn
OCCUPIED = int(C.VoxelState.OCCUPIED)


def listed():
    small = dict(hx=100, hy=100, hz=20, res=0.1)    # 201 x 201 x 41
    middle = dict(hx=200, hy=200, hz=40, res=0.1)   # 401 x 401 x 81
    readme = dict(hx=350, hy=350, hz=75, res=0.1)   # 701 x 701 x 151
    stress = dict(hx=512, hy=512, hz=128, res=0.05)  # 1025 x 1025 x 257
    lidar16 = dict(beams=16, azimuths=1024, elev=15.0, max_range=20.0, boxes=40)
    lidar64 = dict(beams=64, azimuths=1024, elev=22.5, max_range=50.0, boxes=400)
    lidar128 = dict(beams=128, azimuths=2048, elev=22.5, max_range=100.0, boxes=1500)
    return [
        # the smallest call: one planner query of a few hundred points
        dict(name="query_256", kind="query", n=256, **middle),
        # a small robot: 16-beam scan, 20 m map; the scan that steps 1 m away recenters
        dict(name="scan_small", kind="scan", source="pageable", threshold=1.0, step=0.4, checks=4096,
             **small, **lidar16),
        # the reference's published setting: 64-beam scan into a 70 m map, driven slowly
        dict(name="scan_readme", kind="scan", source="pageable", threshold=4.0, step=0.15, checks=16384,
             **readme, **lidar64),
        # the largest map and scan, points already on the device, recentering on every scan
        dict(name="scan_stress", kind="scan", source="device", threshold=0.5, step=0.8, checks=16384,
             **stress, **lidar128),
        # the reference driver's loop, sensor-frame scan to visualisation cloud
        dict(name="driver_cycle", kind="driver", source="pageable", threshold=4.0, step=0.15, radius=25.0,
             shown=4096, **readme, **lidar64),
        # a depth camera on a small robot
        dict(name="depth_640x480", kind="depth", source="pageable", threshold=1.0, step=0.1, checks=4096,
             width=640, height=480, max_range=10.0, boxes=40, **middle),
        # eight robots of the published setting, one scan each per cycle from page-locked memory
        dict(name="batch_8_readme", kind="batch", source="pinned", maps=8, mixed=False, threshold=4.0, step=0.15,
             checks=512, **readme, **lidar64),
        # thirty-two robots with maps of three sizes and scans of uneven length
        dict(name="batch_32_mixed", kind="batch", source="device", maps=32, mixed=True, threshold=4.0, step=0.2,
             checks=512, hx=256, hy=256, hz=64, res=0.1, beams=32, azimuths=4096, elev=15.0, max_range=30.0,
             boxes=200),
        # the served form: four robots, a scan and a planner's fetch of every state near 256 places each
        dict(name="served_4", kind="served", source="pageable", maps=4, threshold=4.0, step=0.15, centres=256,
             radius=0.5, **readme, **lidar64),
        # a planner's fetch: occupied voxels around 256 places
        dict(name="fetch_256_occupied", kind="fetch", centres=256, radius=1.5, filter=OCCUPIED, **readme),
        # every voxel around 1,000 places, samples to the host
        dict(name="fetch_1000_all", kind="fetch", centres=1000, radius=1.0, filter=-1, **small),
        # a real-time loop that owns its buffers on the device
        dict(name="noalloc_readme", kind="noalloc", **readme, **lidar64),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _centres_of(rng, radius, half, lo, hi):
    """Centres of a drawn fetch: no more voxels than the largest listed one looks at."""
    return max(8, min(_log(rng, lo, hi), int(1e6 / (radius / half["res"]) ** 3)))


def draw(rng):
    """One more case of the listed kinds, sizes over the whole range."""
    kind = rng.choice(["query", "scan", "scan", "scan", "driver", "depth", "batch", "batch", "served", "fetch", "noalloc"])
    half = dict(hx=_log(rng, 60, 420), hy=_log(rng, 60, 420), hz=_log(rng, 12, 90), res=rng.choice([0.05, 0.1, 0.1, 0.2]))
    lidar = dict(beams=rng.choice([8, 16, 32, 40, 64, 128]), azimuths=_log(rng, 200, 2000),
                 elev=round(rng.uniform(10.0, 25.0), 2), max_range=round(rng.uniform(8.0, 60.0), 2),
                 boxes=_log(rng, 20, 400))
    if kind == "query":
        return dict(kind=kind, n=_log(rng, 1, 60000), **half)
    if kind == "scan":
        return dict(kind=kind, source=rng.choice(["pageable", "pinned", "device"]),
                    threshold=rng.choice([0.5, 1.0, 4.0]), step=round(rng.uniform(0.1, 1.2), 3),
                    checks=_log(rng, 100, 20000), **half, **lidar)
    if kind == "driver":
        half = dict(half, hx=max(150, half["hx"]), hy=max(150, half["hy"]), hz=max(30, half["hz"]), res=0.1)
        lidar["boxes"] = max(100, lidar["boxes"])
        return dict(kind=kind, source="pageable", threshold=4.0, step=round(rng.uniform(0.1, 0.8), 3),
                    radius=round(rng.uniform(5.0, 25.0), 2), shown=lidar["beams"] * lidar["azimuths"] // 128,
                    **half, **lidar)
    if kind == "depth":
        w = rng.choice([160, 320, 424, 640])
        return dict(kind=kind, source="pageable", threshold=1.0, step=round(rng.uniform(0.05, 0.5), 3),
                    checks=_log(rng, 100, 20000), width=w, height=rng.choice([w * 3 // 4, w * 9 // 16]),
                    max_range=round(rng.uniform(4.0, 12.0), 2), boxes=_log(rng, 20, 100), **half)
    if kind == "batch":
        half["hx"], half["hy"] = min(half["hx"], 256), min(half["hy"], 256)
        lidar["azimuths"] = min(lidar["azimuths"], 1024)
        return dict(kind=kind, source=rng.choice(["pageable", "pinned", "device"]), maps=rng.randint(2, 16),
                    mixed=rng.random() < 0.5, threshold=4.0, step=round(rng.uniform(0.1, 0.8), 3),
                    checks=_log(rng, 64, 4096), **half, **lidar)
    if kind == "served":
        lidar["azimuths"] = min(lidar["azimuths"], 1024)
        radius = round(rng.uniform(0.3, 0.8), 2)
        return dict(kind=kind, source="pageable", maps=rng.randint(2, 4), threshold=4.0,
                    step=round(rng.uniform(0.1, 0.8), 3), centres=min(256, _centres_of(rng, radius, half, 16, 256)),
                    radius=radius, **half, **lidar)
    if kind == "fetch":
        radius = round(2.0 * 0.2 ** rng.random(), 3)
        return dict(kind=kind, centres=_centres_of(rng, radius, half, 8, 1000), radius=radius,
                    filter=rng.choice([-1, 0, 1, 2, 2]), **half)
    lidar["azimuths"] = min(lidar["azimuths"], 1024)
    return dict(kind=kind, **half, **lidar)


# ---- inputs ---------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _scene(g, boxes, extent):
    """Boxes standing on the ground within +-extent, clear of the path (y = 0)."""
    c = _uniform(g, -extent, extent, boxes, 2)
    side = _uniform(g, 0.3, 3.0, boxes, 3)
    near = (c[:, 1].abs() < side[:, 1] / 2 + 1.5)
    c[:, 1] += torch.where(near, torch.where(c[:, 1] < 0, -4.0, 4.0), 0.0)
    lo = torch.cat([c - side[:, :2] / 2, torch.zeros(boxes, 1, device="cuda", dtype=torch.float64)], 1)
    hi = torch.cat([c + side[:, :2] / 2, side[:, 2:]], 1)
    return lo, hi


def _cast(scene, origin, dirs):
    """Distance along each direction to the ground or the first box (inf: none)."""
    lo, hi = scene
    t = torch.where(dirs[:, 2] < 0, -origin[2] / dirs[:, 2], torch.inf)
    step = max(1, (1 << 26) // max(1, lo.shape[0]))
    for a in range(0, dirs.shape[0], step):
        inv = 1.0 / dirs[a:a + step, None, :]
        t0, t1 = (lo[None] - origin) * inv, (hi[None] - origin) * inv
        near = torch.minimum(t0, t1).amax(2)
        far = torch.maximum(t0, t1).amin(2)
        hit = torch.where((near <= far) & (near > 0), near, torch.inf).amin(1)
        t[a:a + step] = torch.minimum(t[a:a + step], hit)
    return t


def _pose(case, k):
    return torch.tensor([case["step"] * k, 0.0, 1.8], device="cuda", dtype=torch.float64)


def _lidar_scan(g, case, scene, origin, yaw, azimuths):
    """(N, 3) float32 world points, azimuth-major; beams without a return end
    at 1.5 x max_range."""
    el = torch.deg2rad(torch.linspace(-case["elev"], case["elev"], case["beams"], device="cuda", dtype=torch.float64))
    az = yaw + 2 * torch.pi * torch.arange(azimuths, device="cuda", dtype=torch.float64) / azimuths
    d = torch.stack([az.cos()[:, None] * el.cos(), az.sin()[:, None] * el.cos(), el.sin().expand(azimuths, -1)], 2)
    d = d.reshape(-1, 3)
    r = _cast(scene, origin, d)
    r = r + 0.02 * torch.randn(r.shape, generator=g, device="cuda", dtype=torch.float64)
    r = torch.where(torch.isfinite(r) & (r <= case["max_range"]), r.clamp(min=1e-3), 1.5 * case["max_range"])
    return (origin + r[:, None] * d).float()


def _extent(case):
    return 1.2 * min(case["max_range"], max(case["hx"], case["hy"]) * case["res"])


def _scans(case, seed, m=0, azimuths=None):
    """POSES scans of robot m: device tensors (N, 3), and the sensor positions."""
    g = _gen(seed * 1009 + m)
    scene = _scene(g, case["boxes"], _extent(case))
    origins = [_pose(case, k) for k in range(POSES)]
    clouds = [_lidar_scan(g, case, scene, o, 0.1 * k, azimuths or case["azimuths"]) for k, o in enumerate(origins)]
    return clouds, [o.float().cpu().numpy() for o in origins]


def _as_source(case, t):
    if case["source"] == "device":
        return t
    h = t.cpu()
    return (h.pin_memory() if case["source"] == "pinned" else h).numpy()


def _checks(g, case, n):
    """Points a planner checks: around the robot, within the window."""
    reach = 0.8 * min(10.0, min(case["hx"], case["hy"]) * case["res"])
    p = torch.cat([_uniform(g, -reach, reach, n, 2), _uniform(g, 0.0, 3.0, n, 1)], 1)
    return p.float().cpu().numpy()


def _configure(case, g, max_range):
    g.setLogOddsParams(*C.yaml_log_odds())
    g.setMaxRaycastRange(max_range)
    return g


def _half(case):
    return (case["hx"], case["hy"], case["hz"])


ORIGIN = (9, -12, 4)  # window origin of a built map, global voxel index


def _stored_map(case, seed):
    """Stored log-odds of a built map in hash order (slots x, y, z): rough
    ground, unknown below it, occupied on it, mostly free above with things
    standing about.  What is where is the same for every seed (so that a
    fetch finds as many samples); how sure the map is of it is not."""
    n = [2 * h + 1 for h in _half(case)]
    fixed = _gen(1)
    ground = (torch.rand(n[0], n[1], 1, generator=fixed, device="cuda") * 0.3 * n[2]).int()
    what = torch.rand(n[0], n[1], n[2], generator=fixed, device="cuda")
    sure = torch.rand(n[0], n[1], n[2], generator=_gen(seed), device="cuda")
    z = torch.arange(n[2], device="cuda").view(1, 1, -1)
    occ = torch.where((z > ground) & (what > 0.1), -0.05 - 1.9 * sure, torch.zeros_like(sure))
    occ = torch.where((z == ground) | (what > 0.97), 1.8 + 1.6 * sure, occ)
    return occ.reshape(-1).cpu().numpy()


def _built_grid(case, seed):
    g = _configure(case, C.OccupancyGrid(_half(case), case["res"], False, 4.0), 50.0)
    g.set_origin_index(ORIGIN)
    g.import_(_stored_map(case, seed))
    return g


def _centres(case, seed):
    """The same places for every seed, asked for in another order."""
    reach = 0.7 * np.minimum(100, np.array(_half(case))) * case["res"]
    u = np.random.default_rng(5).uniform(-1.0, 1.0, (case["centres"], 3))
    u = u[np.random.default_rng(seed).permutation(case["centres"])]
    return (np.array(ORIGIN) * case["res"] + u * reach).astype(np.float32)


class MapView(ctypes.Structure):
    """cublox_map_view."""
    _fields_ = [("occ", ctypes.c_void_p), ("cnt", ctypes.c_void_p), ("hit", ctypes.c_void_p),
                ("half", ctypes.c_int * 3), ("origin", ctypes.c_int * 3), ("resolution", ctypes.c_float),
                ("at_center", ctypes.c_int), ("max_range", ctypes.c_float), ("l_hit", ctypes.c_float),
                ("l_miss", ctypes.c_float), ("l_min", ctypes.c_float), ("l_max", ctypes.c_float)]


def _prepare_batch(case, seed):
    b = C.Batch()
    b.set_option(C.BATCH_OPT_GRAPHS, 1)
    halves = [(case["hx"], case["hy"], case["hz"])]
    if case["mixed"]:
        halves += [(case["hx"] * 3 // 4, case["hy"] * 3 // 4, case["hz"] * 3 // 4),
                   (case["hx"] // 2, case["hy"] // 2, case["hz"] // 2)]
    rng = np.random.default_rng(seed)
    grids, clouds, sensors = [], [], []
    for m in range(case["maps"]):
        grids.append(_configure(case, b.add_grid(halves[m % len(halves)], case["res"], False, case["threshold"]),
                                case["max_range"]))
        az = case["azimuths"]
        if case["mixed"]:
            az = int(rng.integers(max(1, az // 16), az + 1))
        c, s = _scans(case, seed, m, az)
        clouds.append(c)
        sensors.append(s)
    steps = []
    for k in range(POSES):
        off = np.zeros(case["maps"] + 1, np.int64)
        off[1:] = np.cumsum([c[k].shape[0] for c in clouds])
        steps.append((_as_source(case, torch.cat([c[k] for c in clouds])), np.stack([s[k] for s in sensors]), off))
    while b.tuning():  # the batch settles its launch shape on a program's first updates
        b.update(grids, steps[0][0], steps[0][1], offsets=steps[0][2])
    b.synchronize()
    for g in grids:
        g.reset()
    checks = _checks(_gen(seed + 3), case, case["checks"])
    return dict(case=case, k=0, batch=b, grids=grids, steps=steps, checks=checks)


def _prepare_served(case, seed):
    s = C.Server(hbm_budget_bytes=24 << 30)
    lo = C.yaml_log_odds()
    add = lambda half: s.add_map(half, case["res"], False, case["threshold"],  # noqa: E731
                                 max_range=case["max_range"], log_odds=lo)
    maps = [add(_half(case)) for _ in range(case["maps"])]
    scans = [_scans(case, seed, m) for m in range(case["maps"])]
    scans = [([_as_source(case, c) for c in clouds], sensors) for clouds, sensors in scans]
    centres = [np.ascontiguousarray(_checks(_gen(11 * m), case, case["centres"])) for m in range(case["maps"])]
    # the server's batch settles its launch shape on its first ticks: those of a robot of the same kind
    other = add(_half(case))
    for _ in range(36):
        r = s.submit_scan(other, scans[0][0][0], scans[0][1][0])
        s.wait(r)
        s.release(r)
    s.drain()
    return dict(case=case, k=0, server=s, maps=maps, scans=scans, centres=centres)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "query":
        return dict(case=case, grid=_built_grid(case, seed), points=_checks(_gen(seed + 3), case, case["n"]))
    if kind == "fetch":
        return dict(case=case, grid=_built_grid(case, seed), centres=_centres(case, seed))
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "served":
        return _prepare_served(case, seed)
    if kind == "noalloc":
        return _prepare_noalloc(case, seed)
    g = _configure(case, C.OccupancyGrid(_half(case), case["res"], False, case["threshold"]), case["max_range"])
    state = dict(case=case, k=0, grid=g)
    if kind == "depth":
        images, state["K"], state["R"], state["sensors"] = _depth_images(case, seed)
        state["images"] = [i.cpu().numpy() for i in images]
    else:
        clouds, state["sensors"] = _scans(case, seed)
        if kind == "driver":
            R = [_yaw(0.1 * k) for k in range(POSES)]
            state["R"] = R
            clouds = [((c.double() - _pose(case, k)) @ torch.from_numpy(R[k]).double().cuda()).float().contiguous()
                      for k, c in enumerate(clouds)]
        state["clouds"] = [_as_source(case, c) for c in clouds]
    if "checks" in case:
        state["checks"] = _checks(_gen(seed + 3), case, case["checks"])
    return state


def _yaw(a):
    return np.array([[np.cos(a), -np.sin(a), 0], [np.sin(a), np.cos(a), 0], [0, 0, 1]], np.float32)


def _depth_images(case, seed):
    """16-bit millimetre images of a camera looking along +x."""
    g = _gen(seed)
    scene = _scene(g, case["boxes"], _extent(case))
    w, h = case["width"], case["height"]
    f = 525.0 * w / 640.0
    u = (torch.arange(w, device="cuda", dtype=torch.float64) - w / 2) / f
    v = (torch.arange(h, device="cuda", dtype=torch.float64) - h / 2) / f
    R = torch.tensor([[0, 0, 1], [-1, 0, 0], [0, -1, 0]], device="cuda", dtype=torch.float64)
    d = torch.stack([u.expand(h, w), v[:, None].expand(h, w), torch.ones(h, w, device="cuda", dtype=torch.float64)], 2)
    world = d.reshape(-1, 3) @ R.T + 1e-9
    images, sensors = [], []
    for k in range(POSES):
        o = _pose(case, k)
        z = _cast(scene, o, world) + 0.005 * torch.randn(w * h, generator=g, device="cuda", dtype=torch.float64)
        z = torch.where(torch.isfinite(z) & (z < 60.0), z * 1000.0, torch.zeros_like(z))
        images.append(z.round().clamp(0, 65535).to(torch.int32).to(torch.uint16).view(h, w))
        sensors.append(o.float().cpu().numpy())
    return images, np.array([f, f, w / 2, h / 2], np.float32), R.float().cpu().numpy(), sensors


def _prepare_noalloc(case, seed):
    fn = C.lib().cublox_integrate_noalloc
    fn.argtypes = [ctypes.POINTER(MapView), ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.c_float),
                   ctypes.c_void_p]
    fn.restype = ctypes.c_int
    clouds, sensors = _scans(dict(case, step=0.15), seed)
    v = 1
    for h in _half(case):
        v *= 2 * h + 1
    occ = torch.zeros(v, dtype=torch.float32, device="cuda")
    cnt = torch.zeros(v, dtype=torch.int32, device="cuda")
    hit = torch.zeros(v, dtype=torch.int32, device="cuda")
    lo = C.yaml_log_odds()
    view = MapView(occ.data_ptr(), cnt.data_ptr(), hit.data_ptr(), (ctypes.c_int * 3)(*_half(case)),
                   (ctypes.c_int * 3)(0, 0, int(1.8 / case["res"])), case["res"], 0, case["max_range"], *lo[:4])
    return dict(case=case, k=0, fn=fn, view=view, keep=(cnt, hit), occ=occ,
                clouds=[c.T.contiguous() for c in clouds],
                sensors=[(ctypes.c_float * 3)(*s.tolist()) for s in sensors])


# ---- one pass -------------------------------------------------------------

def run(state):
    kind = state["case"]["kind"]
    if kind == "query":
        return state["grid"].query_states(state["points"])
    if kind == "fetch":
        c = state["case"]
        return state["grid"].fetch_batch(state["centres"], c["radius"], None if c["filter"] < 0 else c["filter"])
    k = state["k"] % POSES
    state["k"] += 1
    if kind == "scan":
        g, sensor = state["grid"], state["sensors"][k]
        g.update(state["clouds"][k], sensor)
        return g.recenter(sensor), g.query_states(state["checks"])
    if kind == "driver":
        g, t, c = state["grid"], state["sensors"][k], state["case"]
        g.update_pose(state["clouds"][k], state["R"][k], t)
        return g.recenter(t), g.fetch_viz(t, c["radius"], OCCUPIED, max_points=c["shown"])
    if kind == "depth":
        g, t = state["grid"], state["sensors"][k]
        g.update_depth(state["images"][k], state["K"], state["R"], t)
        return g.recenter(t), g.query_states(state["checks"])
    if kind == "batch":
        xyz, sensors, off = state["steps"][k]
        state["batch"].update(state["grids"], xyz, sensors, offsets=off)
        actions = state["batch"].recenter(state["grids"], sensors)
        return actions, [g.query_states(state["checks"]) for g in state["grids"]]
    if kind == "served":
        return _run_served(state, k)
    cloud = state["clouds"][k]
    rc = state["fn"](ctypes.byref(state["view"]), cloud.data_ptr(), cloud.shape[1], state["sensors"][k],
                     torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError("cublox_integrate_noalloc returned %d" % rc)
    return state["occ"]


def _run_served(state, k):
    s, c = state["server"], state["case"]
    scans = [s.submit_scan(m, clouds[k], sensors[k]) for m, (clouds, sensors) in zip(state["maps"], state["scans"])]
    fetches = [s.submit_fetch(m, centres, c["radius"]) for m, centres in zip(state["maps"], state["centres"])]
    out = [s.wait(r) for r in scans]
    for r in fetches:
        s.wait(r)
        out.append(s.fetch_result(r, c["centres"]))
    for r in scans + fetches:
        s.release(r)
    return out


# ---- what a pass cannot do without ------------------------------------------

def _touched(case, rays):
    """Distinct voxels that a scan of `rays` rays visits, about: a ray walks 0.66
    of the way to the nearer of its range and the window's side, 1.3 voxels a
    cell side, and 0.4 of what the rays of a scan visit is new."""
    reach = min(case["max_range"], min(case["hx"], case["hy"]) * case["res"]) / case["res"]
    cells = (2 * case["hx"] + 1) * (2 * case["hy"] + 1) * (2 * case["hz"] + 1)
    return min(0.4 * rays * 0.66 * 1.3 * reach, cells)


def _sphere(case):
    return 4.19 * (case["radius"] / case["res"]) ** 3


def work(case):
    """Points in, touched voxels' stored values in and out, results out."""
    kind = case["kind"]
    if kind == "query":
        return {"bytes": 17 * case["n"], "flops": 0}
    if kind == "fetch":
        kept = {-1: 1.0, 0: 0.35, 1: 0.55, 2: 0.1}[case["filter"]] * _sphere(case) * case["centres"]
        return {"bytes": 12 * case["centres"] + 4 * _sphere(case) * case["centres"] + 13 * kept, "flops": 0}
    if kind == "depth":
        n = case["width"] * case["height"]
        return {"bytes": 2 * n + 8 * _touched(case, n) + 17 * case["checks"], "flops": 0}
    n = case["beams"] * case["azimuths"]
    one = 12 * n + 8 * _touched(case, n)
    if kind == "driver":
        zs = min(2 * case["hz"] + 1, 2 * case["radius"] / case["res"])
        one += 4 * 3.14 * (case["radius"] / case["res"]) ** 2 * zs
    if kind == "scan":
        one += 17 * case["checks"]
    if kind == "batch":
        one = case["maps"] * (one * (0.3 if case["mixed"] else 1.0) + 17 * case["checks"])
    if kind == "served":
        one = case["maps"] * (one + 12 * case["centres"] + 17 * _sphere(case) * case["centres"])
    return {"bytes": one, "flops": 0}


# ---- the same in 64 bits ----------------------------------------------------

def exact(case, seed):
    """What a first pass returns, in 64 bits, where it is a computed number:
    sample positions of a fetch, stored log-odds of noalloc (the states are
    whole values, and the visualisation cloud's colours are packed bits)."""
    if case["kind"] == "fetch":
        return None, _exact_positions(case, seed), None
    if case["kind"] == "noalloc":
        return _exact_log_odds(case, seed)
    return None


def _exact_positions(case, seed):
    """Centres of the voxels whose single-precision distance is within the
    radius, of the wanted state, in the order of x, y, z."""
    f = np.float32
    res, inv = f(case["res"]), f(1.0) / f(case["res"])
    half, origin = np.array(_half(case)), np.array(ORIGIN)
    n = 2 * half + 1
    occ = _stored_map(case, seed).reshape(n)
    lo = C.yaml_log_odds()
    state = np.where(occ >= f(lo[5]), 2, np.where(occ < f(lo[4]), 1, 0))
    rows = []
    for c in _centres(case, seed):
        cg = np.floor(c * inv).astype(int)
        margin = (half - np.abs(cg - origin))[:2]
        if margin.min() < 0:
            continue
        r = min(f(case["radius"]), f(margin.min()) * res)
        if r <= 0:
            continue
        g0 = np.maximum(np.floor((c - r) * inv).astype(int), origin - half)
        g1 = np.minimum(np.floor((c + r) * inv).astype(int), origin + half)
        if (g1 < g0).any():
            continue
        g = np.stack(np.meshgrid(*[np.arange(a, b + 1) for a, b in zip(g0, g1)], indexing="ij"), -1).reshape(-1, 3)
        d = ((g.astype(f) + f(0.5)) * res - c).astype(np.float64)
        s = f(d[:, 1] * d[:, 1]).astype(np.float64)
        s = f(d[:, 0] * d[:, 0] + s).astype(np.float64)
        g = g[f(d[:, 2] * d[:, 2] + s) <= r * r]
        slot = (g + half) % n
        if case["filter"] >= 0:
            g = g[state[slot[:, 0], slot[:, 1], slot[:, 2]] == case["filter"]]
        rows.append((g + 0.5) * np.float64(res))
    return np.concatenate(rows) if rows else np.empty((0, 3))


def _exact_log_odds(case, seed):
    """The reference's single-precision traversal (it decides which voxels a
    ray visits), and the visits' log-odds summed in 64 bits."""
    f = np.float32
    clouds, sensors = _scans(dict(case, step=0.15), seed)
    p, o = clouds[0].cpu().numpy(), sensors[0].astype(f)
    half = np.array(_half(case))
    n = 2 * half + 1
    origin = np.array([0, 0, int(1.8 / case["res"])])
    res, inv, most = f(case["res"]), f(1.0) / f(case["res"]), f(case["max_range"])
    d = (p - o).astype(f)
    q = d.astype(np.float64)
    s = f(q[:, 1] * q[:, 1]).astype(np.float64)
    s = f(q[:, 0] * q[:, 0] + s).astype(np.float64)
    length = np.sqrt(f(q[:, 2] * q[:, 2] + s))
    clipped = length > most
    k = np.where(clipped, most / length, f(1.0))[:, None]
    p = np.where(clipped[:, None], o + d * k, p)
    d = np.where(clipped[:, None], d * k, d)
    length = np.where(clipped, most, length)
    u = d * (f(1.0) / length)[:, None]
    ids = np.tile(np.floor(o * inv).astype(np.int64), (len(p), 1))
    ends = np.floor(p * inv).astype(np.int64)
    step = (u > 0).astype(np.int64) - (u < 0)
    with np.errstate(divide="ignore", invalid="ignore"):
        tD = np.where(step == 0, f(np.inf), np.abs(res / u))
        tM = np.where(step == 0, f(np.inf), ((ids + (step > 0)).astype(f) * res - o) / u)
    limit = np.abs(ends - ids).sum(1) + 4
    op = np.zeros(int(np.prod(n)), np.int64)
    hit = np.zeros_like(op)

    def cells(g):
        slot = (g + half) % n
        return (slot[:, 0] * n[1] + slot[:, 1]) * n[2] + slot[:, 2]

    inside = (np.abs(ends - origin) <= half).all(1)
    np.add.at(op, cells(ends[inside]), 1)
    np.add.at(hit, cells(ends[inside & ~clipped]), 1)
    live = np.arange(len(p))
    for i in range(int(limit.max())):
        live = live[(i < limit[live]) & (ids[live] != ends[live]).any(1)]
        rel = ids[live] - origin
        gone = ((np.abs(rel) > half) & (rel * step[live] >= 0)).any(1)
        live, rel = live[~gone], rel[~gone]
        if not len(live):
            break
        np.add.at(op, cells(ids[live][(np.abs(rel) <= half).all(1)]), 1)
        t = tM[live]
        axis = np.where(t[:, 0] < t[:, 1], np.where(t[:, 0] < t[:, 2], 0, 2), np.where(t[:, 1] < t[:, 2], 1, 2))
        ids[live, axis] += step[live, axis]
        tM[live, axis] += tD[live, axis]
    lo = [np.float64(f(v)) for v in C.yaml_log_odds()]
    out = np.clip(lo[1] * np.maximum(op - hit, 0) + lo[0] * hit, lo[2], lo[3])
    return np.where(op > 0, out, 0.0)
