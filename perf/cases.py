"""The measured cases: what programs built on this package have it do, pass by pass.

Kinds of case, each one pass of a user's loop through the Python front end:

* ``scan``   one robot's mapping loop: insert_point_cloud of the next scan of a
             moving sensor, then the planner's is_occupied / is_free lookups.
* ``ros``    the ROS node's cloud callback: a sensor-frame cloud in host memory
             with dropped returns (NaN) and no range limit, then the occupied
             voxels of a height band as a 2-D obstacle layer on the GPU.
* ``tick``   many robots, one map each: Batch.insert of one scan per map, then
             lookups on every eighth map.
* ``serve``  clients of a Server: each sends one scan and one lookup request
             and waits for its answers.
* ``lookup`` isOccupied / isUnknown / isFree of a batch of coordinates.
* ``grid``   a VoxelGrid<T> that is updated in place and read back.
* ``cloud``  a VoxelGrid<T> rebuilt from a host point cloud, with cells erased.
* ``save``   a map saved (serialize) and loaded into a grid (deserialize).

Inputs are synthetic: a spinning LiDAR in a scene of boxes, a pinhole depth
camera in a furnished room, and points sampled on a room's surfaces in no order
(a registered cloud); all made on the GPU from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import bonxai_gb300 as bx

DEV = "cuda"
N_WARM = 2     # scans a map holds before the first pass
N_POSES = 4    # scans that the passes take in turn

_DTYPES = {"float32": (np.float32, torch.float32), "float64": (np.float64, torch.float64),
           "int32": (np.int32, torch.int32), "uint8": (np.uint8, torch.uint8)}


def listed():
    return [
        # a 16-beam LiDAR sector or a strongly downsampled cloud: the smallest
        # call that robots make, latency and launches count
        dict(name="scan_2k", kind="scan", scene="lidar", n=2048, res=0.1, max_range=20.0,
             dtype="float32", lookups=1000),
        # one revolution of a 64-beam LiDAR, the size the reference is quoted on
        dict(name="scan_lidar_131k", kind="scan", scene="lidar", n=131072, res=0.1,
             max_range=30.0, dtype="float32", lookups=65536),
        # a 640x480 depth frame at 2 cm
        dict(name="scan_depth_307k", kind="scan", scene="depth", n=307200, res=0.02,
             max_range=5.0, dtype="float32", lookups=65536),
        # a registered cloud in double precision: odd size, neighbours in memory
        # are not neighbours in space
        dict(name="scan_room_f64", kind="scan", scene="room", n=60013, res=0.05,
             max_range=10.0, dtype="float64", lookups=4099),
        # the ROS node with its defaults: host cloud, NaN returns, no range limit
        dict(name="ros_cycle_29k", kind="ros", n=28813, res=0.05, min_z=0.2, max_z=2.0),
        # a small fleet of small clouds
        dict(name="tick_8", kind="tick", maps=8, n_lo=2000, n_hi=20000, max_range=10.0,
             lookups=1000),
        # the 64-map uneven workload of the benchmark: the largest
        dict(name="tick_64", kind="tick", maps=64, n_lo=10000, n_hi=500000, max_range=10.0,
             lookups=1000),
        # a handful of served clients
        dict(name="serve_6", kind="serve", clients=6, n=20011, res=0.1, max_range=10.0,
             lookups=5000),
        # a planner's or a mesher's bulk lookup
        dict(name="lookup_1m", kind="lookup", n=1 << 20, res=0.02, mode="occupied"),
        # the reference's create/update/iterate cloud size, updated in place
        dict(name="grid_f32_300k", kind="grid", n=300000, res=0.02, dtype="float32",
             inner_bits=2, leaf_bits=3, lookups=30011),
        # a byte grid (semantic labels) with other node sizes, rebuilt per cloud
        dict(name="cloud_u8_50k", kind="cloud", n=50021, res=0.03, dtype="uint8",
             inner_bits=3, leaf_bits=2, lookups=10007),
        # a map written to and read from the reference's file format
        dict(name="save_load", kind="save", n=40009, res=0.1, max_range=20.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan", "scan", "tick", "tick", "ros", "serve", "lookup",
                       "grid", "cloud", "save"])
    if kind == "scan":
        scene = rng.choice(["lidar", "depth", "room"])
        res = rng.choice([0.02, 0.05, 0.1])
        reach = {0.02: 8.0, 0.05: 20.0, 0.1: 40.0}[res]
        return dict(kind=kind, scene=scene, n=_log(rng, 500, 300000), res=res,
                    max_range=round(rng.uniform(reach / 4, reach), 2),
                    dtype=rng.choice(["float32", "float32", "float64"]),
                    lookups=_log(rng, 100, 100000))
    if kind == "tick":
        hi = _log(rng, 4000, 500000)
        return dict(kind=kind, maps=_log(rng, 2, 64), n_lo=max(1000, hi // 30), n_hi=hi,
                    max_range=round(rng.uniform(4.0, 10.0), 2), lookups=_log(rng, 100, 10000))
    if kind == "ros":
        return dict(kind=kind, n=_log(rng, 2000, 100000), res=rng.choice([0.05, 0.1, 0.2]),
                    min_z=round(rng.uniform(0.0, 0.5), 2), max_z=round(rng.uniform(1.0, 4.0), 2))
    if kind == "serve":
        return dict(kind=kind, clients=rng.randint(2, 8), n=_log(rng, 2000, 50000),
                    res=rng.choice([0.05, 0.1]), max_range=round(rng.uniform(4.0, 15.0), 2),
                    lookups=_log(rng, 100, 50000))
    if kind == "lookup":
        return dict(kind=kind, n=_log(rng, 100, 1 << 20), res=rng.choice([0.02, 0.05]),
                    mode=rng.choice(["occupied", "unknown", "free"]))
    if kind == "save":
        return dict(kind=kind, n=_log(rng, 2000, 60000), res=rng.choice([0.1, 0.2]),
                    max_range=round(rng.uniform(5.0, 20.0), 2))
    inner_bits, leaf_bits = rng.choice([(2, 3), (2, 3), (1, 2), (3, 2), (2, 4), (3, 3)])
    return dict(kind=kind, n=_log(rng, 300, 400000 if kind == "grid" else 150000),
                res=round(rng.uniform(0.01, 0.1), 3),
                dtype=rng.choice(["float32", "float64", "int32", "uint8"]),
                inner_bits=inner_bits, leaf_bits=leaf_bits, lookups=_log(rng, 100, 50000))


# ----------------------------------------------------------------------------
# synthetic sensors (torch on the GPU)
# ----------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, device=DEV, generator=g) * (hi - lo) + lo


def _first_box(o, d, lo, hi):
    """Distance along each direction d [n,3] from o to the first box, inf if none."""
    best = torch.full((d.shape[0],), math.inf, device=DEV)
    step = max(1, (1 << 25) // max(1, lo.shape[0]))
    for a in range(0, d.shape[0], step):
        inv = 1.0 / torch.where(d[a:a + step] == 0, torch.full_like(d[:1], 1e-20), d[a:a + step])
        tmin = tmax = None
        for ax in range(3):
            t0 = inv[:, ax:ax + 1] * (lo[None, :, ax] - o[ax])
            t1 = inv[:, ax:ax + 1] * (hi[None, :, ax] - o[ax])
            near, far = torch.minimum(t0, t1), torch.maximum(t0, t1)
            tmin = near if tmin is None else torch.maximum(tmin, near)
            tmax = far if tmax is None else torch.minimum(tmax, far)
        hit = (tmax >= tmin) & (tmin > 1e-6)
        best[a:a + step] = torch.where(hit, tmin, torch.full_like(tmin, math.inf)).amin(1)
    return best


def _lidar(g, n, n_scans, n_boxes=120):
    """[(directions [n,3], distances [n] (inf: no return), origin [3])] of a LiDAR
    moving 0.4 m per scan through a 40 x 40 m scene of boxes on a floor."""
    size = _uniform(g, 0.5, 4.0, n_boxes, 3)
    c = _uniform(g, -20.0, 20.0, n_boxes, 2)
    side = torch.where(c[:, 1] < 0, -1.0, 1.0)  # the corridor |y| < 1.5 stays clear
    c[:, 1] = side * (1.5 + size[:, 1] / 2 + c[:, 1].abs() * 0.85)
    lo = torch.stack([c[:, 0] - size[:, 0] / 2, c[:, 1] - size[:, 1] / 2,
                      torch.zeros(n_boxes, device=DEV)], 1)
    hi = torch.stack([c[:, 0] + size[:, 0] / 2, c[:, 1] + size[:, 1] / 2, size[:, 2]], 1)
    beams = 64 if n >= 16384 else 16
    cols = -(-n // beams)
    el = torch.linspace(math.radians(-25.0), math.radians(15.0), beams, device=DEV)
    az = torch.arange(cols, device=DEV) * (2 * math.pi / cols)
    e, a = torch.meshgrid(el, az, indexing="ij")
    d = torch.stack([e.cos() * a.cos(), e.cos() * a.sin(), e.sin()], -1).reshape(-1, 3)[:n]
    x0 = float(torch.rand((), generator=g, device=DEV)) * 4 - 6
    out = []
    for k in range(n_scans):
        o = torch.tensor([x0 + 0.4 * k, 0.07 * k, 1.7], device=DEV)
        t = _first_box(o, d, lo, hi)
        floor = torch.where(d[:, 2] < 0, -o[2] / d[:, 2].clamp(max=-1e-9),
                            torch.full_like(t, math.inf))
        t = torch.minimum(t, floor)
        out.append((d, t + 0.01 * torch.randn(n, device=DEV, generator=g), o))
    return out


def _depth(g, n, n_scans):
    """[(points, origin)]: frames of a pinhole camera walking in an 8 x 6 x 3 m
    room with 50 boxes, pixels in row order."""
    size = _uniform(g, 0.2, 1.2, 50, 3)
    cx, cy = _uniform(g, 1.4, 3.4, 50), _uniform(g, -2.4, 2.4, 50)
    cx = cx * torch.where(torch.arange(50, device=DEV) % 2 == 0, 1.0, -1.0)
    lo = torch.stack([cx - size[:, 0] / 2, cy - size[:, 1] / 2, torch.zeros(50, device=DEV)], 1)
    hi = torch.stack([cx + size[:, 0] / 2, cy + size[:, 1] / 2, size[:, 2]], 1)
    w = max(1, round(math.sqrt(n * 4 / 3)))
    idx = torch.arange(n, device=DEV)
    u, v = (idx % w).float() / w - 0.5, (idx // w).float() / max(1, -(-n // w)) - 0.5
    cam = torch.stack([torch.ones_like(u), -u * 640 / 525, -v * 480 / 525], 1)
    wall_lo = torch.tensor([-4.0, -3.0, 0.0], device=DEV)
    wall_hi = torch.tensor([4.0, 3.0, 3.0], device=DEV)
    yaw0 = float(torch.rand((), generator=g, device=DEV)) * 6.28
    out = []
    for k in range(n_scans):
        yaw = yaw0 + 0.03 * k
        r = torch.tensor([[math.cos(yaw), -math.sin(yaw), 0], [math.sin(yaw), math.cos(yaw), 0],
                          [0, 0, 1]], device=DEV)
        d = cam @ r.T
        o = torch.tensor([0.04 * k, 0.03 * k, 1.4], device=DEV)
        safe = torch.where(d == 0, torch.full_like(d, 1e-20), d)
        t = torch.maximum((wall_lo - o) / safe, (wall_hi - o) / safe).amin(1)
        t = torch.minimum(t, _first_box(o, d, lo, hi))
        t = t * (1 + 0.002 * torch.randn(n, device=DEV, generator=g))
        out.append((o + t[:, None] * d, o))
    return out


def _room_surface(g, n):
    """n points on the faces of a 6 x 4 x 3 m room and on 20 spheres, in no order."""
    half = torch.tensor([3.0, 2.0, 1.5], device=DEV)
    p = _uniform(g, -1.0, 1.0, n, 3) * half
    face = torch.randint(0, 26, (n,), device=DEV, generator=g)  # 20 of 26: a face
    for ax, (a, b) in enumerate(((0, 6), (6, 14), (14, 20))):   # shares as their areas
        on = (face >= a) & (face < b)
        p[:, ax] = torch.where(on, torch.sign(p[:, ax]) * half[ax], p[:, ax])
    centre = _uniform(g, -1.0, 1.0, 20, 3) * (half - 0.5)
    radius = _uniform(g, 0.1, 0.5, 20)
    s = torch.randint(0, 20, (n,), device=DEV, generator=g)
    d = torch.randn(n, 3, device=DEV, generator=g)
    ball = centre[s] + radius[s, None] * d / d.norm(dim=1, keepdim=True)
    p = torch.where((face >= 20)[:, None], ball, p)
    return p + 0.005 * torch.randn(n, 3, device=DEV, generator=g)


def _scans(g, scene, n, n_scans, max_range, n_boxes=120):
    """[(world points [n,3] float32, origin [3] numpy float32)]"""
    if scene == "lidar":
        out = []
        for d, t, o in _lidar(g, n, n_scans, n_boxes):
            t = torch.where(torch.isfinite(t), t, torch.full_like(t, 2 * max_range))
            out.append((o + t[:, None] * d, o))
    elif scene == "depth":
        out = _depth(g, n, n_scans)
    else:
        out = [(_room_surface(g, n), torch.tensor([0.03 * k, 0.02 * k, 0.01 * k], device=DEV))
               for k in range(n_scans)]
    return [(p.contiguous(), o.cpu().numpy().astype(np.float32)) for p, o in out]


def _around(g, points, origin, res, n):
    """n int32 cells to look up: half on the scan's surfaces, half around the sensor."""
    k = n // 2
    pick = torch.randint(0, points.shape[0], (k,), device=DEV, generator=g)
    o = torch.as_tensor(np.asarray(origin, np.float32), device=DEV)
    reach = float((points.float() - o).abs().median()) * 1.5 + 4 * res
    box = o + _uniform(g, -1.0, 1.0, n - k, 3) * reach
    xyz = torch.cat([points[pick].float(), box])
    return torch.floor(xyz / res).to(torch.int32).contiguous()


# ----------------------------------------------------------------------------
# states
# ----------------------------------------------------------------------------
class _State:
    def __init__(self, case):
        self.case = case
        self.k = 0  # passes so far

    def turn(self, items):
        item = items[self.k % len(items)]
        self.k += 1
        return item


def prepare(case, seed):
    s = _State(case)
    globals()["_prepare_" + case["kind"]](s, case, _gen(seed))
    torch.cuda.synchronize()
    return s


def _prepare_scan(s, c, g):
    scans = _scans(g, c["scene"], c["n"], N_WARM + N_POSES, c["max_range"])
    if c["dtype"] == "float64":
        scans = [(p.double(), o.astype(np.float64)) for p, o in scans]
    torch.cuda.synchronize()
    s.map = bx.ProbabilisticMap(c["res"])
    for p, o in scans[:N_WARM]:
        s.map.insert_point_cloud(p, o, c["max_range"])
    s.scans = [(p, o, _around(g, p, o, c["res"], c["lookups"])) for p, o in scans[N_WARM:]]
    s.occupied = torch.zeros(c["lookups"], dtype=torch.uint8, device=DEV)
    s.free = torch.zeros(c["lookups"], dtype=torch.uint8, device=DEV)


def _run_scan(s, c):
    points, origin, cells = s.turn(s.scans)
    updates = s.map.insert_point_cloud(points, origin, c["max_range"])
    s.map.is_occupied(cells, s.occupied)
    s.map.is_free(cells, s.free)
    return {"updates": updates, "occupied": s.occupied, "free": s.free}


def _prepare_ros(s, c, g):
    s.clouds = []
    for k, (d, t, o) in enumerate(_lidar(g, c["n"], N_WARM + N_POSES)):
        # a sensor that sees 100 m and drops one return in a hundred
        lost = ~(t < 100.0) | (torch.rand(c["n"], device=DEV, generator=g) < 0.01)
        p = torch.where(lost[:, None], torch.full_like(d, math.nan), d * t[:, None])
        yaw = 0.02 * k  # the cloud in the frame of a sensor turned by yaw
        r = torch.tensor([[math.cos(yaw), -math.sin(yaw), 0], [math.sin(yaw), math.cos(yaw), 0],
                          [0, 0, 1]], device=DEV)
        pose = np.eye(4, dtype=np.float32)
        pose[:3, :3] = r.cpu().numpy()
        pose[:3, 3] = o.cpu().numpy()
        s.clouds.append(((p @ r).cpu().numpy(), pose))
    # the node's GPU work and the layer's share one stream
    s.stream = torch.cuda.Stream()
    s.map = bx.ProbabilisticMap(c["res"], bx.Config(stream=s.stream.cuda_stream))
    for p, pose in s.clouds[:N_WARM]:
        s.map.insert_sensor_cloud(p, pose, -1.0)
    s.clouds = s.clouds[N_WARM:]
    s.occupied = torch.zeros(1 << 19, 3, device=DEV)
    s.side = int(80.0 / c["res"])
    s.layer = torch.zeros(s.side * s.side, dtype=torch.uint8, device=DEV)


def _run_ros(s, c):
    points, pose = s.turn(s.clouds)
    updates = s.map.insert_sensor_cloud(points, pose, -1.0)
    n = s.map.export_occupied(c["min_z"], c["max_z"], out=s.occupied)
    with torch.cuda.stream(s.stream):
        s.layer.zero_()
        cell = torch.floor(s.occupied[:n, :2] / c["res"] + 0.5).long() + s.side // 2
        cell.clamp_(0, s.side - 1)
        s.layer[cell[:, 1] * s.side + cell[:, 0]] = 1
    return {"updates": updates, "voxels": n, "layer": s.layer}


def _prepare_tick(s, c, g):
    rng = np.random.default_rng(int(torch.randint(1 << 30, (), generator=g, device=DEV)))
    m = c["maps"]
    # the sizes are the same ones for every seed, spread over the range
    at = (np.arange(m) * 0.6180339887 % 1.0) if m > 1 else np.array([0.5])
    sizes = np.exp(math.log(c["n_lo"]) + at * (math.log(c["n_hi"]) - math.log(c["n_lo"])))
    sizes = np.maximum(1, sizes + rng.integers(-30, 31, m)).astype(np.int64)
    s.maps, scans, s.res = [], [], []
    for i in range(m):
        s.res.append([0.02, 0.05, 0.1][i % 3])
        s.maps.append(bx.ProbabilisticMap(s.res[-1]))
        scans.append(_scans(g, "room" if i % 2 == 0 else "lidar", int(sizes[i]), 2,
                            c["max_range"], 40))
    s.offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    s.ticks = []
    for k in range(2):
        s.ticks.append((torch.cat([x[k][0] for x in scans]),
                        np.stack([x[k][1] for x in scans])))
    s.asked = [(s.maps[i], _around(g, scans[i][1][0], scans[i][1][1], s.res[i], c["lookups"]),
                torch.zeros(c["lookups"], dtype=torch.uint8, device=DEV))
               for i in range(0, m, 8)]
    s.ranges = np.full(m, c["max_range"])
    torch.cuda.synchronize()
    s.batch = bx.Batch()
    s.batch.insert(s.maps, s.ticks[0][0], s.offsets, s.ticks[0][1], s.ranges)
    s.k = 1  # the next tick is the maps' second


def _run_tick(s, c):
    points, origins = s.turn(s.ticks)
    updates = s.batch.insert(s.maps, points, s.offsets, origins, s.ranges)
    for m, cells, out in s.asked:
        m.is_free(cells, out)
    return {"updates": updates.astype(np.int64), "free": [out for _, _, out in s.asked]}


def _prepare_serve(s, c, g):
    s.server = bx.Server([c["res"]] * c["clients"])
    s.rounds = []
    per_client = [_scans(g, "lidar" if i % 2 else "room", c["n"] + 101 * i, 3, c["max_range"], 60)
                  for i in range(c["clients"])]
    for k in range(3):
        s.rounds.append([(p[k][0].cpu().numpy(), p[k][1],
                          _around(g, p[k][0], p[k][1], c["res"], c["lookups"]).cpu().numpy())
                         for p in per_client])
    _serve(s, c)


def _serve(s, c):
    tickets = []
    for i, (points, origin, cells) in enumerate(s.turn(s.rounds)):
        tickets.append((s.server.insert(i, points, origin, c["max_range"]),
                        s.server.query(i, cells)))
    updates, answers = [], []
    for insert, query in tickets:
        updates.append(s.server.wait_insert(insert)["ray_cells"])
        answers.append(s.server.wait_query(query, c["lookups"])[1])
    return {"updates": updates, "occupied": answers}


_run_serve = _serve


def _prepare_lookup(s, c, g):
    scans = _scans(g, "depth", 307200, 3, 5.0)
    torch.cuda.synchronize()
    s.map = bx.ProbabilisticMap(c["res"])
    for p, o in scans:
        s.map.insert_point_cloud(p, o, 5.0)
    half = torch.tensor([4.0, 3.0, 1.5], device=DEV) / c["res"]
    s.cells = []
    for _ in range(3):
        xyz = _uniform(g, -1.0, 1.0, c["n"], 3) * half
        xyz[:, 2] += half[2]
        s.cells.append(torch.floor(xyz).to(torch.int32).contiguous())
    s.ask = getattr(s.map, "is_" + c["mode"])
    s.out = torch.zeros(c["n"], dtype=torch.uint8, device=DEV)


def _run_lookup(s, c):
    return s.ask(s.turn(s.cells), s.out)


def _values(g, n, dtype):
    t = _DTYPES[dtype][1]
    if t.is_floating_point:
        return torch.randn(n, device=DEV, generator=g, dtype=t)
    return torch.randint(0, 256 if dtype == "uint8" else 1 << 30, (n,), device=DEV,
                         generator=g).to(t)


def _grid_inputs(c, g):
    """[(coords [n,3], values [n], cells to look up)] of the passes."""
    out = []
    for _ in range(N_POSES):
        xyz = torch.floor(_room_surface(g, c["n"]).double() / c["res"]).to(torch.int32)
        pick = torch.randint(0, c["n"], (c["lookups"],), device=DEV, generator=g)
        out.append((xyz.contiguous(), _values(g, c["n"], c["dtype"]), xyz[pick].contiguous()))
    return out


def _prepare_grid(s, c, g):
    s.inputs = _grid_inputs(c, g)
    torch.cuda.synchronize()
    s.grid = bx.VoxelGrid(c["res"], c["inner_bits"], c["leaf_bits"], _DTYPES[c["dtype"]][0])
    # arrays that live on the GPU go through the C ABI, as from C++
    s.lib = bx.load_library()
    s.found = torch.zeros(c["lookups"], dtype=_DTYPES[c["dtype"]][1], device=DEV)
    s.on = torch.zeros(c["lookups"], dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    coords, values, _ = s.inputs[-1]
    _ok(s.lib.bxg_grid_set_values(s.grid.h, coords.data_ptr(), values.data_ptr(), c["n"], None))


def _ok(status):
    if status:
        raise bx.BonxaiError(status, "grid call")


def _run_grid(s, c):
    coords, values, cells = s.turn(s.inputs)
    _ok(s.lib.bxg_grid_set_values(s.grid.h, coords.data_ptr(), values.data_ptr(), c["n"], None))
    _ok(s.lib.bxg_grid_get_values(s.grid.h, cells.data_ptr(), c["lookups"], s.found.data_ptr(),
                                  s.on.data_ptr(), 0))
    return {"values": s.found, "on": s.on}


def _prepare_cloud(s, c, g):
    s.inputs = []
    for _ in range(N_POSES):
        p = _room_surface(g, c["n"])
        cells = torch.floor(p.double() / c["res"]).to(torch.int32)
        pick = torch.randint(0, c["n"], (c["lookups"] + c["n"] // 10,), device=DEV, generator=g)
        look = cells[pick].cpu().numpy()
        s.inputs.append((p.cpu().numpy(), _values(g, c["n"], c["dtype"]).cpu().numpy(),
                         look[:c["lookups"]], look[c["lookups"]:]))
    s.grid = bx.VoxelGrid(c["res"], c["inner_bits"], c["leaf_bits"], _DTYPES[c["dtype"]][0])


def _run_cloud(s, c):
    points, values, cells, erased = s.turn(s.inputs)
    s.grid.clear()
    s.grid.set_values_at_points(points, values)
    was_on = s.grid.set_cells_off(erased)
    return {"was_on": was_on, "on": s.grid.is_cell_on(cells), "values": s.grid.get_values(cells)[0]}


def _prepare_save(s, c, g):
    s.map = bx.ProbabilisticMap(c["res"])
    scans = _scans(g, "lidar", c["n"], 3, c["max_range"])
    torch.cuda.synchronize()
    for p, o in scans:
        s.map.insert_point_cloud(p, o, c["max_range"])
    s.view = s.map.grid()
    s.loaded = bx.VoxelGrid(c["res"], dtype=np.int32)
    s.file = np.zeros(_file_room(c), np.uint8)


def _file_room(c):
    """Bytes set aside for a saved map of this case (some more than it takes)."""
    return 1 << max(16, math.ceil(math.log2(
        16 * _ray_cells("lidar", c["n"], c["res"], c["max_range"]))))


def _run_save(s, c):
    data = s.view.serialize()
    s.file[:len(data)] = np.frombuffer(data, np.uint8)
    s.loaded.clear()
    s.loaded.deserialize(data)
    return {"bytes": len(data), "file": s.file, "cells": s.loaded.active_cells_count()}


def run(state):
    return globals()["_run_" + state.case["kind"]](state, state.case)


# ----------------------------------------------------------------------------
# floors and exact values
# ----------------------------------------------------------------------------
def _ray_cells(scene, n, res, max_range):
    """About how many cells one scan updates (within a third of what was counted):
    the endpoints, and the cells that its rays visit at least once in the volume
    they sweep."""
    reach = min(max_range, {"lidar": 17.0, "depth": 3.0, "room": 2.2}[scene])
    volume = {"lidar": 4500.0, "depth": 13.0, "room": 60.0}[scene]
    volume *= min(1.0, max_range / {"lidar": 30.0, "depth": 5.0, "room": 3.5}[scene]) ** 2
    visits, room = n * reach / res / 1.3, volume / res ** 3
    return visits / (1 + visits / room) + n / 4


def work(case):
    """Bytes a pass cannot do without: points and coordinates in, answers out,
    every updated cell read and written once. The arithmetic is a few operations
    per point and per cell."""
    c, kind = case, case["kind"]
    if kind == "scan":
        size = 24 if c["dtype"] == "float64" else 12
        cells = _ray_cells(c["scene"], c["n"], c["res"], c["max_range"])
        n_bytes = size * c["n"] + 8 * cells + 2 * 17 * c["lookups"]
    elif kind == "ros":
        cells = 0.75 * _ray_cells("lidar", c["n"], c["res"], 12.0)  # returns only
        n_bytes = 12 * c["n"] + 8 * cells + (80.0 / c["res"]) ** 2
    elif kind == "tick":
        mean = (c["n_hi"] - c["n_lo"]) / max(1e-9, math.log(c["n_hi"] / c["n_lo"]))
        cells = [_ray_cells("room" if i % 2 == 0 else "lidar", mean, [0.02, 0.05, 0.1][i % 3],
                            c["max_range"]) for i in range(c["maps"])]
        n_bytes = 12 * mean * c["maps"] + 8 * sum(cells) + 17 * c["lookups"] * c["maps"] / 8
    elif kind == "serve":
        cells = [_ray_cells("lidar" if i % 2 else "room", c["n"], c["res"], c["max_range"])
                 for i in range(c["clients"])]
        n_bytes = c["clients"] * (12 * c["n"] + 17 * c["lookups"]) + 8 * sum(cells)
    elif kind == "lookup":
        n_bytes = 17 * c["n"]
    elif kind in ("grid", "cloud"):
        size = np.dtype(_DTYPES[c["dtype"]][0]).itemsize
        n_bytes = (12 + 2 * size) * c["n"] + (13 + 2 * size) * c["lookups"]
    else:
        cells = 1.3 * _ray_cells("lidar", c["n"], c["res"], c["max_range"])  # of three scans
        n_bytes = 4 * 4 * cells  # pool to file, file to pool
    return {"bytes": float(n_bytes), "flops": float(20 * c.get("n", 0))}


def exact(case, seed):
    """What is read back from an updated grid: the last value written to each
    cell. The other outputs are whole numbers and bytes."""
    if case["kind"] != "grid" or not case["dtype"].startswith("float"):
        return None
    coords, values, cells = (x.cpu().numpy() for x in _grid_inputs(case, _gen(seed))[0])
    last = {}
    for i, xyz in enumerate(map(tuple, coords.tolist())):
        last[xyz] = i
    at = np.array([last[xyz] for xyz in map(tuple, cells.tolist())])
    return {"values": values.astype(np.float64)[at], "on": None}
