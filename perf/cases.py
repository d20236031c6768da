"""Work that users of the mapping framework have it do, as cases to measure.

Each case is one pass of a program around the public entry points of
``vdb_mapping_gb300``: scans inserted into a resident or an empty map, an
accumulation window with its change set, batches of maps, fast mode, raytrace
queries, and a map section passed on to another map. The sensors, voxel sizes
and ranges are those of the benchmark configurations (room and street LiDARs,
depth cameras, long random rays far from the world origin). A pass that
inserts scans ends as a robot's does: with the map section around the sensor
that its planner or its visualisation reads.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) the inputs and the maps a program has in hand
  run(state)          one pass, and what it computed
  work(case)          the bytes and operations a pass cannot do without
  exact(case, seed)   the log-odds of the sections in 64 bits (torch)
"""
import math

import numpy as np
import torch

from vdb_mapping_gb300 import Config, MapBatch, OccupancyVDBMapping

F64 = torch.float64
PROB_HIT, PROB_MISS, THRES_MIN, THRES_MAX = 0.7, 0.4, 0.12, 0.97
PLANNER_BOX = (49, 47, 21)  # half extents, in voxels, of the section read after the scans


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # A small robot's 16-beam LiDAR in a room, coarse voxels: the smallest
        # calls, where launches and latency count.
        dict(name="insert-2k", kind="insert", sensor="lidar", scene="room", rows=16, cols=128, voxel=0.2,
             range=30.0, step=0.2, resident=2, scans=8, host=True),
        # The "small" configuration: a 64-beam LiDAR in a room at 0.1 m, host
        # clouds, into a map that already holds the room.
        dict(name="insert-65k", kind="insert", sensor="lidar", scene="room", rows=64, cols=1024, voxel=0.1,
             range=30.0, step=0.2, resident=2, scans=6, host=True),
        # A depth camera of the serving configuration: 640 x 480 pixels, short
        # rays, 0.02 m voxels, host clouds.
        dict(name="insert-depth", kind="insert", sensor="depth", scene="room", rows=480, cols=640, voxel=0.02,
             range=5.0, step=0.05, resident=2, scans=4, host=True),
        # The same room mapped anew: the map is reset and every leaf is
        # allocated again.
        dict(name="fresh-65k", kind="fresh", sensor="lidar", scene="room", rows=64, cols=1024, voxel=0.1,
             range=30.0, step=0.2, resident=0, scans=4, host=True),
        # The headline "dense" configuration: 262,144 points per scan along a
        # street at 0.05 m, clouds already on the GPU.
        dict(name="insert-dense", kind="insert", sensor="lidar", scene="street", rows=128, cols=2048, voxel=0.05,
             range=60.0, step=1.0, resident=2, scans=6, host=False),
        # The precision-stress configuration, a quarter of its rays: up to
        # 10,000 voxels per ray, far from the world origin, few rays per leaf.
        dict(name="insert-stress", kind="insert", sensor="sphere", scene="none", rows=1, cols=16381, voxel=0.02,
             range=250.0, step=0.0, resident=0, scans=1, host=False),
        # An accumulation window of an odd-sized sensor: four clouds collected,
        # integrated together, and the changes sent on (remote mapping).
        dict(name="window-33k", kind="window", sensor="lidar", scene="room", rows=33, cols=997, voxel=0.05,
             range=25.0, step=0.05, resident=2, scans=4, host=True),
        # The "batched" configuration: 32 independent maps of mixed sensors,
        # one scan per map per step, clouds on the GPU.
        dict(name="batch-32", kind="batch", sensor="mixed", scene="room", maps=32, n_min=2000, n_max=307200,
             resident=1, scans=3, host=False),
        # Fast mode on the street: only voxels that are active are cleared.
        dict(name="fast-dense", kind="fast", sensor="lidar", scene="street", rows=128, cols=2048, voxel=0.05,
             range=60.0, step=0.1, resident=5, scans=6, host=False),
        # Raytrace queries: a planner's thousand, and a sensor simulation's
        # million, in the street map.
        dict(name="trace-1k", kind="trace", sensor="lidar", scene="street", rows=64, cols=1024, voxel=0.1,
             range=60.0, step=0.05, resident=6, queries=1000, length=30.0),
        dict(name="trace-1m", kind="trace", sensor="lidar", scene="street", rows=128, cols=2048, voxel=0.05,
             range=60.0, step=0.05, resident=6, queries=1048576, length=60.0),
        # A section of one robot's map, closed (smoothed) and applied to
        # another robot's map.
        dict(name="section-close", kind="section", sensor="lidar", scene="room", rows=64, cols=1024, voxel=0.1,
             range=30.0, step=0.02, resident=8, box_x=101, box_y=99, box_z=31, iterations=2),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    while True:
        kind = rng.choice(["insert", "insert", "insert", "fresh", "window", "batch", "fast", "trace", "section"])
        if kind == "batch":
            n_max = log_int(20000, 307200)
            return dict(kind="batch", sensor="mixed", scene="room", maps=rng.randint(3, 32), n_min=2000,
                        n_max=n_max, resident=1, scans=rng.randint(1, 2), host=rng.random() < 0.3)
        sensor = rng.choice(["lidar", "lidar", "depth", "sphere"]) if kind in ("insert", "fresh") else "lidar"
        scene = "none" if sensor == "sphere" else "room" if sensor == "depth" else rng.choice(["room", "street"])
        c = dict(kind=kind, sensor=sensor, scene=scene)
        if sensor == "lidar":
            c.update(rows=rng.choice([16, 32, 33, 64, 128]), cols=log_int(64, 2048),
                     voxel=rng.choice([0.05, 0.1, 0.2]), range=round(rng.uniform(20.0, 60.0), 1))
        elif sensor == "depth":
            rows = log_int(60, 480)
            c.update(rows=rows, cols=rows * 4 // 3 + rng.randint(0, 1), voxel=rng.choice([0.02, 0.05]), range=5.0)
        else:
            c.update(rows=1, cols=log_int(500, 16381), voxel=rng.choice([0.02, 0.05]), range=250.0)
        c["step"] = round(rng.uniform(0.02, 0.2), 2)
        c["resident"] = 0 if kind == "fresh" or sensor == "sphere" else rng.randint(1, 4)
        if kind in ("fast", "trace", "section"):
            c["resident"] = rng.randint(6, 8)  # (a voxel turns active at its fifth hit)
        if kind in ("insert", "fresh", "window", "fast"):
            c.update(scans=1 if sensor == "sphere" else rng.randint(2, 6), host=rng.random() < 0.5)
        elif kind == "trace":
            c.update(queries=log_int(1000, 1048576), length=round(rng.uniform(10.0, 60.0), 1))
        else:
            c.update(box_x=rng.randint(20, 101), box_y=rng.randint(20, 99), box_z=rng.randint(5, 31),
                     iterations=rng.randint(1, 2))
        return c


# ---------------------------------------------------------------------------
# Scenes and sensors (float64 on the GPU, from the seed alone)
# ---------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(x):
    return torch.as_tensor(x, dtype=F64, device=_device())


class Scene:
    """A room (walls, boxes) or a street (ground, buildings, cars, poles), or
    nothing (the sphere sensor brings its own ranges)."""

    def __init__(self, kind, seed, size=1.0):
        rng = np.random.default_rng([seed, 17])
        self.kind = kind
        boxes, cyls = [], []
        if kind == "room":
            self.lo, self.hi = np.array([-20.0, -20.0, 0.0]) * size, np.array([20.0, 20.0, 6.0]) * size
            while len(boxes) < 20:
                c = rng.uniform([-18, -18], [18, 18]) * size
                s = rng.uniform([0.3, 0.3, 0.5], [3.0, 3.0, 3.0])
                if abs(c[0] - 1.0) < 2.5 + s[0] / 2 and abs(c[1]) < 1.5 + s[1] / 2:
                    continue  # the sensor's path
                boxes.append([c[0] - s[0] / 2, c[1] - s[1] / 2, 0.0, c[0] + s[0] / 2, c[1] + s[1] / 2, s[2]])
        elif kind == "street":
            self.lo, self.hi = np.array([-100.0, -100.0, 0.0]), np.array([100.0, 100.0, 20.0])
            for side in (-1, 1):
                x = -100.0
                while x < 100.0:
                    w, depth, h = rng.uniform(8, 25), rng.uniform(10, 30), rng.uniform(5, 20)
                    y0 = side * rng.uniform(10, 14)
                    y1 = y0 + side * depth
                    boxes.append([x, min(y0, y1), 0.0, x + w, max(y0, y1), h])
                    x += w + rng.uniform(1, 6)
            for _ in range(60):
                cx, cy = rng.uniform(-100, 100), rng.choice([-1, 1]) * rng.uniform(5.5, 8.0)
                boxes.append([cx - 2.2, cy - 0.9, 0.0, cx + 2.2, cy + 0.9, 1.5])
            for _ in range(80):
                cyls.append([rng.uniform(-100, 100), rng.choice([-1, 1]) * rng.uniform(8.5, 9.8),
                             rng.uniform(0.08, 0.5), rng.uniform(3, 9)])
        self.boxes, self.cyls = boxes, cyls

    def origin(self, k, step):
        if self.kind == "none":
            return np.array([5000.0, -3000.0, 40.0]) + k * step * np.array([0.86, -0.49, 0.12])
        if self.kind == "street":
            return np.array([-20.0 + step * k, 0.0, 1.8])
        return np.array([step * k, 0.0, 1.5])

    def distances(self, o, d):
        """Distance along each unit ray to the first surface (inf: none)."""
        inv = 1.0 / torch.where(d == 0, torch.full_like(d, 1e-300), d)
        lo, hi = _t(self.lo), _t(self.hi)
        out = torch.maximum((lo - o) * inv, (hi - o) * inv).amin(dim=1)  # leaving the enclosure
        t = torch.full_like(out, math.inf)
        if self.kind == "street":
            t = torch.where(d[:, 2] < 0, -o[2] * inv[:, 2], t)
        for b in self.boxes:
            t1, t2 = (_t(b[:3]) - o) * inv, (_t(b[3:]) - o) * inv
            near, far = torch.minimum(t1, t2).amax(dim=1), torch.maximum(t1, t2).amin(dim=1)
            t = torch.where((far >= near) & (near > 1e-6) & (near < t), near, t)
        a = d[:, 0] ** 2 + d[:, 1] ** 2
        for cx, cy, r, z1 in self.cyls:
            ox, oy = o[0] - cx, o[1] - cy
            b = 2 * (ox * d[:, 0] + oy * d[:, 1])
            disc = b * b - 4 * a * (ox * ox + oy * oy - r * r)
            s = (-b - torch.sqrt(disc.clamp(min=0))) / (2 * a).clamp(min=1e-12)
            z = o[2] + s * d[:, 2]
            t = torch.where((disc >= 0) & (s > 1e-6) & (z >= 0) & (z <= z1) & (s < t), s, t)
        if self.kind == "room":
            return torch.minimum(t, out)
        return torch.where(t <= out, t, torch.full_like(t, math.inf))


def directions(case, gen):
    """Unit rays of the sensor, (N, 3)."""
    rows, cols = case["rows"], case["cols"]
    if case["sensor"] == "sphere":
        v = torch.randn(rows * cols, 3, generator=gen, dtype=F64, device=_device())
        return v / v.norm(dim=1, keepdim=True)
    if case["sensor"] == "depth":
        tx = math.tan(math.radians(45.0)) * torch.linspace(-1, 1, cols, dtype=F64, device=_device())
        ty = math.tan(math.radians(30.0)) * torch.linspace(-1, 1, rows, dtype=F64, device=_device())
        gy, gx = torch.meshgrid(ty, tx, indexing="ij")
        v = torch.stack([torch.ones_like(gx), gx, gy - 0.1], dim=-1).reshape(-1, 3)
        return v / v.norm(dim=1, keepdim=True)
    el = torch.deg2rad(torch.linspace(-25.0, 15.0, rows, dtype=F64, device=_device()))[:, None]
    az = (torch.arange(cols, dtype=F64, device=_device()) * (2 * math.pi / cols))[None, :]
    return torch.stack([torch.cos(el) * torch.cos(az), torch.cos(el) * torch.sin(az),
                        torch.sin(el).expand(rows, cols)], dim=-1).reshape(-1, 3)


def clouds(case, seed, count):
    """`count` scans along the sensor's path: [(points (N, 4) float32, origin)].
    Ranges carry 1 cm of noise; 3% of the beams return nothing and end at twice
    the range, so that they only clear space."""
    gen = torch.Generator(device=_device()).manual_seed(int(seed) * 1000003 + 7)
    scene = Scene(case["scene"], seed, case.get("size", 1.0))
    out = []
    for k in range(count):
        d = directions(case, gen)
        o = scene.origin(k, case["step"])
        n = d.shape[0]
        if case["sensor"] == "sphere":
            u = torch.rand(n, generator=gen, dtype=F64, device=_device())
            r = torch.exp(math.log(0.5) + u * (math.log(200.0) - math.log(0.5)))
        else:
            r = scene.distances(_t(o), d)
            r = r + 0.01 * torch.randn(n, generator=gen, dtype=F64, device=_device())
            lost = (torch.rand(n, generator=gen, dtype=F64, device=_device()) < 0.03) | ~torch.isfinite(r)
            r = torch.where(lost, torch.full_like(r, 2.0 * case["range"]), r)
        pts = torch.ones(n, 4, dtype=torch.float32, device=_device())
        pts[:, :3] = (_t(o) + d * r[:, None]).to(torch.float32)
        out.append((pts, o))
    return out


def config(case, fast=False):
    return Config(max_range=case["range"], fast_mode=fast, accumulation_period=0.0, prob_hit=PROB_HIT,
                  prob_miss=PROB_MISS, prob_thres_min=THRES_MIN, prob_thres_max=THRES_MAX)


def members(case, seed):
    """The single-map cases of a batch's maps: mixed sensors of mixed sizes."""
    rng = np.random.default_rng([case["maps"], case["n_max"], 4])
    out = []
    for i in range(case["maps"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        c = dict(scene="room", voxel=float(rng.choice([0.02, 0.05, 0.1, 0.2])), step=0.1, seed=int(seed) * 1009 + i)
        if rng.random() < 0.5:
            cols = max(4, min(640, int(round(math.sqrt(n * 4.0 / 3.0)))))
            c.update(sensor="depth", cols=cols, rows=max(3, min(480, n // cols)), range=5.0)
        else:
            rows = int(rng.choice([16, 32, 64, 128]))
            c.update(sensor="lidar", rows=rows, cols=max(8, n // rows), range=round(float(rng.uniform(30, 60)), 1),
                     size=2.0)
            c["voxel"] = max(c["voxel"], 0.05)  # (one such map at 0.02 m would be most of the batch)
        out.append(c)
    return out


class Buffers:
    """A program's own arrays for leaves it reads (room for the most there can
    be; the rows past the last leaf are zero)."""

    def __init__(self, room, **rows):
        self.room, self.used = room, 0
        self.arrays = {k: np.zeros((room,) + shape, dtype) for k, (shape, dtype) in rows.items()}

    def take(self, **new):
        n = min(self.room, max(len(x) for x in new.values()))
        for k, x in new.items():
            self.arrays[k][:n] = x[:n]
            if n < self.used:
                self.arrays[k][n:self.used] = 0
        self.used = n
        return dict(self.arrays)


def section_buffers(boxes):
    """Buffers for the sections of index boxes [(lo, hi)], one after the other."""
    room = sum(int(np.prod((np.asarray(hi) >> 3) - (np.asarray(lo) >> 3) + 1)) for lo, hi in boxes)
    return Buffers(room, origins=((3,), np.int32), values=((512,), np.float32), masks=((8,), np.int64))


def box_of(case, o, half=PLANNER_BOX):
    """Index box around the sensor voxel of a scan taken from `o`."""
    if case["kind"] == "section":
        half = (case["box_x"], case["box_y"], case["box_z"])
    c = to_index(_t(o)[None, :], case["voxel"])[0].cpu().numpy()
    h = np.array(half)
    return (c - h).astype(np.int32), (c + h - 1).astype(np.int32)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ms = members(case, seed)
        total = case["resident"] + case["scans"]
        per_map = [clouds(c, c["seed"], total) for c in ms]
        counts = [s[0][0].shape[0] for s in per_map]
        steps = [(torch.cat([s[k][0] for s in per_map]), [s[k][1] for s in per_map]) for k in range(total)]
        b = MapBatch([c["voxel"] for c in ms])
        for i, c in enumerate(ms):
            b.setConfig(i, config(c))
        for pts, origins in steps[:case["resident"]]:
            b.insert_packed(pts, counts, origins)
        todo = steps[case["resident"]:]
        if case["host"]:
            todo = [(p.cpu().numpy(), o) for p, o in todo]
        boxes = [box_of(dict(c, kind="batch"), todo[-1][1][i], (17, 15, 9)) for i, c in enumerate(ms)]
        torch.cuda.synchronize()
        return dict(case=case, batch=b, counts=counts, steps=todo, boxes=boxes, out=section_buffers(boxes))

    scans = clouds(case, seed, case["resident"] + case.get("scans", 0))
    m = OccupancyVDBMapping(case["voxel"])
    m.setConfig(config(case))
    m.addInputSource("sensor", case["range"], 0)
    if kind == "window":
        m.trackChanges()
    for pts, o in scans[:case["resident"]]:
        m.insertPointCloud(pts, o, "sensor")
    if kind == "fast":
        m.setConfig(config(case, fast=True))
    st = dict(case=case, map=m)
    if kind == "trace":
        rng = np.random.default_rng([seed, 3])
        n = case["queries"]
        d = rng.normal(size=(n, 3))
        d[:, 2] *= 0.3  # mostly near the horizon
        at = rng.integers(0, len(scans), n)
        st.update(origins=np.array([o for _, o in scans])[at], directions=d)
    elif kind == "section":
        st["box"] = box_of(case, scans[-1][1])
        other = OccupancyVDBMapping(case["voxel"])
        other.setConfig(config(case))
        other.addInputSource("sensor", case["range"], 0)
        st["other"] = other
    else:
        todo = scans[case["resident"]:]
        st["box"] = box_of(case, todo[-1][1])
        st["scans"] = [(p.cpu().numpy() if case["host"] else p, o) for p, o in todo]
    if kind == "window":
        st["out"] = Buffers(1 << 17, origins=((3,), np.int32), active=((8,), np.int64), value=((8,), np.int64))
    elif "box" in st:
        st["out"] = section_buffers([st["box"]])
    torch.cuda.synchronize()
    return st


def _counts(stats):
    return [int(stats[k]) for k in ("rays", "visits", "hits", "updates", "touched_leaves", "new_leaves")]


def _section(out, s):
    origins, values, masks = s
    return out.take(origins=origins, values=values, masks=masks.view(np.int64))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        stats = [_counts(b.insert_packed(p, state["counts"], o)) for p, o in state["steps"]]
        # The sections of all maps, one after the other, in one set of arrays.
        parts = [b.getMapSection(i, lo, hi, full=True) for i, (lo, hi) in enumerate(state["boxes"])]
        return {"stats": np.array(stats), "leaves": np.array([len(p[0]) for p in parts]),
                "section": _section(state["out"], tuple(np.concatenate([p[j] for p in parts]) for j in range(3)))}
    m = state["map"]
    if kind == "trace":
        ok, ends = m.raytrace(state["origins"], state["directions"], case["length"])
        return {"ok": ok, "ends": ends}
    if kind == "section":
        lo, hi = state["box"]
        origins, _, masks = m.getMapSection(lo, hi)
        state["other"].applyMapSectionStates(lo, hi, origins, masks, smooth=True, iterations=case["iterations"])
        return {"section": _section(state["out"], state["other"].getMapSection(lo, hi))}
    if kind == "window":
        for cloud, o in state["scans"]:
            m.accumulateUpdate(cloud, o, "sensor")
        m.integrateUpdate()
        origins, active, value = m.exportChanges()
        return {"stats": np.array(_counts(m.last_stats)),
                "changes": state["out"].take(origins=origins, active=active.view(np.int64), value=value.view(np.int64))}
    if kind == "fresh":
        m.resetMap()
    stats = []
    for cloud, o in state["scans"]:
        m.insertPointCloud(cloud, o, "sensor")
        stats.append(_counts(m.last_stats))
    return {"stats": np.array(stats), "section": _section(state["out"], m.getMapSection(*state["box"], full=True))}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

# As measured on these scenes: mean length of a ray in metres of voxel steps
# (L1), the share of the visits that update a voxel of their own (the others
# meet a voxel that another ray of the scan visited), and updated voxels per
# touched leaf.
_ROOM, _STREET, _DEPTH, _SPHERE = (19.7, 0.4, 90.0), (23.9, 0.5, 42.0), (6.9, 0.065, 400.0), (49.7, 0.97, 8.9)


def _rays(case):
    length, share, per_leaf = (_SPHERE if case["sensor"] == "sphere" else _DEPTH if case["sensor"] == "depth"
                               else _STREET if case["scene"] == "street" else _ROOM)
    if case["sensor"] == "lidar":
        length = min(length * case.get("size", 1.0), 1.3 * case["range"])
    return case["rows"] * case["cols"], length / case["voxel"], share, per_leaf


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [work(dict(c, kind="insert", scans=case["scans"], resident=1)) for c in members(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "trace":
        # Queries in (7 doubles) and answers out, one map bit per voxel walked,
        # one FP64 addition per voxel.
        steps = 0.4 * case["length"] * 1.3 / case["voxel"]
        return {"bytes": case["queries"] * (56 + 25 + steps / 8), "flops": case["queries"] * steps}
    if kind == "section":
        voxels = 8.0 * case["box_x"] * case["box_y"] * case["box_z"]
        # The states out of one map, into the other, and the result with its values.
        return {"bytes": voxels * (2 * 0.25 + 4), "flops": voxels * 2 * 26 * case["iterations"]}
    n, steps, share, per_leaf = _rays(case)
    visits = n * steps
    updates = share * visits
    if kind == "fast":
        updates, per_leaf = 1.0 * n, 13.0  # only active voxels and the endpoints are updated
    # Points in; per updated voxel its value read and written and two mask
    # bits; per touched leaf its masks; and the section out.
    scan = 12.0 * n + 8.25 * updates + 128.0 * updates / per_leaf
    section = 8.0 * PLANNER_BOX[0] * PLANNER_BOX[1] * PLANNER_BOX[2] * 8.25
    return {"bytes": case["scans"] * scan + section, "flops": case["scans"] * visits}


# ---------------------------------------------------------------------------
# The sections in 64 bits
# ---------------------------------------------------------------------------

def to_index(p, voxel):
    """World to voxel index: a coordinate that is no multiple of the voxel size
    moves up by half a voxel, then is scaled and floored."""
    res = torch.full((), voxel, dtype=F64, device=p.device)
    shifted = torch.where(torch.fmod(p, res) != 0.0, p + voxel / 2.0, p)
    return torch.floor(shifted * (1.0 / voxel)).to(torch.int64)


class Window:
    """The voxels of an index box: log-odds in 64 bits and states."""

    def __init__(self, lo, hi, voxel):
        self.lo, self.voxel = torch.as_tensor(lo, device=_device()).to(torch.int64), voxel
        self.dims = [int(b) - int(a) + 1 for a, b in zip(lo, hi)]
        self.v = torch.zeros(math.prod(self.dims), dtype=F64, device=_device())
        self.on = torch.zeros_like(self.v, dtype=torch.bool)

    def place(self, vox, keep):
        """Flat index of the voxels inside the box; one past the end for the others."""
        r = vox - self.lo
        inside = keep & (r >= 0).all(dim=1) & (r < torch.tensor(self.dims, device=r.device)).all(dim=1)
        flat = (r[:, 0] * self.dims[1] + r[:, 1]) * self.dims[2] + r[:, 2]
        return torch.where(inside, flat, torch.full_like(flat, self.v.numel())), inside

    def mark(self, pts, o, rng):
        """Voxels that the scan visits and hits: Amanatides-Woo from the sensor
        voxel to each endpoint's voxel, ties to the higher axis."""
        p, o = pts[:, :3].to(F64), _t(o)
        d = p - o
        length = torch.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])
        clipped = (length > rng) if rng > 0 else torch.zeros_like(length, dtype=torch.bool)
        p = torch.where(clipped[:, None], o + d / length[:, None] * rng, p)
        end, start = to_index(p, self.voxel), to_index(o[None, :], self.voxel)
        visited = torch.zeros(self.v.numel() + 1, dtype=torch.bool, device=p.device)
        hit = torch.zeros_like(visited)
        hit[self.place(end, ~clipped)[0]] = True
        vox = start.expand_as(end).clone()
        delta = (end - start).to(F64)
        step = torch.sign(delta).to(torch.int64)
        huge = torch.full_like(delta, 1.7976931348623157e308)
        inv = 1.0 / delta
        moving = delta != 0
        pos = vox.to(F64) + 0.5
        nxt = torch.where(moving, ((vox + (step > 0)).to(F64) - pos) * inv, huge)
        inc = torch.where(moving, step.to(F64) * inv, huge)
        alive = moving.any(dim=1)
        # A ray that leaves the box (the sensor is inside it, or outside by
        # less than the path's length) does not come back.
        entered = torch.zeros_like(alive)
        for _ in range(sum(self.dims) * 4):
            at, inside = self.place(vox, alive)
            visited[at] = True
            entered |= inside
            alive = alive & (inside | ~entered)
            x, y, z = nxt.unbind(1)
            ax = (x < y) & (x < z)
            ay = ~ax & (y < z)
            axis = torch.stack([ax, ay, ~ax & ~ay], dim=1)
            alive = alive & (torch.where(axis, nxt, torch.zeros_like(nxt)).sum(dim=1) <= 1.0)
            vox = vox + torch.where(axis, step, torch.zeros_like(step))
            nxt = torch.where(axis, nxt + inc, nxt)
            if not bool(alive.any()):
                break
        return visited[:-1], hit[:-1]

    def update(self, visited, hit):
        odds = {k: math.log(p) - math.log(1 - p) for k, p in
                (("hit", PROB_HIT), ("miss", PROB_MISS), ("lo", THRES_MIN), ("hi", THRES_MAX), ("max", 0.99))}
        miss = visited & ~hit
        v = torch.where(hit, self.v + odds["hit"], torch.where(miss, self.v + odds["miss"], self.v))
        up, down = hit & (v > odds["hi"]), miss & (v < odds["lo"])
        self.v = torch.where(up, v.clamp(max=odds["max"]), torch.where(down, v.clamp(min=-odds["max"]), v))
        self.on = (self.on | up) & ~down

    def insert(self, pts, o, rng, fast=False):
        visited, hit = self.mark(pts, o, rng)
        self.update(visited & self.on if fast else visited, hit)

    def leaves(self, values):
        """`values` of the box as leaves sorted by origin (8^3 voxels, x outermost),
        those with an active voxel or a value other than 0."""
        lo = self.lo.cpu().numpy()
        first = lo // 8 * 8
        pad = [int(a) for a in lo - first]
        n = [-(-(p + d) // 8) for p, d in zip(pad, self.dims)]
        got = []
        for x in (values, self.on):
            g = torch.zeros([8 * k for k in n], dtype=x.dtype, device=x.device)
            g[pad[0]:pad[0] + self.dims[0], pad[1]:pad[1] + self.dims[1], pad[2]:pad[2] + self.dims[2]] = \
                x.reshape(self.dims)
            got.append(g.reshape(n[0], 8, n[1], 8, n[2], 8).permute(0, 2, 4, 1, 3, 5).reshape(-1, 512))
        kept = (got[0] != 0).any(dim=1) | got[1].any(dim=1)
        return got[0][kept].cpu().numpy()


def _padded(boxes, parts):
    out = section_buffers(boxes).arrays["values"].astype(np.float64)
    got = np.concatenate(parts)
    out[:len(got)] = got
    return {"origins": None, "values": out, "masks": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("trace", "window"):
        return None  # end points are voxel corners found by look-up; change sets are bits
    if kind == "batch":
        parts, boxes = [], []
        for c in members(case, seed):
            scans = clouds(c, c["seed"], case["resident"] + case["scans"])
            boxes.append(box_of(dict(c, kind="batch"), scans[-1][1], (17, 15, 9)))
            w = Window(*boxes[-1], c["voxel"])
            for pts, o in scans:
                w.insert(pts, o, c["range"])
            parts.append(w.leaves(w.v))
        return {"stats": None, "leaves": None, "section": _padded(boxes, parts)}
    scans = clouds(case, seed, case["resident"] + case.get("scans", 0))
    box = box_of(case, scans[-1][1])
    w = Window(*box, case["voxel"])
    for k, (pts, o) in enumerate(scans):
        w.insert(pts, o, case["range"], fast=kind == "fast" and k >= case["resident"])
    if kind == "section":
        # The active voxels closed: dilated, then eroded, by the 26 neighbours.
        it = case["iterations"]
        x = torch.nn.functional.pad(w.on.reshape(1, 1, *w.dims).to(torch.float32), [2 * it] * 6)
        for grow in [True] * it + [False] * it:
            x = torch.nn.functional.max_pool3d(x if grow else 1 - x, 3, stride=1, padding=1)
            x = x if grow else 1 - x
        x = x[0, 0, 2 * it:-2 * it, 2 * it:-2 * it, 2 * it:-2 * it].reshape(-1)
        w.on = x > 0
        return {"section": _padded([box], [w.leaves(x.to(F64))])}
    return {"stats": None, "section": _padded([box], [w.leaves(w.v)])}
