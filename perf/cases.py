"""The framework's performance cases: what a user has it do, through its public entry points.

listed() holds the cases by name, draw() more of the same ranges, prepare()
the inputs a program holds before the call, run() one pass, work() what that
pass cannot do without and exact() its floating results in 64 bits.

Scenes stand in for the indoor scans, LiDAR scans and volumes of the
benchmark configurations (``flashknn_exprepo_b200/synthetic.py``), generated
here on the GPU: rooms (surfaces with 5 mm noise, millimetre coordinates,
random point order), ray-cast scans (points in scan order, density falling
with the range) and uniform cubes.
"""
import math

import numpy as np
import torch

import flashknn_exprepo_b200 as fk
from flashknn_exprepo_b200.hierarchy import build_flash_hierarchy

DEV = "cuda"


def listed():
    return [
        # The smallest call: one small volume, K=16 (latency and launches count).
        {"name": "cube_k16", "kind": "self", "scene": "cube", "n": 16384, "clouds": 1, "k": 16,
         "voxel": 0.0197, "num_down": 2, "train": False},
        # Inference over a batch of 16 uneven clouds: the benchmark's own step.
        {"name": "batch16_k16", "kind": "self", "scene": "mixed", "n": 1464355, "clouds": 16,
         "k": 16, "voxel": 0.05, "num_down": 2, "train": False},
        # A training step's query: forward, then the gradient of the squared distances.
        {"name": "train_batch6_k16", "kind": "self", "scene": "mixed", "n": 550007, "clouds": 6,
         "k": 16, "voxel": 0.05, "num_down": 2, "train": True},
        # The reference's drop-in call on an indoor scan, K=32, int64 indices.
        {"name": "room_grid_k32", "kind": "grid", "scene": "room", "n": 80000, "clouds": 1,
         "k": 32, "voxel": 0.04, "num_down": 2},
        # The drop-in call on a raw LiDAR scan with coarse parent cells: many
        # candidates a query in the near field.
        {"name": "lidar_grid_k16_alpha8", "kind": "grid", "scene": "scan", "n": 115003,
         "clouds": 1, "k": 16, "voxel": 0.05, "num_down": 3},
        # A strided layer: every fourth point of an indoor scan asks for K=32.
        {"name": "room_selected_k32", "kind": "selected", "scene": "room", "n": 80000,
         "clouds": 1, "k": 32, "voxel": 0.04, "num_down": 2, "stride": 4},
        # Feature interpolation in a decoder: 3 nearest coarse points of every fine point.
        {"name": "interp_batch4_k3", "kind": "general", "scene": "mixed", "n": 300007,
         "clouds": 4, "k": 3, "voxel": 0.05, "num_down": 2, "stride": 4},
        # Ball query of an indoor scan: up to 32 points within 10 cm.
        {"name": "room_ball_k32", "kind": "ball", "scene": "room", "n": 80000, "clouds": 1,
         "k": 32, "radius": 0.1},
        # Dense-to-subset map of a batch onto its 10 cm representatives.
        {"name": "back_batch8_k1", "kind": "back", "scene": "mixed", "n": 700001, "clouds": 8,
         "k": 1, "voxel": 0.05, "size": 0.1},
        # The adaptive octree on a raw LiDAR scan.
        {"name": "adaptive_lidar_k16", "kind": "adaptive", "scene": "scan", "n": 115003,
         "clouds": 1, "k": 16, "voxel": 0.05},
        # A whole data-loading step of a point network: the index hierarchy of one scan.
        {"name": "hierarchy_lidar_k24", "kind": "hierarchy", "scene": "thinned", "n": 72003,
         "clouds": 1, "k": 24, "voxel": 0.06},
        # An attention layer's neighbourhoods in training: query, gather of 64
        # channels with the relative positions, and its backward.
        {"name": "group_train_k16_c64", "kind": "group", "scene": "mixed", "n": 200003,
         "clouds": 3, "k": 16, "voxel": 0.05, "num_down": 2, "c": 64, "with_xyz": True},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["self", "self", "self", "grid", "grid", "selected", "general", "ball",
                       "back", "adaptive", "hierarchy", "group", "group"])
    case = {"kind": kind, "scene": rng.choice(["room", "mixed", "thinned"]), "clouds": 1,
            "k": rng.choice([5, 8, 12, 16, 16, 24, 32]), "voxel": 0.05}
    n_hi = 150000
    if kind == "self":
        case.update(num_down=2, train=rng.random() < 0.4)
        if rng.random() < 0.3:
            case["scene"] = "cube"
        n_hi = 550000 if case["k"] > 16 or case["train"] else 1400000
    elif kind == "grid":
        case.update(num_down=rng.choice([2, 2, 3]))
        if rng.random() < 0.4:
            case["scene"] = "scan"
    elif kind == "selected":
        case.update(num_down=2, stride=rng.choice([2, 3, 4, 8]))
    elif kind == "general":
        case.update(num_down=2, k=rng.choice([1, 3, 4, 8, 16]), stride=rng.choice([2, 4, 6]))
        n_hi = 300000
    elif kind == "ball":
        case.update(radius=rng.choice([0.08, 0.1, 0.15]), k=rng.choice([8, 16, 32]))
    elif kind == "back":
        case.update(k=1, size=rng.choice([0.1, 0.12, 0.16]))
        n_hi = 700000
    elif kind == "adaptive":
        case.update(scene=rng.choice(["scan", "room", "thinned"]))
        n_hi = 115000
    elif kind == "hierarchy":
        case.update(scene=rng.choice(["thinned", "room"]), k=rng.choice([16, 24]), voxel=0.06)
        n_hi = 72000
    else:
        case.update(num_down=2, k=rng.choice([8, 16]), c=rng.choice([16, 32, 48, 64, 96]),
                    with_xyz=rng.random() < 0.5)
        n_hi = 130000
    case["n"] = _between(rng, 4096, n_hi)
    if case["scene"] == "cube":
        # parent cells of about two mean spacings
        case["voxel"] = round(0.5 * case["n"] ** (-1.0 / 3.0), 5)
    elif kind in ("self", "general", "back", "group"):
        case["scene"] = "mixed"
        case["clouds"] = rng.randint(1, max(1, min(16, case["n"] // 8000)))
    elif case["scene"] == "mixed":
        case["scene"] = "room"
    return case


# ------------------------------------------------------------------- scenes

def _first_of_voxel(xyz, voxel):
    """Ascending indices of the first point of every occupied voxel."""
    g = torch.floor(xyz / voxel).long()
    g = g - g.min(0).values
    ext = g.max(0).values + 1
    key = (g[:, 0] * ext[1] + g[:, 1]) * ext[2] + g[:, 2]
    uniq, inv = torch.unique(key, return_inverse=True)
    first = torch.full((uniq.numel(),), len(xyz), dtype=torch.int64, device=xyz.device)
    first.scatter_reduce_(0, inv, torch.arange(len(xyz), device=xyz.device), "amin")
    return first.sort().values


def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device=DEV)


def _cube(gen, n, voxel):
    pts = torch.empty((0, 3), device=DEV)
    while len(pts) < n:
        pts = torch.cat([pts, _rand(gen, n, 3)])
        pts = pts[_first_of_voxel(pts, voxel)]
    return pts[:n].contiguous()


def _room(gen, rng, n, voxel):
    """Floor, ceiling, walls and ten boxes; one point per voxel, random order."""
    scale = max(1.0, (n / 60000.0) ** 0.5)
    raw = int(n * 1.6)
    while True:
        dims = np.array([6.0 * scale, 8.0 * scale, 3.0])
        faces = []  # (fixed axis, value, lo, hi) of every rectangle
        for axis in range(3):
            for value in (0.0, dims[axis]):
                faces.append((axis, value, np.zeros(3), dims))
        for _ in range(10):
            size = np.array([rng.uniform(0.4, 2.0), rng.uniform(0.4, 2.0), rng.uniform(0.4, 1.8)])
            lo = np.array([rng.uniform(0.1, dims[0] - size[0] - 0.1),
                           rng.uniform(0.1, dims[1] - size[1] - 0.1), 0.0])
            hi = lo + size
            faces += [(2, hi[2], lo, hi), (0, lo[0], lo, hi), (0, hi[0], lo, hi),
                      (1, lo[1], lo, hi), (1, hi[1], lo, hi)]
        area = np.array([np.prod([h[a] - l[a] for a in range(3) if a != ax])
                         for ax, _, l, h in faces])
        count = np.maximum(1, raw * area / area.sum()).astype(np.int64)
        lo = torch.tensor(np.array([f[2] for f in faces]), dtype=torch.float32, device=DEV)
        hi = torch.tensor(np.array([f[3] for f in faces]), dtype=torch.float32, device=DEV)
        for i, (ax, v, _, _) in enumerate(faces):
            lo[i, ax] = hi[i, ax] = v
        which = torch.repeat_interleave(torch.arange(len(faces), device=DEV),
                                        torch.tensor(count, device=DEV))
        pts = lo[which] + _rand(gen, len(which), 3) * (hi - lo)[which]
        pts = pts + 0.005 * torch.randn(pts.shape, generator=gen, device=DEV)
        pts = torch.round((pts - pts.min(0).values) * 1000.0) / 1000.0
        pts = pts[torch.randperm(len(pts), generator=gen, device=DEV)]
        pts = pts[_first_of_voxel(pts, voxel)]
        if len(pts) >= n:
            return pts[:n].contiguous()
        raw = int(raw * 1.5)
        scale *= 1.05


def _scan(gen, rng, n, voxel, thinned):
    """A spinning-LiDAR scan: ground, cylinders, boxes and facades, 10 % of the
    returns dropped; thinned: one point per voxel.  The n points nearest to a
    random one, in scan order."""
    rings, azimuths = 64, 2048
    while rings * azimuths * (0.45 if thinned else 0.85) < n:
        rings, azimuths = (2 * rings, azimuths) if rings * 32 <= azimuths else (rings, 2 * azimuths)
    while True:
        elev = torch.deg2rad(torch.linspace(-24.8, 2.0, rings, device=DEV))
        az = torch.arange(azimuths, device=DEV) * (2 * math.pi / azimuths)
        e, a = torch.meshgrid(elev, az, indexing="ij")
        d = torch.stack([e.cos() * a.cos(), e.cos() * a.sin(), e.sin()], -1).reshape(-1, 3)
        t = torch.where(d[:, 2] < -1e-6, -1.7 / d[:, 2], math.inf)
        flat = d[:, 0] ** 2 + d[:, 1] ** 2
        for _ in range(60):
            r, ang, rad = rng.uniform(4.0, 45.0), rng.uniform(0, 2 * math.pi), rng.uniform(.15, .8)
            cx, cy, top = r * math.cos(ang), r * math.sin(ang), rng.uniform(0.5, 8.0) - 1.7
            b = -2 * (d[:, 0] * cx + d[:, 1] * cy)
            disc = b * b - 4 * flat * (cx * cx + cy * cy - rad * rad)
            s = (-b - disc.clamp(min=0).sqrt()) / (2 * flat)
            z = s * d[:, 2]
            hit = (disc > 0) & (s > 0) & (z >= -1.7) & (z <= top)
            t = torch.where(hit & (s < t), s, t)
        inv = 1.0 / torch.where(d.abs() < 1e-12, 1e-12, d)
        for _ in range(40):
            r, ang = rng.uniform(6.0, 48.0), rng.uniform(0, 2 * math.pi)
            cx, cy = r * math.cos(ang), r * math.sin(ang)
            sx, sy, sz = rng.uniform(1.0, 8.0), rng.uniform(1.0, 8.0), rng.uniform(1.0, 10.0)
            lo = torch.tensor([cx - sx / 2, cy - sy / 2, -1.7], device=DEV) * inv
            hi = torch.tensor([cx + sx / 2, cy + sy / 2, -1.7 + sz], device=DEV) * inv
            s = torch.minimum(lo, hi).amax(1)
            hit = (torch.maximum(lo, hi).amin(1) >= s.clamp(min=0)) & (s > 0)
            t = torch.where(hit & (s < t), s, t)
        sector = (torch.atan2(d[:, 1], d[:, 0]) % (2 * math.pi) / (2 * math.pi) * 24).long() % 24
        wall = torch.tensor(rng.uniform(40.0, 48.0, 24), dtype=torch.float32, device=DEV)[sector]
        top = torch.tensor(rng.uniform(4.0, 20.0, 24), dtype=torch.float32, device=DEV)[sector]
        s = wall / flat.sqrt()
        t = torch.where((s * d[:, 2] <= top - 1.7) & (s < t), s, t)
        keep = torch.isfinite(t) & (t <= 50.0) & (_rand(gen, len(t)) >= 0.1)
        t = t + 0.02 * torch.randn(t.shape, generator=gen, device=DEV)
        pts = (d * t[:, None])[keep]
        if thinned:
            pts = pts[_first_of_voxel(pts, voxel)]
        if len(pts) >= n:
            break
        azimuths *= 2
    centre = pts[int(rng.integers(len(pts)))]
    near = ((pts - centre) ** 2).sum(1).sort(stable=True).indices[:n]
    return pts[near.sort().values].contiguous()


def _points(case, seed):
    """(xyz f32 [n,3], cumulative cloud ends int64 [clouds]) on the GPU."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    clouds, n = case["clouds"], case["n"]
    share = np.exp(rng.uniform(0.0, math.log(10.0), clouds))
    counts = np.maximum(1, (n * share / share.sum())).astype(np.int64)
    counts[-1] += n - counts.sum()
    voxel = case.get("voxel", 0.04)
    out = []
    for i, count in enumerate(counts.tolist()):
        scene = case["scene"]
        if scene == "mixed":
            scene = "thinned" if i % 2 else "room"
        if scene == "cube":
            out.append(_cube(gen, count, voxel))
        elif scene == "room":
            out.append(_room(gen, rng, count, voxel))
        else:
            out.append(_scan(gen, rng, count, voxel, scene == "thinned"))
    ends = torch.tensor(np.cumsum(counts), dtype=torch.int64, device=DEV)
    return torch.cat(out).contiguous(), ends, gen


def _cloud_ids(ends):
    counts = torch.diff(ends, prepend=ends.new_zeros(1))
    return torch.repeat_interleave(torch.arange(len(ends), device=ends.device), counts)


def _cells(xyz, voxel):
    """floor(xyz / voxel) as a CUDA tensor divided by a number gives it."""
    inv = float(np.float32(1.0) / np.float32(voxel))
    return torch.floor(xyz * inv).long()


def _ball_voxel(case):
    return case["radius"] / 4


# -------------------------------------------------------------------- cases

def prepare(case, seed):
    if case["kind"] == "hierarchy":
        # level sizes are output shapes, so every seed has one geometry: the scan
        # begun at another point of its order, with x and y swapped or not
        xyz, ends, gen = _points(case, 0)
        xyz = xyz.roll(seed * 7919 % case["n"] + 1, 0)
        if seed % 2:
            xyz = xyz[:, [1, 0, 2]].contiguous()
    else:
        xyz, ends, gen = _points(case, seed)
    kind, n, k = case["kind"], case["n"], case["k"]
    st = {"case": case, "xyz": xyz, "ends": ends}
    if kind in ("grid", "selected", "adaptive"):
        st["grid"] = _cells(xyz, case["voxel"])
        st["batch"] = _cloud_ids(ends)
    if kind == "grid" or kind == "selected":
        st["knn"] = fk.FlashKNN(num_nbr=k, num_down=case["num_down"])
    if kind == "selected":
        st["sel"] = torch.arange(0, n, case["stride"], device=DEV)
    elif kind == "general":
        # the coarse level: a random subset of every cloud, as a strided encoder keeps
        keep = torch.arange(n, device=DEV) % case["stride"] == 0
        keep[ends - 1] = True
        ids = _cloud_ids(ends)
        st["coarse"] = xyz[keep].contiguous()
        st["coarse_ends"] = torch.bincount(ids[keep], minlength=len(ends)).cumsum(0)
    elif kind == "back":
        st["knn"] = fk.FlashKNN(num_nbr=k)
        ids = _cloud_ids(ends)
        st["batch"] = ids
        # clouds apart from one another, so one voxel never mixes two of them
        apart = xyz.double() + ids[:, None] * xyz.new_tensor([1e3, 0.0, 0.0])
        st["sel"] = _first_of_voxel(apart, case["size"])
    elif kind == "adaptive":
        st["knn"] = fk.AdaptiveNeighborhoodFlashKNN(num_nbr=k)
    elif kind == "group":
        st["feat"] = torch.randn((n, case["c"]), generator=gen, device=DEV).requires_grad_(True)
        width = case["c"] + (3 if case["with_xyz"] else 0)
        st["grad"] = torch.randn((n, k, width), generator=gen, device=DEV)
        if case["with_xyz"]:
            st["xyz"].requires_grad_(True)
    if kind == "self" and case["train"]:
        st["xyz"].requires_grad_(True)
        st["grad"] = torch.randn((n, k), generator=gen, device=DEV)
    return st


def run(st):
    case = st["case"]
    kind, k, xyz = case["kind"], case["k"], st["xyz"]
    if kind == "self":
        idx, dist = fk.knn_query(k, xyz, st["ends"], voxel_size=case["voxel"],
                                 num_down=case["num_down"])
        if not case["train"]:
            return idx, dist
        (grad,) = torch.autograd.grad(dist, xyz, st["grad"])
        return idx, dist.detach(), grad
    if kind == "grid":
        return st["knn"].query(st["grid"], st["batch"], xyz)
    if kind == "selected":
        return st["knn"].selected_query(xyz, st["grid"], st["sel"], st["batch"])
    if kind == "general":
        return fk.knn_query(k, st["coarse"], st["coarse_ends"], xyz, st["ends"],
                            voxel_size=case["voxel"] * 2, num_down=case["num_down"])
    if kind == "ball":
        return fk.ball_query(k, case["radius"], 0.0, xyz, st["ends"])
    if kind == "back":
        return st["knn"].back_query(xyz, st["sel"], 2 * case["size"], case["size"], st["batch"])
    if kind == "adaptive":
        return st["knn"].query(st["grid"], st["batch"], xyz)
    if kind == "hierarchy":
        return build_flash_hierarchy(xyz, ks=(k,) * 4)
    out, idx = fk.knn_query_and_group(st["feat"], xyz, st["ends"], nsample=k,
                                      with_xyz=case["with_xyz"], voxel_size=case["voxel"],
                                      num_down=case["num_down"])
    wrt = [st["feat"], xyz] if case["with_xyz"] else [st["feat"]]
    return (out.detach(), idx) + tuple(torch.autograd.grad(out, wrt, st["grad"]))


def work(case):
    """Inputs read once and outputs written once; 8 operations for every distance returned."""
    kind, n, k = case["kind"], case["n"], case["k"]
    flops = 8 * n * k
    if kind == "self":
        total = n * (12 + 8 * k) + (n * (12 + 4 * k) if case["train"] else 0)
    elif kind == "grid":
        total = n * (12 + 24 + 8 + 8 * k)
    elif kind == "selected":
        m = -(-n // case["stride"])
        total, flops = n * (12 + 24 + 8) + m * (8 + 8 * k), 8 * m * k
    elif kind == "general":
        total = n * 12 + n // case["stride"] * 12 + n * 8 * k
    elif kind == "ball":
        total = n * (12 + 8 * k)
    elif kind == "back":
        total = n * (12 + 8) + n * (8 if k == 1 else 12 * k)
    elif kind == "adaptive":
        total = n * (12 + 24 + 8 + 8 * k)
    elif kind == "hierarchy":
        total = n * (12 + 8 * k + 3 * 8)
    else:
        width = case["c"] + (3 if case["with_xyz"] else 0)
        total = n * (12 + 4 * case["c"]) + n * k * 4 * width * 2 + n * (4 * k + 4 * width)
    return {"bytes": float(total), "flops": float(flops)}


# -------------------------------------------------------------------- exact

def _neighbours(sup, sup_cloud, qry, qry_cloud, k, voxel, num_down, cut_r2=math.inf):
    """Row numbers [m,k] of the k nearest support points (-1: none) among the
    27 parent cells around each query: ascending by the FP32 squared distance,
    then by row number."""
    both = torch.cat([_cells(sup, voxel), _cells(qry, voxel)]) >> num_down
    lo = both.min(0).values - 1
    ext = both.max(0).values - lo + 2

    def key(cell, cloud):
        c = cell - lo
        return ((cloud * ext[0] + c[:, 0]) * ext[1] + c[:, 1]) * ext[2] + c[:, 2]

    order = key(both[: len(sup)], sup_cloud).sort(stable=True)
    steps = torch.tensor([(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)],
                         device=sup.device)
    shift = (steps[:, 0] * ext[1] + steps[:, 1]) * ext[2] + steps[:, 2]
    around = key(both[len(sup):], qry_cloud)[:, None] + shift
    start = torch.searchsorted(order.values, around)
    count = torch.searchsorted(order.values, around, right=True) - start
    total = count.sum(1)
    out = torch.full((len(qry), k), -1, dtype=torch.int64, device=sup.device)
    rows = total.sort().indices
    sizes = total[rows].cumsum(0)
    none = torch.iinfo(torch.int64).max
    a = 0
    while a < len(rows):
        done = int(sizes[a - 1]) if a else 0
        b = int(torch.searchsorted(sizes, done + (1 << 25), right=True))
        b = min(max(b, a + 1), len(rows))
        while b > a + 1 and (b - a) * int(total[rows[b - 1]]) > 1 << 26:
            b = a + (b - a) // 2
        r = rows[a:b]
        a = b
        width = int(total[r[-1]])
        if not width:
            continue
        cnt, st = count[r], start[r]
        before = cnt.cumsum(1) - cnt
        pair_row = torch.repeat_interleave(torch.arange(len(r), device=r.device), cnt.sum(1))
        run_no = torch.repeat_interleave(torch.arange(cnt.numel(), device=r.device), cnt.flatten())
        at = torch.arange(len(run_no), device=r.device)
        at = at - (cnt.flatten().cumsum(0) - cnt.flatten())[run_no]
        cand = order.indices[st.flatten()[run_no] + at]
        dif = (sup[cand] - qry[r][pair_row]).double()
        dy = (dif[:, 1] * dif[:, 1]).float().double()
        d = (dif[:, 0] * dif[:, 0] + dy).float().double()
        d = (dif[:, 2] * dif[:, 2] + d).float()
        packed = (d.view(torch.int32).long() << 32) | cand
        packed[~(d < cut_r2)] = none
        table = torch.full((len(r), max(width, k)), none, dtype=torch.int64, device=r.device)
        table[pair_row, before.flatten()[run_no] + at] = packed
        best = table.topk(k, 1, largest=False, sorted=True).values
        out[r] = torch.where(best == none, -1, best & 0xFFFFFFFF)
    return out


def _sq_dist(sup, qry, nbr, none):
    d = ((sup.double()[nbr.clamp(min=0)] - qry.double()[:, None]) ** 2).sum(-1)
    return torch.where(nbr < 0, none, d)


def exact(case, seed):
    kind, k = case["kind"], case["k"]
    if kind not in ("self", "general", "ball", "group"):
        return None
    st = prepare(case, seed)
    xyz, ends = st["xyz"].detach(), st["ends"]
    ids = _cloud_ids(ends)
    if kind == "general":
        sup, sup_ends = st["coarse"], st["coarse_ends"]
        nbr = _neighbours(sup, _cloud_ids(sup_ends), xyz, ids, k, case["voxel"] * 2,
                          case["num_down"])
        return None, _sq_dist(sup, xyz, nbr, math.inf)
    if kind == "ball":
        r2 = float(np.float32(case["radius"]) * np.float32(case["radius"]))
        nbr = _neighbours(xyz, ids, xyz, ids, k, _ball_voxel(case), 2, r2)
        return None, _sq_dist(xyz, xyz, nbr, 1e10).sqrt()
    nbr = _neighbours(xyz, ids, xyz, ids, k, case["voxel"], case["num_down"])
    x = xyz.double()
    if kind == "self":
        dist = _sq_dist(xyz, xyz, nbr, math.inf)
        if not case["train"]:
            return None, dist
        g = torch.where(nbr < 0, 0.0, 2 * st["grad"].double())
        term = g[..., None] * (x[:, None] - x[nbr.clamp(min=0)])
        grad = term.sum(1)
        grad.index_add_(0, nbr.clamp(min=0).flatten(), -term.reshape(-1, 3))
        return None, dist, grad
    # a self query pads with the point's own index
    nbr = torch.where(nbr < 0, torch.arange(len(xyz), device=DEV)[:, None], nbr)
    feat, grad = st["feat"].detach().double(), st["grad"].double()
    flat = nbr.flatten()
    if not case["with_xyz"]:
        g = torch.zeros_like(feat).index_add_(0, flat, grad.reshape(len(flat), -1))
        return feat[nbr], None, g
    out = torch.cat([x[nbr] - x[:, None], feat[nbr]], -1)
    rows = grad.reshape(len(flat), -1)
    g = torch.zeros_like(feat).index_add_(0, flat, rows[:, 3:])
    gx = torch.zeros_like(x).index_add_(0, flat, rows[:, :3]) - grad[..., :3].sum(1)
    return out, None, g, gx
