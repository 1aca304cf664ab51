"""Performance cases: the calls a program built on this package makes per frame, per batch step and per session.

Every case is a dict of plain values; `prepare` builds what the calling program already holds (depth frames, volumes,
pyramids, a tracker), `run` is one pass through the package's entry points, `work` counts what that pass cannot do
without, and `exact` restates the computed numbers in 64-bit torch. Inputs are rendered here with torch: a room of
walls, spheres and boxes seen by a moving depth camera, with the axial noise and the dropout of a real sensor.

The sizes are those of the package's own configurations (CONFIGS, c4_configs), and `draw` spreads over the same ranges.
"""
import math

import numpy as np
import torch

import openfusion_b200 as of
from openfusion_b200 import learned

DEV = "cuda"


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # the smallest call: one frame of the smallest camera that the batched workload has (launches and latency)
        {"name": "preprocess_160x120", "kind": "preprocess", "w": 160, "h": 120, "sigma": 4.5, "levels": 3},
        # depth pre-processing of one frame at the full-size camera
        {"name": "preprocess_640x480", "kind": "preprocess", "w": 640, "h": 480, "sigma": 4.5, "levels": 3},
        # a camera's own clean-up chain: median, gradient, two averages (what the GIP camera applies to each frame)
        {"name": "filters_640x480", "kind": "filters", "w": 640, "h": 480, "chain": "gip"},
        # fusion of one frame into the small volume
        {"name": "integrate_320x240_128", "kind": "integrate", "w": 320, "h": 240, "n": 128, "size": 2000.0,
         "trunc": 60.0, "storage": "i16"},
        # fusion of one frame into the full-size volume
        {"name": "integrate_640x480_512", "kind": "integrate", "w": 640, "h": 480, "n": 512, "size": 3000.0,
         "trunc": 30.0, "storage": "i16"},
        # surface prediction from the full-size volume
        {"name": "raycast_640x480_512", "kind": "raycast", "w": 640, "h": 480, "n": 512, "size": 3000.0,
         "trunc": 30.0, "storage": "i16", "tile": 5},
        # the high-resolution half-float volume of the precision study: fusion and surface prediction
        {"name": "fuse_640x480_1024_f16", "kind": "fuse", "w": 640, "h": 480, "n": 1024, "size": 4000.0,
         "trunc": 30.0, "storage": "f16", "tile": 0},
        # tracking of one frame against the model, three levels of 10/5/4 iterations
        {"name": "icp_640x480", "kind": "icp", "w": 640, "h": 480},
        # the whole frame loop: a frame in pinned host memory in, its pose out
        {"name": "track_640x480_512", "kind": "track", "w": 640, "h": 480, "n": 512, "size": 3000.0, "trunc": 30.0,
         "storage": "i16", "tile": 5},
        # many independent cameras tracked and fused together, one step of all of them
        {"name": "batch_16_streams", "kind": "batch", "streams": 16, "mix": 4000},
        # one training step of the warm-start network at the trainer's batch size
        {"name": "train_256", "kind": "train", "batch": 256},
        # the surface mesh of a finished reconstruction
        {"name": "mesh_512", "kind": "mesh", "w": 640, "h": 480, "n": 512, "size": 3000.0, "trunc": 30.0,
         "storage": "i16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["preprocess", "preprocess", "filters", "integrate", "integrate", "raycast", "raycast", "icp",
                       "icp", "track", "track", "batch", "train", "mesh"])
    w = _log_int(rng, 120, 640)
    h = max(90, min(480, int(w * rng.uniform(0.6, 0.9))))
    c = {"kind": kind}
    if kind == "train":
        c["batch"] = _log_int(rng, 17, 256)
        return c
    if kind == "batch":
        c.update(streams=rng.randint(2, 16), mix=rng.randint(1, 9999))
        return c
    c.update(w=w, h=h)
    if kind == "preprocess":
        c.update(sigma=rng.choice([2.0, 3.0, 4.0, 4.5, 5.0, 5.5]), levels=rng.randint(1, 4))
    if kind == "filters":
        c.update(chain=rng.choice(["gip", "softkinetic", "median"]))
    if kind in ("integrate", "raycast", "track", "mesh"):
        n = 8 * _log_int(rng, 12, 64)
        size = round(rng.uniform(2000.0, 3000.0), 1)
        c.update(n=n, size=size, trunc=round(max(30.0, 4.0 * size / n), 2), storage=rng.choice(["i16", "i16", "f16"]))
    if kind in ("raycast", "track"):
        c["tile"] = rng.choice([0, 1, 5, 5, 6])
    return c


# ------------------------------------------------------------ the scene --

def _config(c):
    """The package's configuration of a case (a 640-pixel camera has 525 px focal length)."""
    w, h = c.get("w", 640), c.get("h", 480)
    f = 525.0 * w / 640.0
    return of.Config(
        name="case", width=w, height=h, fx=f, fy=f, cx=(w - 1) / 2.0, cy=(h - 1) / 2.0, resolution=c.get("n", 512),
        size_mm=c.get("size", 3000.0), trunc_mm=c.get("trunc", 30.0), storage=c.get("storage", "i16"),
        sigma_space_px=c.get("sigma", 4.5), levels=c.get("levels", 3), ray_tile=c.get("tile", 0))


class _Room:
    """Floor, three walls and 20 spheres and boxes in a cube of edge S mm, and a smooth path around them."""

    def __init__(self, seed, S):
        r = np.random.default_rng([seed, 11])
        self.S, self.floor = S, -0.37 * S
        n = 10
        rad, half = r.uniform(100.0, 400.0, n), r.uniform(80.0, 300.0, (n, 3))

        def centre(below, behind):
            return np.stack([r.uniform(-0.33 * S, 0.33 * S, n), r.uniform(self.floor + below, 0.12 * S),
                             r.uniform(-0.42 * S + behind, 0.02 * S)], 1)

        self.sphere_c, self.sphere_r = centre(rad, rad), rad
        self.box_c, self.box_h, self.box_yaw = centre(half[:, 1], half[:, 2]), half, r.uniform(0.0, 0.5 * np.pi, n)
        self.tgt = np.array([0.0, -0.05 * S, -0.12 * S]) + r.uniform(-0.02, 0.02, 3) * S
        self.phase, self.th0 = r.uniform(0.0, 2.0 * np.pi, 2), r.uniform(-0.1, 0.1)

    def pose(self, k):
        """Camera-to-world pose k of the path (a few mm and a fraction of a degree from pose k - 1)."""
        th = self.th0 + 0.314 * (math.sin(2 * math.pi * k / 300 + self.phase[0]) - math.sin(self.phase[0]))
        y = (0.05 + 0.02 * math.sin(4 * math.pi * k / 300 + self.phase[1])) * self.S
        eye = self.tgt + np.array([0.43 * self.S * math.sin(th), y, 0.43 * self.S * math.cos(th)])
        z = eye - self.tgt
        z /= np.linalg.norm(z)
        x = np.cross([0.0, 1.0, 0.0], z)
        x /= np.linalg.norm(x)
        P = np.eye(4)
        P[:3, 0], P[:3, 1], P[:3, 2], P[:3, 3] = x, np.cross(z, x), z, eye
        return P

    def depth(self, cfg, P, gen=None, dropout=0.02):
        """Depth image in mm: exact (float64) without a generator, else what a sensor gives (int16)."""
        v, u = torch.meshgrid(torch.arange(cfg.height, device=DEV, dtype=torch.float64),
                              torch.arange(cfg.width, device=DEV, dtype=torch.float64), indexing="ij")
        dc = torch.stack([-(u - cfg.cx) / cfg.fx, -(v - cfg.cy) / cfg.fy, -torch.ones_like(u)], -1).reshape(-1, 3)
        Pt = torch.from_numpy(P).to(DEV)
        d, o = dc @ Pt[:3, :3].T, Pt[:3, 3]
        far = torch.tensor(1e9, device=DEV, dtype=torch.float64)
        best = torch.full((d.shape[0],), 1e9, device=DEV, dtype=torch.float64)

        def nearer(t):
            return torch.minimum(best, torch.where(t > 1e-6, t, far))

        for axis, at in ((1, self.floor), (2, -0.45 * self.S), (0, -0.45 * self.S), (0, 0.45 * self.S)):
            best = nearer((at - o[axis]) / d[:, axis])
        a = (d * d).sum(1)
        for c, r in zip(self.sphere_c, self.sphere_r):
            oc = o - torch.from_numpy(c).to(DEV)
            b = d @ oc
            disc = b * b - a * (oc @ oc - r * r)
            t = (-b - disc.clamp_min(0).sqrt()) / a
            best = torch.where(disc >= 0, nearer(t), best)
        for c, half, yaw in zip(self.box_c, self.box_h, self.box_yaw):
            R = torch.tensor([[math.cos(yaw), 0.0, -math.sin(yaw)], [0.0, 1.0, 0.0],
                              [math.sin(yaw), 0.0, math.cos(yaw)]], device=DEV, dtype=torch.float64)
            lo, ld = R @ (o - torch.from_numpy(c).to(DEV)), d @ R.T
            hh = torch.from_numpy(half).to(DEV)
            t0, t1 = (-hh - lo) / ld, (hh - lo) / ld
            tn, tf = torch.minimum(t0, t1).amax(1), torch.maximum(t0, t1).amin(1)
            best = torch.where(tn <= tf, nearer(tn), best)
        best = best.reshape(cfg.height, cfg.width)
        if gen is None:
            return best
        zm = best * 1e-3 - 0.4
        noisy = best + 1000.0 * (0.0012 + 0.0019 * zm * zm) * torch.randn(best.shape, device=DEV, dtype=torch.float64,
                                                                           generator=gen)
        kept = (best < 10000.0) & (torch.rand(best.shape, device=DEV, generator=gen) >= dropout)
        return torch.where(kept, (noisy + 0.5).floor().clamp(1, 20000), torch.zeros_like(best)).to(torch.int16)


def _sequence(cfg, seed, frames, size=None):
    """Room, poses [frames, 4, 4] and sensor frames of one recording."""
    room = _Room(seed, size or cfg.size_mm)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    poses = np.stack([room.pose(3 * k) for k in range(frames)])
    return room, poses, [room.depth(cfg, P, gen) for P in poses]


def _device_pose(P):
    return torch.tensor(np.ascontiguousarray(P).reshape(16), dtype=torch.float64, device=DEV)


def _views(cfg, pyr, depth):
    """The levels of a pyramid buffer: (depth), vertices and normals."""
    out = []
    for l in range(cfg.levels):
        if depth:
            out.append(of.unpack_depth(cfg, pyr, l))
        out += list(of.unpack_points(cfg, pyr, l))
    return out


class _Device:
    """A device range as the CUDA array interface describes it: a tracker's own buffer, read in place. A tensor made
    from it keeps it, and so the tracker (`owner`), alive."""

    def __init__(self, owner, ptr, n, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (int(ptr), False), "version": 3}


def _state_of(cfg, owner, buffers):
    """Model maps and voxel words that a tracker holds, read in place."""
    pyr = torch.as_tensor(_Device(owner, buffers.model, int(of.pyramid_layout(cfg).total_bytes), "|u1"), device=DEV)
    vol = torch.as_tensor(_Device(owner, buffers.volume, of.volume_bytes(cfg) // 4, "<i4"), device=DEV)
    return _views(cfg, pyr, False) + [vol]


def _to_and_fro(k, n):
    """0, 1, .., n - 1, n - 2, .., 0, 1, ..: a camera that goes back and forth over its path."""
    k %= 2 * (n - 1)
    return k if k < n else 2 * (n - 1) - k


# ---------------------------------------------------------------- prepare --

def prepare(case, seed):
    kind, cfg = case["kind"], _config(case)
    s = {"case": case, "cfg": cfg, "k": 0}
    if kind in ("preprocess", "filters"):
        _, _, s["depth"] = _sequence(cfg, seed, 4)
        if kind == "preprocess":
            s["frame"] = of.new_pyramid(cfg)
            s["out"] = _views(cfg, s["frame"], True)
        else:
            steps = {"gip": ("median5", "gradient", "average"), "softkinetic": ("undistort", "median5", "average"),
                     "median": ("median5",)}[case["chain"]]
            more = {"gip": {"average_passes": 2}, "softkinetic": {"k1": -0.06, "k2": 0.01, "p1": 5e-4, "p2": -5e-4},
                    "median": {}}[case["chain"]]
            s.update(steps=steps, more=more)
    elif kind in ("integrate", "raycast", "fuse", "mesh"):
        _, poses, s["depth"] = _sequence(cfg, seed, 12)
        s["pose"] = [_device_pose(P) for P in poses]
        s["lam"], s["scratch"], s["vol"] = of.lambda_table(cfg), of.integrate_scratch(cfg), of.new_volume(cfg)
        for k in range(8):
            of.integrate(cfg, s["vol"], s["depth"][k], s["pose"][k], s["lam"], s["scratch"])
        if kind in ("raycast", "fuse"):
            s["model"] = of.new_pyramid(cfg)
            s["out"] = _views(cfg, s["model"], False)
        if kind == "mesh":  # the program's own buffers for a mesh of up to 2^21 triangles
            s["tris"] = torch.zeros(1 << 21, 9, device=DEV)
            s["ids"], s["order"] = (torch.zeros(1 << 21, dtype=torch.int64, device=DEV) for _ in range(2))
        s["k"] = 8
    elif kind == "icp":
        room, poses, depth = _sequence(cfg, seed, 6)
        s["frames"] = [_pyramid(cfg, _smooth(cfg, d), None) for d in depth[1:]]
        s["model"] = _pyramid(cfg, room.depth(cfg, poses[0]), poses[0])
        s["ws"], s["pose"] = of.icp_workspace(cfg), _device_pose(poses[0])
    elif kind == "track":
        _, poses, depth = _sequence(cfg, seed, 24)
        s["depth"] = [d.cpu().pin_memory() for d in depth]
        s["tracker"] = of.Tracker(cfg, poses[0])
        s["pose"] = torch.zeros(16, dtype=torch.float64).pin_memory()
        s["out"] = [s["pose"]] + _state_of(cfg, s["tracker"], s["tracker"].buffers())
        for k in range(4):
            s["tracker"].process(s["depth"][k])
        s["k"] = 4
    elif kind == "batch":
        cfgs = of.c4_configs(case["streams"], case["mix"])
        seqs = [_sequence(c, seed + 101 * i, 8) for i, c in enumerate(cfgs)]
        s["depth"] = [[q[2][k] for q in seqs] for k in range(8)]
        s["batch"] = of.Batch(cfgs, [q[1][0] for q in seqs], tuning=(5, 0, 0))
        s["out"] = [_state_of(c, s["batch"], s["batch"].buffers(i))[-1] for i, c in enumerate(cfgs)]
        for k in range(3):
            s["batch"].process(s["depth"][k])
        s["k"] = 3
    elif kind == "train":
        b = case["batch"]
        s["x"], s["y"] = _pairs(seed, b)
        s["net"] = learned.WarmStartNet(DEV, weights=learned.load_weights())
    return s


def _smooth(cfg, depth):
    """Filtered depth as tracking sees it: 5x5 means of the valid neighbours within 60 mm."""
    d = depth.to(torch.float64)
    p = torch.nn.functional.pad(d, (2, 2, 2, 2))
    total, count = torch.zeros_like(d), torch.zeros_like(d)
    for j in range(5):
        for i in range(5):
            q = p[j:j + cfg.height, i:i + cfg.width]
            near = (q > 0) & ((q - d).abs() < 60.0)
            total, count = total + torch.where(near, q, 0.0), count + near
    return torch.where((d > 0) & (count > 0), total / count.clamp_min(1), 0.0)


def _maps(cfg, depth, level):
    """Camera-space vertices, normals and validity of a float64 depth image of one level."""
    cam = of.level_camera(cfg, level)
    h, w = depth.shape
    v, u = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float64),
                          torch.arange(w, device=DEV, dtype=torch.float64), indexing="ij")
    vtx = torch.stack([-depth * (u - cam.cx) / cam.fx, -depth * (v - cam.cy) / cam.fy, -depth], -1)
    n = torch.zeros_like(vtx)
    ok = torch.zeros_like(depth, dtype=torch.bool)
    a, b = vtx[:-1, 1:] - vtx[:-1, :-1], vtx[1:, :-1] - vtx[:-1, :-1]
    c = torch.linalg.cross(a, b)
    length = c.norm(dim=-1)
    good = (depth[:-1, :-1] > 0) & (depth[:-1, 1:] > 0) & (depth[1:, :-1] > 0) & (length > 0)
    n[:-1, :-1] = torch.where(good[..., None], c / length.clamp_min(1e-300)[..., None], torch.zeros_like(c))
    ok[:-1, :-1] = good
    return torch.where((depth > 0)[..., None], vtx, torch.zeros_like(vtx)), n, depth > 0, ok


def _half(cfg, d):
    """Next pyramid level: mean of the 2x2 block's valid depths within three range sigmas of its first one."""
    h, w = d.shape
    p = torch.nn.functional.pad(d, (0, w & 1, 0, h & 1))
    q = torch.stack([p[0::2, 0::2], p[0::2, 1::2], p[1::2, 0::2], p[1::2, 1::2]])
    first = torch.zeros_like(q[0])
    for k in (3, 2, 1, 0):
        first = torch.where(q[k] > 0, q[k], first)
    near = (q > 0) & ((q - first).abs() <= 3.0 * cfg.sigma_range_mm)
    return torch.where(near.any(0), torch.where(near, q, 0.0).sum(0) / near.sum(0).clamp_min(1), 0.0)


def _pyramid(cfg, depth, pose):
    """A pyramid buffer of maps: camera space of a depth image, or a model's world-space maps at `pose`."""
    buf = of.new_pyramid(cfg)
    top = None
    for l in range(cfg.levels):
        d = depth if l == 0 else _half(cfg, d)
        of.unpack_depth(cfg, buf, l).copy_(d)
        v, n, vok, nok = _maps(cfg, d, l)
        if pose is not None:
            if l == 0:
                T = torch.from_numpy(pose).to(DEV)
                top = (v @ T[:3, :3].T + T[:3, 3], n @ T[:3, :3].T, vok, nok)
            v, n, vok, nok = (x[::1 << l, ::1 << l] for x in top)
        V, Nn = of.unpack_points(cfg, buf, l)
        V[..., :3].copy_(torch.where(vok[..., None], v, torch.zeros_like(v)))
        V[..., 3].copy_(vok)
        Nn[..., :3].copy_(torch.where(nok[..., None], n, torch.zeros_like(n)))
        Nn[..., 3].copy_(nok)
    return buf


def _pairs(seed, b):
    """b network inputs (BF16 bits: centred depth and difference of consecutive frames) and their motions."""
    cfg = _config({"w": 80, "h": 60, "size": 3000.0})
    room, gen = _Room(seed, 3000.0), torch.Generator(device=DEV).manual_seed(seed)
    r = np.random.default_rng([seed, 7])
    poses = []
    for k in range(33):
        J = np.eye(4)
        J[:3, :3] = learned.exp_so3(r.uniform(-0.025, 0.025, 3))
        J[:3, 3] = r.uniform(-30.0, 30.0, 3)
        poses.append(room.pose(9 * k) @ J)
    z = torch.stack([room.depth(cfg, P, gen, dropout=0.0) for P in poses]).to(torch.float32) * 1e-3
    i = torch.from_numpy(r.integers(0, 32, b)).to(DEV)
    step = torch.from_numpy(np.where(r.random(b) < 0.5, 1, -1)).to(DEV)
    p, q = torch.where(step > 0, i, i + 1), torch.where(step > 0, i + 1, i)
    prev, cur = z[p], z[q]
    prev = prev + 2e-3 * torch.randn(prev.shape, device=DEV, generator=gen)
    x = torch.stack([prev - prev.mean((1, 2), keepdim=True), cur - prev], 1).to(torch.bfloat16)
    y = np.stack([learned.motion_target(poses[a], poses[c]) for a, c in zip(p.tolist(), q.tolist())])
    return x.reshape(b, -1).view(torch.int16), torch.from_numpy(y.astype(np.float32)).to(DEV)


# -------------------------------------------------------------------- run --

def run(s):
    kind, cfg, k = s["case"]["kind"], s["cfg"], s["k"]
    s["k"] = k + 1
    if kind == "preprocess":
        of.preprocess(cfg, s["depth"][k % 4], s["frame"])
        return s["out"]
    if kind == "filters":
        return of.depth_filter(cfg, s["depth"][k % 4], s["steps"], **s["more"])
    if kind == "integrate":
        i = _to_and_fro(k, 12)
        of.integrate(cfg, s["vol"], s["depth"][i], s["pose"][i], s["lam"], s["scratch"])
        return s["vol"]
    if kind == "raycast":
        of.raycast(cfg, s["vol"], s["pose"][_to_and_fro(k, 12)], s["model"])
        return s["out"]
    if kind == "fuse":
        i = _to_and_fro(k, 12)
        of.integrate(cfg, s["vol"], s["depth"][i], s["pose"][i], s["lam"], s["scratch"])
        of.raycast(cfg, s["vol"], s["pose"][i], s["model"])
        return s["out"] + [s["vol"]]
    if kind == "icp":
        # the pose found for a frame is where the next frame's search starts
        of.icp_track(cfg, s["frames"][_to_and_fro(k, 5)], s["model"], s["pose"], s["ws"])
        return s["pose"]
    if kind == "track":
        s["tracker"].process(s["depth"][_to_and_fro(k, 24)])
        s["tracker"].pose(out=s["pose"])
        return s["out"]
    if kind == "batch":
        s["batch"].process(s["depth"][_to_and_fro(k, 8)])
        return [s["batch"].poses()] + s["out"]
    if kind == "train":
        net = s["net"]
        loss = net.train_step(s["x"], s["y"], 1e-4)
        return [loss, net.grad, net.master, net.params.view(torch.bfloat16)]
    # the triangles come in no order: sorted by their ids, two meshes can be compared
    tris, ids = of.extract_mesh(cfg, s["vol"], max_triangles=1 << 21, with_ids=True)
    n = ids.shape[0]
    torch.sort(ids, out=(s["ids"][:n], s["order"][:n]))
    torch.index_select(tris.view(n, 9), 0, s["order"][:n], out=s["tris"][:n])
    return [s["tris"], s["ids"], n]


# ------------------------------------------------------------------- work --

#: multiply-adds of the network's layers for one pair, forward
_NET_MACS = 1200 * 16 * 50 + 300 * 32 * 144 + 80 * 64 * 288 + 20 * 128 * 576 + 2560 * 160 + 160 * 6
_NET_ACTS = 9600 + 19200 + 9600 + 5120 + 2560 + 160


def work(case):
    kind, cfg = case["kind"], _config(case)
    px = cfg.width * cfg.height
    pyr = sum(-(-cfg.width // 2 ** l) * -(-cfg.height // 2 ** l) for l in range(cfg.levels))
    iters = sum(i * (-(-cfg.width // 2 ** l) * -(-cfg.height // 2 ** l)) for l, i in enumerate(cfg.iters))
    band = int(0.02 * cfg.resolution ** 3)   # voxels that one frame changes: near the surface and not yet saturated
    # a ray reads the 8 voxels of its surface cell and the 32 of its normal
    fuse, cast = 2 * px + 8 * band, px * 40 * 2 + 32 * pyr
    if kind == "preprocess":
        return {"bytes": 2 * px + 36 * pyr, "flops": 8 * px * (2 * cfg.radius() + 1) ** 2}
    if kind == "filters":
        return {"bytes": 4 * px, "flops": 0}
    if kind == "integrate":
        return {"bytes": fuse, "flops": 0}
    if kind == "raycast":
        return {"bytes": cast, "flops": 0}
    if kind == "fuse":
        return {"bytes": fuse + cast, "flops": 0}
    if kind == "icp":
        return {"bytes": 64 * pyr, "flops": 110 * iters}
    if kind == "track":
        return {"bytes": fuse + cast + 2 * px + 36 * pyr + 64 * pyr,
                "flops": 8 * px * (2 * cfg.radius() + 1) ** 2 + 110 * iters}
    if kind == "batch":
        each = [work({"kind": "track", "w": c.width, "h": c.height, "n": c.resolution})
                for c in of.c4_configs(case["streams"], case["mix"])]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    if kind == "train":
        b, n = case["batch"], 508534
        return {"bytes": b * (2 * 9600 + 24) + n * (2 + 4 * 7), "flops": 6 * _NET_MACS * b}
    return {"bytes": 4 * band + 44 * band // 4, "flops": 0}


# ------------------------------------------------------------------ exact --

def exact(case, seed):
    kind = case["kind"]
    if kind == "preprocess":
        s = prepare(case, seed)
        return _exact_preprocess(s["cfg"], s["depth"][0])
    if kind in ("raycast", "fuse"):
        s = prepare(case, seed)
        cfg = s["cfg"]
        if kind == "fuse":  # the volume that the surface is read from holds whole numbers: fused, then read
            of.integrate(cfg, s["vol"], s["depth"][8], s["pose"][8], s["lam"], s["scratch"])
        return _exact_raycast(cfg, s["vol"], s["pose"][8].cpu().numpy().reshape(4, 4)) + [None] * (kind == "fuse")
    if kind == "icp":
        s = prepare(case, seed)
        return _exact_icp(s["cfg"], s["frames"][0], s["model"], s["pose"].cpu().numpy().reshape(4, 4))
    if kind == "train":
        s = prepare(case, seed)
        return _exact_train(s["net"], s["x"], s["y"], 1e-4)
    return None


def _exact_preprocess(cfg, depth):
    R, (h, w) = cfg.radius(), depth.shape
    d = depth.to(torch.float64)
    d = torch.where((d > 0) & (d >= cfg.min_depth_mm) & (d <= cfg.max_depth_mm), d, 0.0)
    p = torch.nn.functional.pad(d, (R, R, R, R))
    total, weight = torch.zeros_like(d), torch.zeros_like(d)
    for j in range(-R, R + 1):
        for i in range(-R, R + 1):
            q = p[R + j:R + j + h, R + i:R + i + w]
            e = (i * i + j * j) / (2 * cfg.sigma_space_px ** 2) + (q - d) ** 2 / (2 * cfg.sigma_range_mm ** 2)
            k = torch.where(q > 0, torch.exp(-e), 0.0)
            total, weight = total + k * q, weight + k
    d = torch.where(d > 0, total / weight.clamp_min(1e-300), 0.0)
    out = []
    for l in range(cfg.levels):
        d = _half(cfg, d) if l else d
        v, n, vok, nok = _maps(cfg, d, l)
        out += [d, torch.cat([v, vok[..., None]], -1), torch.cat([n, nok[..., None]], -1)]
    return out


class _Field:
    """Trilinear tsdf of a volume buffer in float64."""

    def __init__(self, cfg, vol):
        n = cfg.resolution
        self.n, self.nb, self.vs, self.org = n, n // 8, cfg.size_mm / n, -0.5 * cfg.size_mm
        low = vol[:n ** 3].to(torch.int16)  # the low half of a word
        self.v = low.view(torch.float16) if cfg.storage == "f16" else low
        self.scale = 1.0 if cfg.storage == "f16" else 1.0 / 32767.0

    def at(self, i):
        """Values at integer coordinates [.., 3] (bricks of 8^3, x-major, z fastest)."""
        b, r = i >> 3, i & 7
        a = (((b[..., 0] * self.nb + b[..., 1]) * self.nb + b[..., 2]) << 9) | (r[..., 0] << 6) | (r[..., 1] << 3) | r[..., 2]
        return self.v[a].to(torch.float64) * self.scale

    def __call__(self, p):
        g = (p - self.org) / self.vs - 0.5
        i = g.floor().clamp(0, self.n - 2).to(torch.int64)
        f = g - i
        out = 0.0
        for c in range(8):
            o = torch.tensor([c >> 2, (c >> 1) & 1, c & 1], device=DEV)
            out = out + torch.where(o.bool(), f, 1.0 - f).prod(-1) * self.at(i + o)
        return out


def _exact_raycast(cfg, vol, P):
    field = _Field(cfg, vol)
    h, w, T = cfg.height, cfg.width, torch.from_numpy(P).to(DEV)
    v, u = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float64),
                          torch.arange(w, device=DEV, dtype=torch.float64), indexing="ij")
    dc = torch.stack([-(u - cfg.cx) / cfg.fx, -(v - cfg.cy) / cfg.fy, -torch.ones_like(u)], -1).reshape(-1, 3)
    lam = dc.norm(dim=1)
    d, o = (dc @ T[:3, :3].T) / lam[:, None], T[:3, 3]
    lo, hi = field.org + 0.5 * field.vs + 1e-3, -field.org - 0.5 * field.vs - 1e-3
    a, b = (lo - o) / d, (hi - o) / d
    t = torch.maximum(torch.minimum(a, b).amax(1), cfg.min_depth_mm * lam)
    end = torch.minimum(torch.maximum(a, b).amin(1), cfg.max_depth_mm * lam)
    step = cfg.min_step_vox * field.vs
    live = torch.nonzero(t < end)[:, 0]
    long_step = cfg.far_step_frac * cfg.trunc_mm
    prev = torch.ones_like(t)
    prev[live] = field(o + t[live, None] * d[live])
    ta, tb = torch.zeros_like(t), torch.zeros_like(t)
    hit = torch.zeros_like(t, dtype=torch.bool)
    while live.numel():
        tn = t[live] + (long_step * prev[live]).clamp_min(step)
        inside = tn <= end[live]
        live, tn = live[inside], tn[inside]
        f, g = prev[live], field(o + tn[:, None] * d[live])
        found, back = (f > 0) & (g <= 0), (f < 0) & (g > 0)
        ta[live[found]], tb[live[found]], hit[live[found]] = t[live[found]], tn[found], True
        t[live], prev[live] = tn, g
        live = live[~(found | back)]
    at = torch.nonzero(hit)[:, 0]
    ta, tb = ta[at], tb[at]
    for _ in range(int(long_step / step) + 1):  # the first crossing within a long step
        tm = ta + step
        up = field(o + tm[:, None] * d[at]) > 0
        long = tb - ta > 1.0001 * step
        ta, tb = torch.where(long & up, tm, ta), torch.where(long & ~up, tm, tb)
    for _ in range(40):
        tm = 0.5 * (ta + tb)
        up = field(o + tm[:, None] * d[at]) > 0
        ta, tb = torch.where(up, tm, ta), torch.where(up, tb, tm)
    p = o + ta[:, None] * d[at]
    vtx, nrm = torch.zeros(h * w, 4, device=DEV, dtype=torch.float64), torch.zeros(h * w, 4, device=DEV, dtype=torch.float64)
    vtx[at] = torch.cat([p, torch.ones_like(p[:, :1])], 1)
    ok = ((p - field.vs >= lo) & (p + field.vs <= hi)).all(1)
    e = torch.eye(3, device=DEV, dtype=torch.float64) * field.vs
    g = torch.stack([field((p + e[k]).clamp(lo, hi)) - field((p - e[k]).clamp(lo, hi)) for k in range(3)], 1)
    length = g.norm(dim=1)
    ok &= length > 0
    nrm[at] = torch.where(ok[:, None], torch.cat([g / length.clamp_min(1e-300)[:, None], torch.ones_like(p[:, :1])], 1), 0.0)
    vtx, nrm = vtx.reshape(h, w, 4), nrm.reshape(h, w, 4)
    return [x[::1 << l, ::1 << l] for l in range(cfg.levels) for x in (vtx, nrm)]


def _exact_icp(cfg, frame, model, P):
    P = torch.from_numpy(P).to(DEV)
    for l in range(cfg.levels - 1, -1, -1):
        cam = of.level_camera(cfg, l)
        sv, sn = (x.reshape(-1, 4).double() for x in of.unpack_points(cfg, model, l))
        fv, fn = (x.reshape(-1, 4).double() for x in of.unpack_points(cfg, frame, l))
        w, h = cam.width, cam.height
        keep = (sv[:, 3] != 0) & (sn[:, 3] != 0)
        sv, sn = sv[keep, :3], sn[keep, :3]
        for _ in range(cfg.iters[l]):
            R, t = P[:3, :3], P[:3, 3]
            c = (sv - t) @ R
            pu = (cam.fx * c[:, 0] / c[:, 2] + cam.cx + 0.5).floor()
            pv = (cam.fy * c[:, 1] / c[:, 2] + cam.cy + 0.5).floor()
            ok = (c[:, 2] < -1e-6) & (pu >= 0) & (pu < w) & (pv >= 0) & (pv < h)
            q = torch.where(ok, pv * w + pu, torch.zeros_like(pu)).long()
            d, n = fv[q, :3] @ R.T + t, fn[q, :3] @ R.T
            dot = (n * sn).sum(1)
            ok &= (fv[q, 3] != 0) & (fn[q, 3] != 0) & ((d - sv).norm(dim=1) < cfg.dist_thresh_mm)
            ok &= (dot > cfg.normal_thresh) & (dot < 1.0 + 1e-6)
            A = torch.cat([torch.linalg.cross(sn, d), sn], 1)[ok]
            b = (sn * (sv - d)).sum(1)[ok]
            x = torch.linalg.solve(A.T @ A, A.T @ b).cpu().numpy()
            al, be, ga = -x[:3]
            ca, sa, cb, sb, cg, sg = (math.cos(al), math.sin(al), math.cos(be), math.sin(be), math.cos(ga), math.sin(ga))
            D = np.array([[cg * cb, -sg * ca + cg * sb * sa, sg * sa + cg * sb * ca, x[3]],
                          [sg * cb, cg * ca + sg * sb * sa, -cg * sa + sg * sb * ca, x[4]],
                          [-sb, cb * sa, cb * ca, x[5]], [0.0, 0.0, 0.0, 1.0]])
            P = torch.from_numpy(D).to(DEV) @ P
    return P.reshape(16)


def _exact_train(net, x, y, lr):
    spec = [(2, 16, 5, 2), (16, 32, 3, 1), (32, 64, 3, 1), (64, 128, 3, 1)]
    flat, at, params = net.master.double(), 0, []
    low = net.params.view(torch.bfloat16).double()  # the weights the layers use; biases come from the master copy

    def take(*shape, bias=False):
        nonlocal at
        n = math.prod(shape)
        p = (flat if bias else low)[at:at + n].reshape(shape).clone().requires_grad_(True)
        at += n
        params.append(p)
        return p

    a = x.view(torch.bfloat16).double().reshape(-1, 2, 60, 80)
    for ci, co, k, pad in spec:
        wt, b = take(co, ci, k, k), take(co, bias=True)
        a = torch.relu(torch.nn.functional.conv2d(a, wt, b, stride=2, padding=pad))
    w1, b1 = take(160, 2560), take(160, bias=True)
    w2, b2 = take(6, 160), take(6, bias=True)
    out = torch.relu(a.flatten(1) @ w1.T + b1) @ w2.T + b2
    loss = (net.loss_w.double() * (out - y.double()) ** 2).sum(1).mean()
    loss.backward()
    g = torch.cat([p.grad.reshape(-1) for p in params])
    # Adam's first step from zero moments: the corrected moments are g and g^2
    master = flat - lr * g / (g.abs() + 1e-8)
    return [loss.detach().reshape(1), g, master, master]
