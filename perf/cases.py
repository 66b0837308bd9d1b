"""The work this library is used for, as cases that can be timed and compared.

Each case is a dict of plain values; ``prepare`` makes what a user's program
holds before the call (frames, a session with a map, a batch, a server),
``run`` is one pass through the public entry points.  Sizes are those of the
library's own workload presets (160x120, 320x240, 640x480 and 1280x720
frames, 4 to 10 mm voxels, 2^18 to 2^21 hash buckets); ``draw`` gives sizes in
between, odd ones included.

Kinds
  filter     dyn_bilateral_filter on a device depth image: a program with its
             own tracker that only wants the filtered depth
  maps       dyn_depth_to_maps on a device depth image: vertices and normals
  equations  dyn_icp_normal_equations on device images: one Gauss-Newton
             iteration's 6x6 system for a program with its own solver
  solve      dyn_solver_solve: one frame registered against another, host
             images in, pose out
  track      Session: one camera frame tracked, fused into the map and the
             map raycast for the next frame -- the per-frame loop of a robot
             or a scanner, in the three precision forms
  render     Session: one frame fused at a known pose (motion capture, replay
             of a logged trajectory) and the map rendered for a viewer
  batch      Batch: many cameras stepped together
  serve      Server: many clients' frames pushed, one step, results read
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from dynamap_b200 import abi, configs, scene
from dynamap_b200.session import Batch, Server, Session

RING = 8        # frames of a clip; played forwards and backwards
Z_MEAN = 1.8    # typical surface depth of the scenes (metres)
PRECISION = {"fp32": abi.PRECISION_FP32, "mixed": abi.PRECISION_MIXED,
             "band": abi.PRECISION_MIXED_BAND}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a low-resolution depth image, where the launch counts
        dict(name="filter_160x120", kind="filter", rows=120, cols=160, diameter=8),
        # the largest image the presets know
        dict(name="filter_1280x720", kind="filter", rows=720, cols=1280, diameter=8),
        # vertices and normals of a VGA image
        dict(name="maps_640x480", kind="maps", rows=480, cols=640),
        # the photometric system of the finest level of a VGA frame
        dict(name="equations_640x480", kind="equations", rows=480, cols=640, rgb=True),
        # frame-to-frame registration of QVGA images in host memory
        dict(name="solve_320x240", kind="solve", rows=240, cols=320, rgb=False),
        # the plain depth-only stream at QVGA, frames from a file reader (pageable)
        dict(name="track_320x240_fp32", kind="track", rows=240, cols=320, voxel=0.008,
             buckets=1 << 18, blocks=1 << 17, rgb=False, precision="fp32", pinned=False,
             ahead=False),
        # the plain RGB-D stream at VGA with the photometric term
        dict(name="track_640x480_rgb_fp32", kind="track", rows=480, cols=640, voxel=0.005,
             buckets=1 << 20, blocks=1 << 19, rgb=True, precision="fp32", pinned=True,
             ahead=False),
        # the same in the mixed form
        dict(name="track_640x480_rgb_mixed", kind="track", rows=480, cols=640, voxel=0.005,
             buckets=1 << 20, blocks=1 << 19, rgb=True, precision="mixed", pinned=True,
             ahead=False),
        # a 720p depth stream with band allocation, the next frame submitted
        # before the last one's result is read
        dict(name="track_1280x720_band", kind="track", rows=720, cols=1280, voxel=0.004,
             buckets=1 << 21, blocks=1 << 19, rgb=False, precision="band", pinned=True,
             ahead=True),
        # replay at known poses with a viewer, a cropped (ragged) sensor
        dict(name="render_633x471_rgb_fp32", kind="render", rows=471, cols=633, voxel=0.006,
             buckets=1 << 19, blocks=1 << 18, rgb=True, precision="fp32"),
        # 32 cameras of mixed resolution stepped together
        dict(name="batch_32_band", kind="batch", sessions=32, precision="band"),
        # ten clients of mixed resolution served at once, free space carved
        dict(name="serve_10_mixed", kind="serve", sessions=10, precision="mixed"),
    ]


def draw(rng):
    def size(lo, hi):
        rows = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        wide = rng.choice([4 / 3, 4 / 3, 16 / 9])
        cols = int(round(rows * wide)) + rng.choice([0, 0, 1, -3, 5])
        return dict(rows=rows, cols=cols)

    kind = rng.choice(["filter", "maps", "equations", "solve", "track", "track", "track",
                       "render", "batch", "serve"])
    if kind == "filter":
        return dict(kind=kind, diameter=rng.choice([4, 5, 6, 7, 8, 8]), **size(96, 720))
    if kind == "maps":
        return dict(kind=kind, **size(96, 720))
    if kind in ("equations", "solve"):
        return dict(kind=kind, rgb=rng.random() < 0.5, **size(120, 600))
    if kind in ("track", "render"):
        precision = rng.choice(["fp32", "fp32", "mixed", "band"])
        c = dict(kind=kind, precision=precision, rgb=rng.random() < 0.5,
                 voxel=round(rng.uniform(0.005, 0.01), 4), **size(120, 600))
        n = _visible_blocks(_sensor(c), c["voxel"], precision)
        c["blocks"] = 1 << max(14, math.ceil(math.log2(6 * n)))
        c["buckets"] = 1 << max(16, math.ceil(math.log2(6 * n)) + rng.choice([0, 1]))
        if kind == "track":
            c.update(pinned=rng.random() < 0.5, ahead=rng.random() < 0.3)
        return c
    if kind == "batch":
        precision = rng.choice(["fp32", "mixed", "band", "band"])
        most = {"fp32": 10, "mixed": 16, "band": 31}[precision]
        return dict(kind=kind, sessions=rng.randint(3, most), precision=precision)
    return dict(kind=kind, sessions=rng.randint(2, 9),
                precision=rng.choice(["mixed", "band", "band"]))


# ------------------------------------------------------------------ parameters
def _sensor(c):
    """A pinhole sensor of the presets' field of view."""
    f = 525.0 * c["cols"] / 640.0
    return dict(rows=c["rows"], cols=c["cols"], fx=f, fy=f, cx=(c["cols"] - 1) / 2.0,
                cy=(c["rows"] - 1) / 2.0, depth_scaler=1000.0)


def _params(c):
    """A session's parameters in the presets' form."""
    v = c.get("voxel", 0.01)
    p = configs.preset("cfg2" if c.get("rgb") else "cfg1")
    p["sensor"] = _sensor(c)
    p["tsdf"].update(voxel_size=v, truncation_distance=4 * v,
                     num_buckets=c.get("buckets", 1 << 12), num_blocks=c.get("blocks", 1 << 10))
    return p


def _members(c):
    """Parameters of a batch's or a server's sessions."""
    if c["kind"] == "batch":
        return [p for _, p, _ in configs.session_mix(c["sessions"])]
    kinds = configs.SERVING["kinds"]
    return [configs.serving_kind(kinds[i % len(kinds)]) for i in range(c["sessions"])]


# ------------------------------------------------------------------ frames
def _perlin(p, perm):
    """Gradient noise at p (n, 3), the albedo of scene.render, on the GPU."""
    grad = torch.tensor(scene._GRAD, device=p.device)
    i = torch.floor(p).long()
    f = p - i
    i &= 255
    u = f * f * f * (f * (f * 6 - 15) + 10)
    out = 0.0
    for k in range(8):
        o = [k & 1, (k >> 1) & 1, (k >> 2) & 1]
        h = perm[perm[perm[i[:, 0] + o[0]] + i[:, 1] + o[1]] + i[:, 2] + o[2]] & 15
        d = (grad[h] * (f - torch.tensor(o, device=p.device, dtype=p.dtype))).sum(1)
        w = 1.0
        for a in range(3):
            w = w * (u[:, a] if o[a] else 1 - u[:, a])
        out = out + w * d
    return out


def _render(sc, pose, s, gen, with_rgb):
    """One noisy frame of scene 'sc' (scene.render, on the GPU): depth in
    sensor units (int16 bits of uint16) and RGB."""
    dev, f64 = "cuda", torch.float64
    t = lambda a: torch.as_tensor(np.asarray(a), device=dev, dtype=f64)  # noqa: E731
    v, u = torch.meshgrid(torch.arange(s["rows"], device=dev, dtype=f64),
                          torch.arange(s["cols"], device=dev, dtype=f64), indexing="ij")
    d = torch.stack([(u - s["cx"]) / s["fx"], (v - s["cy"]) / s["fy"], torch.ones_like(u)],
                    -1).reshape(-1, 3) @ t(pose[:3, :3]).T
    o = t(pose[:3, 3])
    best = torch.full((d.shape[0],), math.inf, device=dev, dtype=f64)
    prim = torch.zeros(d.shape[0], device=dev, dtype=torch.long)

    def hit(z, ok, k):
        nearer = ok & (z < best)
        best[nearer] = z[nearer]
        prim[nearer] = k

    z = (sc.floor_y - o[1]) / d[:, 1]
    x, y = o[0] + z * d[:, 0], o[2] + z * d[:, 2]
    hit(z, (z > 0) & (x >= sc.floor_lo[0]) & (x <= sc.floor_hi[0]) & (y >= sc.floor_lo[1])
        & (y <= sc.floor_hi[1]), 0)
    colours = [sc.floor_color]
    for b in sc.boxes:
        t1, t2 = (t(b.lo) - o) / d, (t(b.hi) - o) / d
        near = torch.minimum(t1, t2).amax(1)
        far = torch.maximum(t1, t2).amin(1)
        hit(near, (near > 0) & (far >= near), len(colours))
        colours.append(b.color)
    for b in sc.spheres:
        oc = o - t(b.center)
        a, h, q = (d * d).sum(1), d @ oc, float(oc @ oc) - b.radius ** 2
        disc = h * h - a * q
        z = (-h - disc.clamp(min=0).sqrt()) / a
        hit(z, (disc >= 0) & (z > 0), len(colours))
        colours.append(b.color)
    ok = torch.isfinite(best) & (best >= 0.1) & (best <= 4.0)
    z = torch.where(ok, best, 0.0)
    noise = torch.randn(z.shape, generator=gen, device=dev, dtype=torch.float32).double()
    raw = torch.where(ok, torch.round((z + (0.0012 + 0.0019 * (z - 0.4) ** 2) * noise)
                                      * s["depth_scaler"]), 0.0).clamp(0, 32767)
    raw = raw.to(torch.int16).reshape(s["rows"], s["cols"])
    if not with_rgb:
        return raw, None
    p = o + z[:, None] * d
    perm = torch.as_tensor(sc.perm, device=dev)
    shade = (0.65 + 0.35 * _perlin(p * 6.0, perm) + 0.15 * _perlin(p * 23.0 + 17.0, perm))
    rgb = (t(np.stack(colours))[prim] * shade.clamp(0.0, 1.2)[:, None]).clamp(0, 1) * 255.0
    rgb = torch.where(ok[:, None], rgb, 0.0).round().to(torch.uint8)
    return raw, rgb.reshape(s["rows"], s["cols"], 3)


def _clip(s, seed, n, rgb, trans=0.005, rot=0.5):
    """n frames along a smooth seeded trajectory: device frames and poses."""
    sc = scene.make_scene(seed)
    poses = scene.trajectory(sc, max(n, 2), seed, trans, rot)[:n]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [_render(sc, poses[k], s, gen, rgb) for k in range(n)], poses.astype(np.float32)


def _host(frames, pinned):
    """Host arrays of device frames, as a camera driver or a file reader
    hands them over."""
    def one(x, dtype):
        if x is None:
            return None
        x = x.cpu()
        return (x.pin_memory() if pinned else x).numpy().view(dtype)
    return [(one(d, np.uint16), one(c, np.uint8)) for d, c in frames]


def _metres(raw, s):
    return raw.float() / s["depth_scaler"]


class _Player:
    """A clip played forwards and backwards, from its end."""

    def __init__(self, frames):
        n = len(frames)
        self.frames, self.order, self.at = frames, list(range(n - 1, -1, -1)) + list(range(1, n - 1)), 0

    def __call__(self):
        k = self.order[self.at % len(self.order)]
        self.at += 1
        return self.frames[k]


def _normals(d, s, dt):
    """Vertices and normals (zero where undefined) of a depth image:
    n = normalise((V(u+2) - V(u-2)) x (V(v+1) - V(v-1)))."""
    rows, cols = d.shape
    v, u = torch.meshgrid(torch.arange(rows, device=d.device, dtype=dt),
                          torch.arange(cols, device=d.device, dtype=dt), indexing="ij")
    d = d.to(dt)
    f32 = lambda x: float(np.float32(x))  # noqa: E731
    p = torch.stack([(u - f32(s["cx"])) * d / f32(s["fx"]), (v - f32(s["cy"])) * d / f32(s["fy"]), d], -1)
    vert = torch.cat([p, torch.ones_like(p[..., :1])], -1) * (d > 0)[..., None]
    nrm = torch.zeros(rows, cols, 4, device=d.device, dtype=dt)
    if rows > 2 and cols > 4:
        a = p[1:-1, 4:] - p[1:-1, :-4]
        b = p[2:, 2:-2] - p[:-2, 2:-2]
        n = torch.linalg.cross(a, b)
        ok = ((d[1:-1, 2:-2] > 0) & (d[1:-1, 4:] > 0) & (d[1:-1, :-4] > 0) & (d[2:, 2:-2] > 0)
              & (d[:-2, 2:-2] > 0))
        len2 = (n * n).sum(-1)
        ok &= len2 > 0
        nrm[1:-1, 2:-2, :3] = torch.where(ok[..., None], n / len2.clamp(min=1e-300 if dt == torch.float64 else 1e-38).sqrt()[..., None], 0.0)
    return vert, nrm


def _intensity(rgb):
    w = torch.tensor([0.2126, 0.7152, 0.0722], device=rgb.device, dtype=torch.float64)
    return ((rgb.double() / 255.0) @ w).float()


def _pair(c, seed):
    """Two frames half a degree apart as float images: (source, target), each
    (depth, normals, intensity), and the motion between them, perturbed."""
    s = _sensor(c)
    frames, poses = _clip(s, seed, 2, c["rgb"])
    out = []
    for raw, rgb in (frames[1], frames[0]):
        d = _metres(raw, s)
        out.append((d, _normals(d, s, torch.float32)[1].contiguous(),
                    _intensity(rgb) if c["rgb"] else None))
    T = (np.linalg.inv(poses[0].astype(np.float64)) @ poses[1].astype(np.float64))
    T[:3, 3] += np.random.default_rng(seed).uniform(-0.002, 0.002, 3)
    return s, out, T.astype(np.float32)


def _ptr(t):
    return None if t is None else t.data_ptr()


def _gn(c):
    return configs._gn([10, 5, 4], color_weight=0.1 if c.get("rgb") else 0.0)


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    k = case["kind"]
    st = {"kind": k, "lib": abi.load()}
    if k in ("filter", "maps"):
        s = _sensor(case)
        frames, _ = _clip(s, seed, 1, False)
        st["depth"] = _metres(frames[0][0], s).contiguous()
        st["stream"] = torch.cuda.current_stream().cuda_stream
        if k == "filter":
            st["out"] = torch.empty_like(st["depth"])
            st["params"] = abi.BilateralParams(case["diameter"], 10.0, 1.0, 1)
        else:
            st["sensor"] = abi.make_params(s, {}, {})[3]
            st["vertex"] = torch.empty(s["rows"], s["cols"], 4, device="cuda")
            st["normal"] = torch.empty(s["rows"], s["cols"], 4, device="cuda")
        return st
    if k == "equations":
        s, st["images"], T = _pair(case, seed)
        _, st["gn"], _, st["sensor"] = abi.make_params(s, {}, _gn(case))
        st["T"] = (C.c_float * 16)(*T.reshape(16).tolist())
        st["stream"] = torch.cuda.current_stream().cuda_stream
        return st
    if k == "solve":
        s = _sensor(case)
        frames, _ = _clip(s, seed, 2, case["rgb"])
        st["images"] = [(_metres(d, s).cpu().numpy(), None if c is None else c.cpu().numpy())
                        for d, c in frames]
        p = _params(case)
        p["gn"] = _gn(case)
        st["session"] = Session(*configs.structs(p))
        return st
    if k in ("track", "render"):
        p = _params(case)
        fast = case["rgb"] and k == "track"  # the RGB preset moves twice as fast
        frames, poses = _clip(p["sensor"], seed, RING, case["rgb"], 0.01 if fast else 0.005,
                              1.0 if fast else 0.5)
        host = _host(frames, case.get("pinned", False))
        m = Session(*configs.structs(p), precision=PRECISION[case["precision"]])
        st["session"] = m
        if k == "render":
            host = [(d, c, q) for (d, c), q in zip(host, poses)]
            for f in host:
                m.integrate_with_pose(*f)
            st["next"] = _Player(host)
            # a viewer a little off the camera's path, at half resolution
            s = p["sensor"]
            st["view"] = abi.make_params(dict(
                rows=s["rows"] // 2, cols=s["cols"] // 2, fx=s["fx"] / 2, fy=s["fy"] / 2,
                cx=(s["cx"] + 0.5) / 2 - 0.5, cy=(s["cy"] + 0.5) / 2 - 0.5,
                depth_scaler=s["depth_scaler"]), {}, {})[3]
            st["offset"] = np.array([0.03, -0.02, 0.0], np.float32)
            return st
        m.set_pose(poses[0])
        for d, c in host:
            m.process(d, c)
        st["next"] = _Player(host)
        st["ahead"] = case["ahead"]
        if case["ahead"]:
            m.submit(*st["next"]())
        return st
    precision = PRECISION[case["precision"]]
    clips = []
    for i, p in enumerate(_members(case)):
        frames, poses = _clip(p["sensor"], seed + 1000003 * i, RING, False)
        clips.append((p, _host(frames, True), poses[0]))
    steps = _Player([[c[1][j][0] for c in clips] for j in range(RING)])
    if k == "batch":
        st["sessions"] = [Session(*configs.structs(p), precision=precision) for p, _, _ in clips]
        for m, (_, _, q) in zip(st["sessions"], clips):
            m.set_pose(q)
        st["batch"] = Batch(st["sessions"])
        for depths in steps.frames:
            st["batch"].process(depths)
    else:
        sv = Server(budget_bytes=9 << 30, max_sessions=32)
        st["server"] = sv
        st["slots"] = [sv.admit(*configs.structs(p), precision=precision, pose0=q)
                       for p, _, q in clips]
        for depths in steps.frames:
            _serve(sv, st["slots"], depths)
    st["next"] = steps
    return st


# ------------------------------------------------------------------ run
def _counts(f):
    return np.array([f.icp_iterations[0], f.icp_iterations[1], f.icp_iterations[2],
                     f.icp_inliers[2], f.blocks_total, f.blocks_visible], np.int64)


def _serve(sv, slots, depths):
    for slot, d in zip(slots, depths):
        sv.push(slot, d)
    sv.step()
    return [sv.result(slot) for slot in slots]


def run(st):
    k, lib = st["kind"], st["lib"]
    if k == "filter":
        rows, cols = st["depth"].shape
        abi.check("dyn_bilateral_filter", lib.dyn_bilateral_filter(
            st["depth"].data_ptr(), st["out"].data_ptr(), rows, cols, C.byref(st["params"]),
            st["stream"]))
        return st["out"]
    if k == "maps":
        abi.check("dyn_depth_to_maps", lib.dyn_depth_to_maps(
            st["depth"].data_ptr(), C.byref(st["sensor"]), st["vertex"].data_ptr(),
            st["normal"].data_ptr(), st["stream"]))
        return {"vertex": st["vertex"], "normal": st["normal"]}
    if k == "equations":
        (sd, sn, si), (td, tn, ti) = st["images"]
        out = (C.c_double * 29)()
        abi.check("dyn_icp_normal_equations", lib.dyn_icp_normal_equations(
            _ptr(sd), _ptr(sn), _ptr(si), _ptr(td), _ptr(tn), _ptr(ti), C.byref(st["sensor"]),
            C.byref(st["gn"]), st["T"], out, st["stream"]))
        return np.array(out)
    if k == "solve":
        (td, tc), (sd, sc) = st["images"]
        pose = (C.c_float * 16)(*np.eye(4).reshape(16).tolist())
        inc = (C.c_double * 6)()
        arr = lambda a: None if a is None else a.ctypes.data  # noqa: E731
        abi.check("dyn_solver_solve", lib.dyn_solver_solve(
            st["session"].h, arr(td), arr(tc), arr(sd), arr(sc), pose, inc, None))
        return {"pose": np.array(pose, np.float32), "increment": np.array(inc)}
    if k == "track":
        m = st["session"]
        m.submit(*st["next"]())
        pose, stats = m.result()
        return {"pose": pose, "counts": _counts(stats)}
    if k == "render":
        m = st["session"]
        d, c, q = st["next"]()
        m.integrate_with_pose(d, c, q)
        q = q.copy()
        q[:3, 3] += st["offset"]
        depth, vertex, normal, rgb = m.raycast_maps(q, sensor=st["view"], rgb=True)
        return {"depth": depth, "vertex": vertex, "normal": normal, "rgb": rgb}
    if k == "batch":
        poses, stats, _ = st["batch"].process(st["next"]())
        return {"poses": poses, "counts": np.stack([_counts(f) for f in stats])}
    got = _serve(st["server"], st["slots"], st["next"]())
    return {"poses": np.stack([p for p, _ in got]), "counts": np.stack([_counts(f) for _, f in got])}


# ------------------------------------------------------------------ work
def _visible_blocks(s, voxel, precision):
    """Blocks a frame updates: the viewing volume up to the surface, or with
    band allocation the surface's blocks a truncation distance either way."""
    solid = s["rows"] * s["cols"] / (s["fx"] * s["fy"])
    edge = 8 * voxel
    if precision == "band":
        return 2.5 * solid * Z_MEAN ** 2 / edge ** 2
    return solid * Z_MEAN ** 3 / 3 / edge ** 3


def _frame_work(s, voxel, precision, rgb, track):
    """The frame read, the blocks it updates read and written, the next
    target (depth and normals) written; the filter's taps."""
    px = s["rows"] * s["cols"]
    vox = 8 if precision == "fp32" or rgb else 4
    b = px * (5 if rgb else 2) + 2 * 512 * vox * _visible_blocks(s, voxel, precision) + 20 * px
    f = px * 256 * 12
    if track:  # the Gauss-Newton terms, 16 iterations over three levels
        f += px * 70 * (9 / 16 + 4 / 4 + 3)
    return b, f


def work(case):
    k = case["kind"]
    if k in ("batch", "serve"):
        b = f = 0.0
        for p in _members(case):
            x = _frame_work(p["sensor"], p["tsdf"]["voxel_size"], case["precision"], False, True)
            b, f = b + x[0], f + x[1]
        return {"bytes": b, "flops": f}
    s = _sensor(case)
    px = s["rows"] * s["cols"]
    if k == "filter":
        return {"bytes": 8 * px, "flops": px * (2 * case["diameter"]) ** 2 * 12}
    if k == "maps":
        return {"bytes": 36 * px, "flops": 60 * px}
    if k == "equations":
        return {"bytes": px * (48 if case["rgb"] else 40), "flops": 100 * px}
    if k == "solve":
        return {"bytes": 2 * px * (7 if case["rgb"] else 4),
                "flops": px * 70 * (9 / 16 + 4 / 4 + 3)}
    b, f = _frame_work(s, case["voxel"], case["precision"], case["rgb"], k == "track")
    if k == "render":
        b += px / 4 * 39
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """The stages' results in 64 bits, in plain torch; None for the calls
    whose result is a whole tracked or mapped frame."""
    if case["kind"] == "filter":
        return _exact_filter(case, seed)
    if case["kind"] == "maps":
        s = _sensor(case)
        d = _metres(_clip(s, seed, 1, False)[0][0][0], s)
        v, n = _normals(d, s, torch.float64)
        return {"vertex": v, "normal": n}
    if case["kind"] == "equations":
        return _exact_equations(case, seed)
    return None


def _exact_filter(case, seed):
    s, r = _sensor(case), case["diameter"]
    d = _metres(_clip(s, seed, 1, False)[0][0][0], s).double()
    rows, cols = d.shape
    pad = torch.zeros(rows + 2 * r, cols + 2 * r, device=d.device, dtype=d.dtype)
    pad[r:r + rows, r:r + cols] = d
    acc, wp = torch.zeros_like(d), torch.zeros_like(d)
    for i in range(2 * r):
        for j in range(2 * r):
            t = pad[i:i + rows, j:j + cols]
            w = torch.exp(-(t - d) ** 2 / (2 * 10.0 ** 2)) * math.exp(-((i - r) ** 2 + (j - r) ** 2) / 2.0)
            w = torch.where(t > 0, w, 0.0)
            acc += t * w
            wp += w
    return torch.where(d > 0, acc / wp.clamp(min=1e-300), 0.0)


def _exact_equations(case, seed):
    s, ((sd, sn, si), (td, tn, ti)), T = _pair(case, seed)
    f64 = torch.float64
    rows, cols = sd.shape
    f32 = lambda x: float(np.float32(x))  # noqa: E731
    fx, fy, cx, cy = f32(s["fx"]), f32(s["fy"]), f32(s["cx"]), f32(s["cy"])
    gn = _gn(case)
    dmin, dmax, cw = f32(gn["icp_min_depth"]), f32(gn["icp_max_depth"]), f32(gn["color_weight"])
    T = torch.as_tensor(T, device=sd.device, dtype=f64)
    v, u = torch.meshgrid(torch.arange(rows, device=sd.device, dtype=f64),
                          torch.arange(cols, device=sd.device, dtype=f64), indexing="ij")
    z = sd.double()
    p = torch.stack([(u - cx) * z / fx, (v - cy) * z / fy, z], -1) @ T[:3, :3].T + T[:3, 3]
    n_s = sn[..., :3].double()
    ok = (z >= dmin) & (z <= dmax) & (n_s.abs().sum(-1) > 0) & (p[..., 2] > 0)
    zz = torch.where(ok, p[..., 2], 1.0)
    half = lambda x: torch.sign(x) * torch.floor(x.abs() + 0.5)  # noqa: E731  (half away from zero)
    px, py = half(fx * p[..., 0] / zz + cx), half(fy * p[..., 1] / zz + cy)
    ok &= (px >= 0) & (py >= 0) & (px < cols) & (py < rows)
    px, py = torch.where(ok, px, 0.0).long(), torch.where(ok, py, 0.0).long()
    q_d, n = td[py, px].double(), tn[py, px][..., :3].double()
    ok &= (q_d >= dmin) & (q_d <= dmax) & (n.abs().sum(-1) > 0)
    ok &= (n * n_s).sum(-1).abs() > f32(gn["normal_cos_thresh"])
    q = torch.stack([(px - cx) * q_d / fx, (py - cy) * q_d / fy, q_d], -1)
    p, n, q, px, py = p[ok], n[ok], q[ok], px[ok], py[ok]
    J = torch.cat([torch.linalg.cross(p, n), n], -1)
    r = ((p - q) * n).sum(-1)
    A, b = J.T @ J, -(J.T @ r)
    if cw:
        i_t, i_s = ti.double(), si.double()[ok]
        e = i_t[py, px] - i_s
        gx = (i_t[py, px] - i_t[py, (px - 1).clamp(min=0)]) / 2
        gy = (i_t[py, px] - i_t[(py - 1).clamp(min=0), px]) / 2
        Jc = torch.stack([-gy * p[:, 2], gx * p[:, 2], gy * p[:, 0] - gx * p[:, 1], gx, gy,
                          torch.zeros_like(gx)], -1)
        A = (1 - cw) * A + cw * (Jc.T @ Jc)
        b = (1 - cw) * b - cw * (Jc.T @ e)
    i, j = torch.triu_indices(6, 6)
    return torch.cat([A[i, j], b, (r * r).sum()[None], torch.tensor([float(len(r))], device=r.device,
                                                                    dtype=f64)]).cpu().numpy()
