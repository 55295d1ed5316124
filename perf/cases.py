"""Performance cases: the calls a program built on this framework makes, over
the range of sizes and options it makes them with.

Every case is one pass through the public entry points (`fusion_b200.Session`,
`fusion_b200.batch.Batch`, the per-stage functions of `fusion_b200.system` and
the C ABI) on inputs made from a seed: RGB-D frames of the seeded
procedural room (`rgbd_synth`), the sequences the tests and the benchmark use.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs, sessions and handles, on the GPU
    run(state)           one pass; returns its outputs
    work(case)           bytes and flops one pass cannot do without
    exact(case, seed)    the pass's computed numbers in 64 bits, where there
                         is a short way to them without this package

A session's passes walk its sequence forth and back, so that it can be stepped
any number of times: each pass is the next frame of a running camera.
"""
import ctypes

import numpy as np
import torch

import rgbd_synth
from fusion_b200 import Session, load
from fusion_b200 import system as S
from fusion_b200.batch import Batch, mixed_config, mixed_population

CUTOFF, SCALE = 4.0, 5000.0   # metres and depth units per metre of the synthetic sequences


def listed():
    return [
        # a robot's or phone's low-resolution camera: a frame's launches and latency are the cost
        {"name": "live_160x120", "kind": "live", "width": 160, "height": 120, "voxel_mm": 10.0, "trunc": 8,
         "form": "reference", "input": "host"},
        # the full-size camera as the benchmark runs it end to end: the next frame staged while this one runs
        {"name": "live_640x480", "kind": "live", "width": 640, "height": 480, "voxel_mm": 5.0, "trunc": 4,
         "form": "reference", "input": "staged"},
        # a camera cropped to an odd size, in the precision form (6-byte voxels)
        {"name": "live_precision_427x319", "kind": "live", "width": 427, "height": 319, "voxel_mm": 6.0,
         "trunc": 8, "form": "precision", "input": "host"},
        # a high-resolution sensor whose frames a decoder has left in GPU memory
        {"name": "live_1280x960", "kind": "live", "width": 1280, "height": 960, "voxel_mm": 8.0, "trunc": 4,
         "form": "reference", "input": "device"},
        # the interactive viewer: every frame followed by the shaded top-down view of the model
        {"name": "viewer_640x480", "kind": "viewer", "width": 640, "height": 480, "voxel_mm": 6.0, "trunc": 8,
         "form": "reference", "input": "host"},
        # a server stepping many cameras of mixed sizes together, host frames
        {"name": "batch_16", "kind": "batch", "sessions": 16, "mode": 0, "population": 5},
        # offline reconstruction with known poses: FuseMapColor and the model raycast of a dataset's frame
        {"name": "mapping_640x480", "kind": "mapping", "width": 640, "height": 480, "voxel_mm": 4.0, "trunc": 8,
         "form": "reference"},
        # visual odometry on caller images: one ICP step and one photometric step of a Gauss-Newton loop
        {"name": "odometry_323x241", "kind": "odometry", "width": 323, "height": 241},
        # preprocessing of a large odd-sized frame through the per-stage functions
        {"name": "pyramid_1283x721", "kind": "pyramid", "width": 1283, "height": 721},
        # export of the scanned room as a triangle mesh
        {"name": "mesh_5mm", "kind": "mesh", "width": 640, "height": 480, "voxel_mm": 5.0, "trunc": 4,
         "form": "reference"},
        # a full-size camera with key points on: detection, matching, bootstrap pose
        {"name": "keypoints_640x480", "kind": "keypoints", "width": 640, "height": 480, "voxel_mm": 5.0, "trunc": 4,
         "form": "reference", "input": "host"},
        # relocalisation: a frame's descriptors against a key map
        {"name": "match_900x20000", "kind": "match", "queries": 900, "train": 20000},
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def _size(rng, lo, hi):
    """Width over its logarithm, height about 3/4 of it; odd sizes as often as even ones."""
    w = int(_log(rng, lo, hi))
    return w, int(w * rng.uniform(0.55, 0.8))


def draw(rng):
    kind = rng.choice(["live", "live", "live", "viewer", "batch", "mapping", "odometry", "pyramid", "mesh",
                       "keypoints", "match"])
    if kind in ("live", "viewer", "keypoints", "mapping", "mesh"):
        w, h = _size(rng, 320, 640) if kind in ("keypoints", "mesh", "viewer") else _size(rng, 160, 1280)
        voxel = round(_log(rng, 4.0 if kind == "mapping" else 5.0, 20.0), 2)
        # a truncation of 4 voxels holds a camera's noise only where voxels and images are not too small
        trunc = rng.choice([4, 8]) if voxel >= 8.0 and w >= 240 else 8
        case = {"kind": kind, "width": w, "height": h, "voxel_mm": voxel, "trunc": trunc,
                "form": rng.choice(["reference", "reference", "precision"])}
        if kind in ("live", "viewer", "keypoints"):
            case["input"] = rng.choice(["host", "staged", "device"])
        return case
    if kind == "batch":
        return {"kind": kind, "sessions": int(_log(rng, 2, 16.99)), "mode": rng.choice([0, 2]),
                "population": rng.randrange(1000)}
    if kind == "odometry" or kind == "pyramid":
        w, h = _size(rng, 80, 1280 if kind == "odometry" else 2000)
        return {"kind": kind, "width": w, "height": h}
    return {"kind": kind, "queries": int(_log(rng, 30, 1000)), "train": int(_log(rng, 100, 18000))}


# ------------------------------------------------------------------ inputs

def _params(width, height, seed, **more):
    f = 525.0 * width / 640.0
    return rgbd_synth.params(width, height, rgbd_synth.session_seed(31, seed), fx=f, fy=f, cx=width / 2.0,
                             cy=height / 2.0, depth_scale=SCALE, **more)


def _config(case):
    cfg = mixed_config(case["width"], case["height"], case["voxel_mm"] / 1000.0, case["trunc"])
    if case["form"] == "precision":
        cfg.form = 1
    return cfg


def _pinned(a):
    return torch.from_numpy(a).pin_memory().numpy()


class _Frames:
    """A sequence walked forth and back without end."""

    def __init__(self, width, height, seed, count, on_device=False):
        d, c, self.poses = rgbd_synth.render(_params(width, height, seed), 0, count)
        if on_device:
            self.frames = [(torch.from_numpy(d[i]).cuda(), torch.from_numpy(c[i]).cuda()) for i in range(count)]
        else:
            d, c = _pinned(d), _pinned(c)
            self.frames = [(d[i], c[i]) for i in range(count)]
        self.order = list(range(count)) + list(range(count - 2, 0, -1))
        self.at = 0

    def next(self):
        k = self.order[self.at]
        self.at = (self.at + 1) % len(self.order)
        return k, self.frames[k]


class _Camera:
    """A session that has tracked its whole sequence once.  A scene whose first,
    sparse raycast loses the camera (the reference's tracker does) is passed
    over for the seed's next scene, so that every pass is a tracked frame."""

    def __init__(self, cfg, seed, frames=6, input="host", keypoints=False):
        self.cfg, self.input = cfg, input
        for scene in range(16 * seed, 16 * seed + 16):
            self.seq = _Frames(cfg.width, cfg.height, scene, frames, input == "device")
            self.session = Session(cfg)
            if keypoints:
                self.session.set_keypoints(True)
            if input == "staged":
                self.session.stage(*self.seq.next()[1])
            self.step()
            if all([self.step().tracked for _ in self.seq.order]):
                return
            self.session.close()
        raise RuntimeError("no scene of this seed is tracked")

    def step(self):
        if self.input == "staged":
            self.session.stage(*self.seq.next()[1])
            return self.session.grab(None, None)
        depth, rgb = self.seq.next()[1]
        return self.session.grab(depth, rgb, on_device=self.input == "device")


def _camera(case, seed, **more):
    return _Camera(_config(case), seed, input=case.get("input", "host"), **more)


def _maps(h, w):
    return tuple(torch.zeros((h, w, 4), dtype=torch.float32, device="cuda") for _ in range(2))


def prepare(case, seed):
    kind = case["kind"]
    return {"live": _prepare_live, "viewer": _prepare_viewer, "batch": _prepare_batch, "mapping": _prepare_mapping,
            "odometry": _prepare_odometry, "pyramid": _prepare_pyramid, "mesh": _prepare_mesh,
            "keypoints": _prepare_keypoints, "match": _prepare_match}[kind](case, seed)


def run(state):
    return state["run"](state)


# -------------------------------------------------------- sessions: one camera

def _prepare_live(case, seed):
    return {"run": _run_live, "camera": _camera(case, seed)}


def _run_live(st):
    return Session.result_dict(st["camera"].step())


def _prepare_viewer(case, seed):
    h, w = case["height"], case["width"]
    v, n = _maps(h, w)
    return {"run": _run_viewer, "camera": _camera(case, seed), "v": v, "n": n,
            "rgba": torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")}


def _run_viewer(st):
    cam = st["camera"]
    r = cam.step()
    S.render_top_down(cam.session, 4.0, st["v"], st["n"], st["rgba"])
    return {"frame": Session.result_dict(r), "vertex": st["v"], "normal": st["n"], "rgba": st["rgba"]}


def _prepare_keypoints(case, seed):
    return {"run": _run_keypoints, "camera": _camera(case, seed, keypoints=True)}


def _run_keypoints(st):
    r = st["camera"].step()
    return {"frame": Session.result_dict(r), "stats": st["camera"].session.keypoint_stats()}


# ------------------------------------------------------------ sessions: a batch

def _prepare_batch(case, seed):
    pop = mixed_population(case["sessions"], case["population"])
    batch = Batch(mode=case["mode"])
    cameras = [_Camera(mixed_config(w, h, voxel, 8), 1000 * seed + i, 4) for i, (w, h, voxel) in enumerate(pop)]
    st = {"run": _run_batch, "batch": batch, "cameras": cameras, "sessions": [c.session for c in cameras]}
    for _ in range(3):
        _run_batch(st)
    return st


def _run_batch(st):
    rs = st["batch"].step(st["sessions"], [c.seq.next()[1] for c in st["cameras"]])
    return {"pose": np.array([r.pose[:] for r in rs]),
            "counts": np.array([[r.status, r.no_visible, r.no_allocated, r.no_new, r.error_flags] for r in rs])}


# ------------------------------------------------------- mapping at known poses

def _prepare_mapping(case, seed):
    w, h = case["width"], case["height"]
    cfg = _config(case)
    seq = _Frames(w, h, seed, 4, on_device=True)
    K = (cfg.fx, cfg.fy, cfg.cx, cfg.cy)
    frames = []
    for d, c in seq.frames:
        z = d.to(torch.float32) * np.float32(1.0 / SCALE)
        frames.append((z, c, _normals(_vertices(z, K))))
    v, n = _maps(h, w)
    st = {"run": _run_mapping, "session": Session(cfg), "seq": seq, "frames": frames, "v": v, "n": n,
          "K": np.array(K, np.float32)}
    for _ in range(2):
        _run_mapping(st)
    return st


def _run_mapping(st):
    k, _ = st["seq"].next()
    depth, rgb, normal = st["frames"][k]
    T = st["seq"].poses[k]
    visible = S.fuse_map_color(st["session"], depth, rgb, normal, T, st["K"])
    S.raycast(st["session"], st["v"], st["n"], T, st["K"])
    return {"visible": visible, "vertex": st["v"], "normal": st["n"]}


# --------------------------------------------------------------- caller images

def _vertices(z, K):
    """Vertex map of a depth image in its type; NaN where there is no depth."""
    fx, fy, cx, cy = (float(k) for k in K)
    h, w = z.shape
    x = torch.arange(w, device=z.device, dtype=z.dtype)[None, :]
    y = torch.arange(h, device=z.device, dtype=z.dtype)[:, None]
    ok = (z > 0.1) & (z < CUTOFF)
    nan = torch.full_like(z, float("nan"))
    return torch.stack([torch.where(ok, z * (x - cx) / fx, nan), torch.where(ok, z * (y - cy) / fy, nan),
                        torch.where(ok, z, nan), torch.where(ok, torch.ones_like(z), nan)], -1)


def _normals(v):
    """Normal map of a vertex map by forward differences; NaN in the last row and column."""
    n = torch.full_like(v, float("nan"))
    c, r, d = v[:-1, :-1, :3], v[:-1, 1:, :3], v[1:, :-1, :3]
    m = torch.linalg.cross(r - c, d - c)
    m = m / m.norm(dim=-1, keepdim=True)
    n[:-1, :-1, :3] = m
    n[:-1, :-1, 3] = torch.where(torch.isnan(m[..., 0]), m[..., 0], torch.ones_like(m[..., 0]))
    return n


def _odometry_inputs(case, seed, device):
    w, h = case["width"], case["height"]
    f = 525.0 * w / 640.0
    K = np.array([f, f, w / 2.0, h / 2.0], np.float32)
    d, c, T = rgbd_synth.render(_params(w, h, seed, noise=0), 0, 3)
    g = {}
    for name, i in (("last", 0), ("curr", 2)):
        z = torch.from_numpy(d[i].astype(np.float32)) * np.float32(1.0 / SCALE)
        g["v" + name] = _vertices(z, K)
        g["n" + name] = _normals(g["v" + name])
        img = torch.from_numpy(c[i].astype(np.int32))
        g["g" + name] = ((img[..., 0] * 299 + img[..., 1] * 587 + img[..., 2] * 114) // 1000).clamp(1, 255).to(torch.uint8)
    a = g["gcurr"].to(torch.int32)
    dx, dy = torch.zeros_like(a), torch.zeros_like(a)
    dx[1:-1, 1:-1] = (a[:-2, 2:] + 2 * a[1:-1, 2:] + a[2:, 2:]) - (a[:-2, :-2] + 2 * a[1:-1, :-2] + a[2:, :-2])
    dy[1:-1, 1:-1] = (a[2:, :-2] + 2 * a[2:, 1:-1] + a[2:, 2:]) - (a[:-2, :-2] + 2 * a[:-2, 1:-1] + a[:-2, 2:])
    g["dx"], g["dy"] = dx.to(torch.int16), dy.to(torch.int16)
    return {k: v.contiguous().to(device) for k, v in g.items()}, K, S.pose_parts(T[2]), S.pose_parts(T[0])


def _prepare_odometry(case, seed):
    g, K, cur, last = _odometry_inputs(case, seed, "cuda")
    scratch = torch.zeros(S.step_scratch_bytes(case["width"], case["height"]), dtype=torch.uint8, device="cuda")
    return {"run": _run_odometry, "g": g, "K": K, "cur": cur, "last": last, "scratch": scratch}


def _run_odometry(st):
    g, (R, Ri, t), (Rl, Rli, tl) = st["g"], st["cur"], st["last"]
    icp = S.icp_step(g["vcurr"], g["vlast"], g["ncurr"], g["nlast"], R, t, Rl, Rli, tl, st["K"], st["scratch"])
    rgb = S.rgb_step(g["gcurr"], g["glast"], g["vcurr"], g["vlast"], g["dx"], g["dy"], R, Ri, Rl, Rli, t, tl, st["K"],
                     st["scratch"])
    return {"icp": icp, "rgb": rgb}


def _normal_equations(rows):
    """(residual [sum r^2, count], A, b) of rows [n, 7] as the step functions return them."""
    M = rows.T @ rows
    return np.array([float(M[6, 6]), float(len(rows))]), M[:6, :6].numpy(), M[:6, 6].numpy()


def _exact_odometry(case, seed):
    g, K, cur, last = _odometry_inputs(case, seed, "cpu")
    w, h = case["width"], case["height"]
    fx, fy, cx, cy = (float(k) for k in K)
    R, Ri, t = (torch.from_numpy(np.asarray(a, np.float64)) for a in cur)
    Rl, Rli, tl = (torch.from_numpy(np.asarray(a, np.float64)) for a in last)
    v, vl = g["vcurr"].double().reshape(-1, 4), g["vlast"].double().reshape(-1, 4)
    n, nl = g["ncurr"].double().reshape(-1, 4), g["nlast"].double().reshape(-1, 4)
    vg = v[:, :3] @ R.T + t
    p = (vg - tl) @ Rli.T
    pu, pv = p[:, 0] / p[:, 2] * fx + cx, p[:, 1] / p[:, 2] * fy + cy
    seen = ~torch.isnan(v[:, 0]) & torch.isfinite(pu) & torch.isfinite(pv)
    # ICP: pixel by truncation of the coordinate plus a half
    u, q = torch.nan_to_num(pu + 0.5, nan=-9.0).trunc().long(), torch.nan_to_num(pv + 0.5, nan=-9.0).trunc().long()
    ok = seen & (u >= 0) & (q >= 0) & (u < w) & (q < h)
    j = (q * w + u)[ok]
    lg, nc, ng = vl[j, :3] @ Rl.T + tl, n[ok, :3] @ R.T, nl[j, :3] @ Rl.T
    near = ((lg - vg[ok]).norm(dim=1) <= 0.1) & (torch.linalg.cross(nc, ng).norm(dim=1) < 0.6)
    near &= ~torch.isnan(n[ok, 0]) & ~torch.isnan(nl[j, 0])
    a, vc, vll = ng[near] @ Rli.T, p[ok][near], (lg[near] - tl) @ Rli.T
    rows = torch.cat([-a, torch.linalg.cross(a, vll), -(a * (vc - vll)).sum(1, keepdim=True)], 1)
    icp = _normal_equations(rows)
    # photometric: pixel by floor of the coordinate plus a half, 5-pixel border, nonzero gradient
    u, q = torch.nan_to_num(pu + 0.5, nan=-9.0).floor().long(), torch.nan_to_num(pv + 0.5, nan=-9.0).floor().long()
    x = torch.arange(w).repeat(h)
    y = torch.arange(h).repeat_interleave(w)
    dx, dy = g["dx"].double().reshape(-1), g["dy"].double().reshape(-1)
    ok = seen & (u >= 0) & (q >= 0) & (u < w) & (q < h) & (x >= 5) & (x < w - 5) & (y >= 5) & (y < h - 5)
    ok &= (dx != 0) | (dy != 0)
    i = torch.nonzero(ok).squeeze(1)
    j = (q * w + u)[i]
    near = (vl[j] - v[i]).norm(dim=1) < 0.1
    i, j = i[near], j[near]
    diff = g["gcurr"].double().reshape(-1)[i] - g["glast"].double().reshape(-1)[j]
    sigma = (diff.square().sum() / max(1, len(diff))).sqrt()
    wt = 1.0 / (sigma + diff.abs())
    pt = (vl[j, :3] @ Rl.T + tl - t) @ Ri.T
    lx, ly = dx[i] / 9.0 * fx / pt[:, 2], dy[i] / 9.0 * fy / pt[:, 2]
    left = torch.stack([lx, ly, -(lx * pt[:, 0] + ly * pt[:, 1]) / pt[:, 2]], 1)
    rows = torch.cat([left, torch.linalg.cross(pt, left), -diff[:, None]], 1) * wt[:, None]
    return {"icp": icp, "rgb": _normal_equations(rows)}


def _prepare_pyramid(case, seed):
    w, h = case["width"], case["height"]
    d, c, _ = rgbd_synth.render(_params(w, h, seed), 0, 1)
    f = 525.0 * w / 640.0
    st = {"run": _run_pyramid, "depth": torch.from_numpy(d[0]).cuda(), "rgb": torch.from_numpy(c[0]).cuda(),
          "K": (f, f, w / 2.0, h / 2.0), "raw": torch.zeros((h, w), dtype=torch.float32, device="cuda")}
    for name, dtype, lanes in (("filtered", torch.float32, 0), ("gray", torch.uint8, 0), ("vertex", torch.float32, 4),
                               ("normal", torch.float32, 4), ("dx", torch.int16, 0), ("dy", torch.int16, 0)):
        st[name] = [torch.zeros((h >> l, w >> l) + ((lanes,) if lanes else ()), dtype=dtype, device="cuda")
                    for l in range(3)]
    return st


def _run_pyramid(st):
    fx, fy, cx, cy = st["K"]
    S.filter_depth(st["depth"], st["raw"], st["filtered"][0], SCALE, CUTOFF)
    S.image_to_intensity(st["rgb"], st["gray"][0])
    for l in range(3):
        if l:
            S.pyrdown_gauss(st["filtered"][l - 1], st["filtered"][l])
            S.pyrdown_gauss(st["gray"][l - 1], st["gray"][l])
        s = float(1 << l)
        S.compute_vmap(st["filtered"][l], st["vertex"][l], fx / s, fy / s, cx / s, cy / s, CUTOFF)
        S.compute_nmap(st["vertex"][l], st["normal"][l])
        S.compute_derivative_image(st["gray"][l], st["dx"][l], st["dy"][l])
    return {k: st[k] for k in ("raw", "filtered", "gray", "vertex", "normal", "dx", "dy")}


def _exact_pyramid(case, seed):
    w, h = case["width"], case["height"]
    d, _, _ = rgbd_synth.render(_params(w, h, seed), 0, 1)
    z = torch.from_numpy(d[0].astype(np.float64)) / SCALE
    nan = torch.full_like(z, float("nan"))
    raw = torch.where(z < CUTOFF, z, nan)
    # bilateral 5 x 5 whose window ends before the last row and column
    num, den = torch.zeros_like(z), torch.zeros_like(z)
    for j in range(-2, 3):
        for i in range(-2, 3):
            y0, y1, x0, x1 = max(0, -j), min(h, h - 1 - j), max(0, -i), min(w, w - 1 - i)
            if y1 <= y0 or x1 <= x0:
                continue
            c, v = z[y0:y1, x0:x1], z[y0 + j:y1 + j, x0 + i:x1 + i]
            k = torch.exp(-((i * i + j * j) * 0.03125 + (c - v).square() * 2.0))
            num[y0:y1, x0:x1] += k * v
            den[y0:y1, x0:x1] += k
    f = num / den
    filtered = [torch.where(f < CUTOFF, f, nan)]
    g = torch.tensor([1.0, 4.0, 6.0, 4.0, 1.0], dtype=torch.float64)
    for l in range(1, 3):
        src = filtered[-1]
        sh, sw = src.shape
        oh, ow = sh // 2, sw // 2
        num, den = torch.zeros(oh, ow, dtype=torch.float64), torch.zeros(oh, ow, dtype=torch.float64)
        y, x = torch.arange(oh)[:, None], torch.arange(ow)[None, :]
        ty, tx = (2 * y + 3).clamp(max=sh - 1), (2 * x + 3).clamp(max=sw - 1)
        for j in range(5):       # weights counted from the window's clipped end
            for i in range(5):
                cy, cx = ty - 1 - j, tx - 1 - i
                ok = (cy >= (2 * y - 2).clamp(min=0)) & (cx >= (2 * x - 2).clamp(min=0))
                v = src[cy.clamp(min=0).expand(oh, ow), cx.clamp(min=0).expand(oh, ow)]
                ok = ok & ~torch.isnan(v)
                num += torch.where(ok, v * (g[j] * g[i]), torch.zeros_like(v))
                den += torch.where(ok, (g[j] * g[i]).expand(oh, ow), torch.zeros_like(v))
        filtered.append(num / den)
    K = np.array([525.0 * w / 640.0, 525.0 * w / 640.0, w / 2.0, h / 2.0])
    vertex = []
    for l in range(3):
        v = _vertices(filtered[l], (K / (1 << l)).astype(np.float32))
        v[..., 2] = filtered[l]   # the depth lane is kept where the vertex is invalid
        vertex.append(v)
    return {"raw": raw, "filtered": filtered, "gray": None, "vertex": vertex, "normal": [_normals(v) for v in vertex],
            "dx": None, "dy": None}


# -------------------------------------------------------------------- meshing

def _prepare_mesh(case, seed):
    # buffers allocated once, as the reference's CreateModel keeps them, with room for every scanned room
    cap = int(130 * 1.3 * _blocks(case["voxel_mm"]))
    return {"run": _run_mesh, "camera": _camera(case, seed, frames=12), "cap": cap, "lib": load(),
            "v": torch.zeros((3 * cap, 3), dtype=torch.float32, device="cuda"),
            "n": torch.zeros((3 * cap, 3), dtype=torch.float32, device="cuda"),
            "c": torch.zeros((3 * cap, 3), dtype=torch.uint8, device="cuda")}


def _run_mesh(st):
    count = ctypes.c_uint64()
    rc = st["lib"].fb_mesh_scene(st["camera"].session.h, st["v"].data_ptr(), st["n"].data_ptr(), st["c"].data_ptr(),
                                 st["cap"], ctypes.byref(count), None)
    if rc:
        raise RuntimeError("fb_mesh_scene: status %d" % rc)
    return {"triangles": count.value, "vertex": st["v"], "normal": st["n"], "color": st["c"]}


# ------------------------------------------------------------------- matching

def _descriptors(case, seed):
    g = torch.Generator().manual_seed(seed)
    train = torch.randn(case["train"], 64, generator=g)
    train = train / train.norm(dim=1, keepdim=True)
    pick = torch.randint(0, case["train"], (case["queries"],), generator=g)
    query = train[pick] + 0.08 * torch.randn(case["queries"], 64, generator=g)
    return query / query.norm(dim=1, keepdim=True), train


def _prepare_match(case, seed):
    q, t = _descriptors(case, seed)
    return {"run": _run_match, "q": q.cuda(), "t": t.cuda()}


def _run_match(st):
    best, dist = S.match_descriptors(st["q"], st["t"])
    return {"best": best, "dist": dist}


def _exact_match(case, seed):
    q, t = (a.double() for a in _descriptors(case, seed))
    out = [torch.cdist(c, t, compute_mode="donot_use_mm_for_euclid_dist").topk(2, 1, largest=False).values
           for c in q.split(128)]
    return {"best": None, "dist": torch.cat(out)}


def exact(case, seed):
    if case["kind"] == "odometry":
        return _exact_odometry(case, seed)
    if case["kind"] == "pyramid":
        return _exact_pyramid(case, seed)
    if case["kind"] == "match":
        return _exact_match(case, seed)
    return None   # the state of a running session, from many frames' decisions


# ----------------------------------------------------------------------- work

def _blocks(case_voxel_mm):
    """Voxel blocks in view of one camera in the room: its visible surface over a block's face."""
    return 18.3 / (8 * case_voxel_mm / 1000.0) ** 2


def _frame_work(w, h, voxel_mm, form):
    n = float(w * h)
    vis = _blocks(voxel_mm)
    voxel = 6 if form == "precision" else 8
    iters = 10 * n + 5 * n / 4 + 3 * n / 16
    # frame in, the model's maps in and out, the visible blocks' voxels in and out
    return {"bytes": 5 * n + 2 * 32 * n + vis * (2 * 512 * voxel + 16),
            # Gauss-Newton rows and products; the bilateral filter; a voxel's update; a ray's trilinear samples
            "flops": 260 * iters + 250 * n + 60 * 512 * vis + 8 * 35 * n}


def work(case):
    kind = case["kind"]
    if kind in ("live", "keypoints"):
        return _frame_work(case["width"], case["height"], case["voxel_mm"], case["form"])
    if kind == "viewer":
        a = _frame_work(case["width"], case["height"], case["voxel_mm"], case["form"])
        n = case["width"] * case["height"]
        return {"bytes": a["bytes"] + 36 * n, "flops": a["flops"] + 8 * 35 * n + 60 * n}
    if kind == "batch":
        parts = [_frame_work(w, h, v * 1000.0, "reference")
                 for w, h, v in mixed_population(case["sessions"], case["population"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "mapping":
        n, vis = float(case["width"] * case["height"]), _blocks(case["voxel_mm"])
        voxel = 6 if case["form"] == "precision" else 8
        return {"bytes": 23 * n + 32 * n + vis * (2 * 512 * voxel + 16), "flops": 60 * 512 * vis + 8 * 35 * n}
    if kind == "odometry":
        n = float(case["width"] * case["height"])
        return {"bytes": (4 * 16 + 2 + 4) * n, "flops": 2 * 150 * n}
    if kind == "pyramid":
        n = float(case["width"] * case["height"])
        levels = 1 + 1 / 4 + 1 / 16
        return {"bytes": 5 * n + 4 * n + (4 + 1 + 32 + 4) * n * levels, "flops": (200 + 60) * n}
    if kind == "mesh":
        # the room's surface seen by the sequence, a little more than one view
        blocks = 1.3 * _blocks(case["voxel_mm"])
        return {"bytes": blocks * 512 * (6 if case["form"] == "precision" else 8) + blocks * 68 * 3 * 27,
                "flops": blocks * 68 * 3 * 40}
    return {"bytes": (case["queries"] + case["train"]) * 256.0 + case["queries"] * 16.0,
            "flops": 3.0 * 64 * case["queries"] * case["train"]}
