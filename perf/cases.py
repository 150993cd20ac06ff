"""The work that programs on this framework have it do, as cases that can be timed.

listed() names the cases, draw() makes more of the same ranges, prepare() makes what a program
holds before the call, run() is one pass through the public entry points, exact() is the same
result in 64 bits by plain torch, and work() counts the bytes and operations that a pass cannot
do without.

The kinds of case:
    frame    a session takes its next frame, one blocking call (the reference's tracking loop)
    stream   a session takes a burst of frames through submit / wait, two in flight
    view     a session with a visualization volume takes a frame and renders the model
    batch    many equal sessions take one frame each in one step
    serve    a server holds sessions of uneven sizes; half of them have a frame this time
    pyramid  the per-stage calls that turn a raw frame into depth, vertex and normal pyramids
    raycast  the per-stage raycast of a caller's volume
    fuse     the per-stage fusion of a depth map into a caller's volume
    pose     ICP.computePose of vertex pyramids against predicted ones
    solve    one ICP residual matrix and its least-squares solution

Frames come from the package's synthetic scene (a plane, a sphere and a box with sensor noise and
dropouts).  A session goes back and forth over the first frames of the scene's 300-frame loop, so
it can take any number of passes and keeps tracking.
"""
import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.getcwd(), "kinectfusion-cuda_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)
import kfb200  # noqa: E402
from kfb200 import synth  # noqa: E402

WARM = 3      # frames that a session has taken before the first pass
LOOP = 8      # frames that a session goes back and forth over
BURST = 6     # frames of one pass of a stream case
ICP_ITERS = (10, 5, 4)
DIST_THRESH, ANGLE_THRESH = 0.1, math.radians(20.0)
STOP_ANGLE, STOP_DIST = math.radians(0.1), 0.01
MIN_DEPTH, MAX_DEPTH = 0.4, 6.0
STEP_LARGE, STEP_SMALL = 1.99, 0.1
SCALE = 1e-3


def _case(kind, w, h, n, width, mu, **kw):
    case = dict(kind=kind, w=w, h=h, n=n, width=width, mu=mu, f16=False, radius=2, sigma_s=4.5, sigma_r=0.03, levels=3,
                device=False, pinned=False, unmirror=False, vis_n=0, sessions=1, mix=0)
    case.update(kw)
    return case


def listed():
    return [
        # the plain pipeline at its small size (320x240, 128^3): latency and launches count
        _case("frame", 320, 240, 128, 2.0, 0.03, name="frame_320x240_128"),
        # the plain pipeline at full size (640x480, 512^3 over 3 m), one blocking call per frame
        _case("frame", 640, 480, 512, 3.0, 0.02, name="frame_640x480_512"),
        # the same as a capture loop drives it: pinned frames, the next handed over before the last
        # is done
        _case("stream", 640, 480, 512, 3.0, 0.02, pinned=True, name="stream_640x480_512"),
        # a depth camera's 512x424 mirrored frames, already on the device, into 16-bit voxels
        _case("frame", 512, 424, 256, 3.0, 0.03, f16=True, device=True, unmirror=True, radius=3, sigma_s=4.0,
              sigma_r=0.25, name="frame_512x424_256_f16_device"),
        # the reference's own program: 640x480, 256^3 over 8 m, a 512^3 visualization volume over
        # 5 m fused and shown every frame, its filter's 7x7 window
        _case("view", 640, 480, 256, 8.0, 3 * 8 / 255, radius=3, sigma_s=4.0, sigma_r=0.25, vis_n=512,
              name="view_640x480_256_512"),
        # 24 full-size sessions in 16-bit voxels stepped together, pinned frames
        _case("batch", 640, 480, 512, 3.0, 0.02, f16=True, pinned=True, sessions=24, name="batch_24x640x480_512_f16"),
        # a server with 16 sessions of uneven sizes (320x240 and 640x480, 128^3 to 512^3)
        _case("serve", 640, 480, 512, 3.0, 0.02, f16=True, sessions=16, mix=7, name="serve_16_mixed_f16"),
        # a program on the per-stage calls: the measurement side of a frame ...
        _case("pyramid", 640, 480, 0, 3.0, 0.02, radius=3, sigma_s=4.0, sigma_r=0.25, name="pyramid_640x480"),
        # ... the prediction from its own volume ...
        _case("raycast", 640, 480, 512, 3.0, 0.02, name="raycast_640x480_512"),
        # ... the alignment of the two ...
        _case("pose", 640, 480, 0, 3.0, 0.02, name="pose_640x480"),
        # ... and the update of the volume
        _case("fuse", 640, 480, 512, 3.0, 0.02, name="fuse_640x480_512"),
        # one ICP iteration written out by the caller, at a coarse level of odd size
        _case("solve", 161, 119, 0, 3.0, 0.02, levels=1, name="solve_161x119"),
    ]


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "stream", "view", "batch", "serve", "pyramid", "raycast", "pose", "fuse",
                       "solve"])
    w = 4 * round(math.exp(rng.uniform(math.log(40), math.log(160))))
    h = 4 * round(w / 4 * rng.choice([0.75, 0.75, 424 / 512, 0.5625]))
    n = 8 * round(math.exp(rng.uniform(math.log(8), math.log(64))))
    width = rng.choice([2.0, 3.0])
    mu = round(rng.uniform(1.9, 3.5) * width / n, 5)
    filt = rng.choice([(2, 4.5, 0.03), (3, 4.0, 0.25), (rng.randint(1, 5), 4.5, 0.03)])
    kw = dict(f16=rng.random() < 0.4, radius=filt[0], sigma_s=filt[1], sigma_r=filt[2])
    if kind in ("frame", "stream"):
        kw.update(device=kind == "frame" and rng.random() < 0.4, pinned=kind == "stream", unmirror=rng.random() < 0.3, levels=rng.choice([2, 3, 3]))
    elif kind == "view":
        kw.update(vis_n=8 * rng.randint(16, 64))
    elif kind in ("batch", "serve"):
        kw.update(f16=True, pinned=kind == "batch" and rng.random() < 0.7, sessions=rng.randint(4, 16),
                  mix=rng.randint(1, 1000) if kind == "serve" else 0)
    elif kind == "solve":
        w, h, kw["levels"] = w - rng.randint(0, 3), h - rng.randint(0, 3), 1
    if kind in ("pyramid", "pose", "solve"):
        n, kw["f16"] = 0, False
    return _case(kind, w, h, n, width, mu, **kw)


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _camera(case, level=0):
    """fx, fy, cx, cy of a pyramid level (float32 steps, as a program computes them)."""
    f = np.float32(525.0 * case["w"] / 640)
    cx, cy = np.float32(case["w"] / 2 - 0.5), np.float32(case["h"] / 2 - 0.5)
    s, half = np.float32(1.0 / (1 << level)), np.float32(0.5)
    return f * s, f * s, (cx + half) * s - half, (cy + half) * s - half


def _matrix(case, level=0):
    fx, fy, cx, cy = _camera(case, level)
    return np.array([[fx, 0, cx], [0, fy, cy], [0, 0, 1]], np.float32)


def _inverse(case, level=0):
    return np.linalg.inv(_matrix(case, level).astype(np.float64)).astype(np.float32)


def _poses(case, seed, count):
    return synth.trajectory(synth.LOOP, count, seed, min(case["width"], 3.0))


def _render(case, seed, pose, frame, level=0, noise=True):
    fx, fy, cx, cy = (float(v) for v in _camera(case, level))
    img, true = synth.render(synth.scene(min(case["width"], 3.0)), pose, case["w"] >> level, case["h"] >> level, fx, fy, cx,
                             cy, seed, frame, noise, true_depth=True)
    if case["unmirror"]:
        img = np.ascontiguousarray(img[:, ::-1])
    return img, true


def _frames(case, seed, count=LOOP):
    poses = _poses(case, seed, count)
    frames = [_render(case, seed, poses[i], i)[0] for i in range(count)]
    if case["pinned"] and torch.cuda.is_available():
        frames = [torch.from_numpy(f).pin_memory().numpy() for f in frames]
    return frames, poses


def _config(case, pose):
    fx, fy, cx, cy = (float(v) for v in _camera(case))
    return kfb200.default_config(
        width=case["w"], height=case["h"], fx=fx, fy=fy, cx=cx, cy=cy, depth_scale=SCALE, unmirror=int(case["unmirror"]),
        levels=case["levels"], iters=ICP_ITERS[:case["levels"]], dist_thresh=DIST_THRESH, angle_thresh=ANGLE_THRESH,
        bilateral_sigma_s=case["sigma_s"], bilateral_sigma_r=case["sigma_r"], bilateral_radius=case["radius"],
        volume_n=case["n"], volume_width=case["width"], mu=case["mu"],
        tsdf_format=kfb200.KF_TSDF_F16U16 if case["f16"] else kfb200.KF_TSDF_F32F32, initial_pose=pose,
        vis_volume_n=case["vis_n"], vis_volume_width=5.0, vis_mu=2 * 5.0 / max(case["vis_n"] - 1, 1))


def _members(case):
    """The configurations' cases of a batch or server: equal ones, or uneven ones of a mix."""
    if not case["mix"]:
        return [case] * case["sessions"]
    rng = np.random.default_rng(case["mix"])
    members = []
    for i in range(case["sessions"]):
        if i % 2:   # every second session at half the frame size, with a small volume
            n = 8 * int(rng.integers(min(16, case["n"] // 8), max(case["n"] // 16, 17) + 1))
            w, h = (case["w"] // 8) * 4, (case["h"] // 8) * 4
            members.append(dict(case, w=w, h=h, n=n, width=2.0, mu=max(0.03, 1.9 * 2.0 / n)))
        else:
            n = 8 * int(rng.integers(max(case["n"] * 3 // 32, 8), max(case["n"] // 8, 8) + 1))
            members.append(dict(case, n=n, mu=max(case["mu"], 1.9 * case["width"] / n)))
    return members


class _Memory:
    """A device array that a session owns, for torch to read in place; keeps the session."""

    def __init__(self, address, n, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n, n, n), "typestr": kind, "data": (address, False), "version": 2}


def _grid(volume, owner):
    """The distance and weight arrays of a session's volume (16-bit weights as their bits)."""
    kinds = ("<f2", "<i2") if volume.format == kfb200.KF_TSDF_F16U16 else ("<f4", "<f4")
    return [torch.as_tensor(_Memory(a, volume.n, k, owner), device="cuda") for a, k in zip((volume.f, volume.w), kinds)]


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------------------------------
# the stages in 64 bits
# ------------------------------------------------------------------------------------------
def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=_device())


def _valid(d):
    return (d > 0.01) & torch.isfinite(d)


def _pyramid64(case, raw):
    """Unfiltered metres, and depth and vertex maps (x, y, z, tag) of every level."""
    d = torch.as_tensor(raw.astype(np.float32), device=_device()).half().double() * float(np.float32(SCALE))
    if case["unmirror"]:
        d = d.flip(1)
    r, h, w = case["radius"], case["h"], case["w"]
    pad = torch.nn.functional.pad(d[None, None], (r, r, r, r), mode="replicate")[0, 0]
    total, acc = torch.zeros_like(d), torch.zeros_like(d)
    ss, sr = float(np.float32(case["sigma_s"])), float(np.float32(case["sigma_r"]))
    for x in range(-r, r + 1):
        for y in range(-r, r + 1):
            cur = pad[r + y:r + y + h, r + x:r + x + w]
            e = torch.exp(-(x * x + y * y) / ss ** 2 - ((d - cur) / sr) ** 2)
            total += e
            acc += e * cur
    depths = [acc / total]
    for _ in range(case["levels"] - 1):
        a, b, c, e = (depths[-1][i::2, j::2] for i, j in ((0, 0), (0, 1), (1, 0), (1, 1)))
        total, count = a.clone(), torch.ones_like(a)
        for o in (b, c, e):
            near = (a - o).abs() <= 3 * sr
            total += torch.where(near, o, torch.zeros_like(o))
            count += near
        depths.append(total / count)
    return d, depths, [_vertices64(case, z, level) for level, z in enumerate(depths)]


def _rays64(h, w, inverse):
    j, i = torch.meshgrid(torch.arange(h, device=_device()), torch.arange(w, device=_device()), indexing="ij")
    return torch.stack([i + 0.5, j + 0.5, torch.ones_like(i)], -1).double() @ _t(inverse).T


def _vertices64(case, depth, level, pose=None):
    ok = _valid(depth)
    v = _rays64(*depth.shape, np.linalg.inv(_matrix(case, level).astype(np.float64))) * depth[..., None]
    if pose is not None:
        v = v @ _t(pose[:3, :3]).T + _t(pose[:3, 3])
    v = torch.where(ok[..., None], v, torch.zeros_like(v))
    return torch.cat([v, torch.where(ok, -1.0, -2.0)[..., None].double()], -1)


def _normals64(v):
    """Normalised cross products of the neighbours to the right and below (x, y, z, tag)."""
    p, ok = v[..., :3], v[..., 3] == -1
    n = torch.cross(p[:-1, 1:] - p[:-1, :-1], p[1:, :-1] - p[:-1, :-1], dim=-1)
    n = n / n.norm(dim=-1, keepdim=True)
    ok = ok[:-1, :-1] & ok[:-1, 1:] & ok[1:, :-1]
    out = torch.zeros_like(v)
    out[..., 3] = -2
    out[:-1, :-1, :3] = torch.where(ok[..., None], n, torch.zeros_like(n))
    out[:-1, :-1, 3] = torch.where(ok, -1.0, -2.0).double()
    return out


def _axes(n, width):
    """Voxel coordinates as the volume's layout defines them: x = y in float steps from the edge,
    z accumulated in float."""
    res, base = np.float32(width) / np.float32(n - 1), np.float32(-width * 0.5)
    x = base + np.arange(n, dtype=np.float32) * res
    z = np.cumsum(np.concatenate([[base + (-res)], np.full(n, res, np.float32)]), dtype=np.float32)[1:]
    return _t(x), _t(z)


def _fuse64(F, W, width, mu, depth, K, pose, max_weight=0.0):
    """One depth map into the volume (float64 distances and weights, [z, y, x]), in place."""
    n, (h, w) = F.shape[0], depth.shape
    xs, zs = _axes(n, width)
    R, t = _t(pose[:3, :3]), _t(pose[:3, 3])
    fx, fy, cx, cy = (float(K[i, j]) for i, j in ((0, 0), (1, 1), (0, 2), (1, 2)))
    mu, flat = float(np.float32(mu)), depth.reshape(-1)
    slab = max(1, (1 << 24) // (n * n))
    for k in range(0, n, slab):
        q = [zs[k:k + slab, None, None] - t[2], xs[None, :, None] - t[1], xs[None, None, :] - t[0]]
        ex, ey, ez = (R[0, a] * q[2] + R[1, a] * q[1] + R[2, a] * q[0] for a in range(3))
        px, py = fx * ex / ez + cx, fy * ey / ez + cy
        ok = (ez >= MIN_DEPTH) & (ez < MAX_DEPTH) & (px >= 0) & (px < w) & (py >= 0) & (py < h)
        at = torch.where(ok, py.floor() * w + px.floor(), torch.zeros_like(px)).long()
        d = flat[at]
        diff = d - ez
        ok &= _valid(d) & (diff >= -mu)
        f, g = F[k:k + slab], W[k:k + slab]
        new = 1.0 / torch.where(ok, d, torch.ones_like(d))
        fused = (f * g + (diff / mu).clamp(max=1.0) * new) / (g + new)
        f.copy_(torch.where(ok, fused, f))
        g.copy_(torch.where(ok, g + new, g))


def _empty64(n):
    return torch.full((n, n, n), 2.0, device=_device(), dtype=torch.float64), \
        torch.zeros((n, n, n), device=_device(), dtype=torch.float64)


def _sample64(f, p):
    """Trilinear samples at texel coordinates p (..., 3), clamped at the edges."""
    n = f.shape[0]
    base = p.floor()
    a, i = p - base, base.long()
    lo, hi = i.clamp(0, n - 1), (i + 1).clamp(0, n - 1)
    flat, out = f.reshape(-1), 0.0
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                x, y, z = (hi if dx else lo)[..., 0], (hi if dy else lo)[..., 1], (hi if dz else lo)[..., 2]
                weight = 1.0
                for axis, up in ((0, dx), (1, dy), (2, dz)):
                    weight = weight * (a[..., axis] if up else 1 - a[..., axis])
                out = out + weight * flat[(z * n + y) * n + x].double()
    return out


def _raycast64(f, width, mu, pose, inverse, h, w, outside=-2.0):
    """Vertex and normal maps (x, y, z, tag) of the march: steps of 1.99 mu, steps of 0.1 mu from
    the first sample below 0.99 (or mu before the first negative one) to the first negative one.
    `outside`: the tag of rays that do not meet the volume's box."""
    n, width, mu = f.shape[0], float(np.float32(width)), float(np.float32(mu))
    dirs = _rays64(h, w, inverse).reshape(-1, 3) @ _t(pose[:3, :3]).T
    o = _t(pose[:3, 3])
    t0, t1 = (-width / 2 - o) / dirs, (width / 2 - o) / dirs
    enter, leave = torch.minimum(t0, t1).amax(-1), torch.maximum(t0, t1).amin(-1)
    leave = torch.where(leave < enter, torch.full_like(leave, -1.0), leave)
    near, far = enter.clamp(min=MIN_DEPTH), leave.clamp(max=MAX_DEPTH)
    met = (leave >= 0) & (near < far)

    def value(rows, t):
        return _sample64(f, (o + dirs[rows][:, None] * t[..., None]) * (n / width) + (0.5 * n - 0.5))

    large, small, ahead = mu * STEP_LARGE, mu * STEP_SMALL, 32
    hit = torch.zeros_like(near)
    rows = met.nonzero()[:, 0]
    base, idx, prev = near[rows].clone(), torch.zeros_like(rows), torch.zeros_like(near[rows])
    fine = torch.zeros_like(rows, dtype=torch.bool)
    k = torch.arange(ahead, device=base.device)
    while rows.numel():
        inc = torch.where(fine, small, large)
        t = base[:, None] + (idx[:, None] + k) * inc[:, None]
        inside = t < far[rows][:, None]
        s = torch.where(inside, value(rows, t), torch.ones_like(t))
        event = inside & ((s < 0) | (~fine[:, None] & (s < 0.99)))
        any_event = event.any(1)
        e = torch.where(any_event, event.int().argmax(1), torch.full_like(rows, ahead - 1))
        te, se = t.gather(1, e[:, None])[:, 0], s.gather(1, e[:, None])[:, 0]
        before = torch.where(e > 0, s.gather(1, (e - 1).clamp(min=0)[:, None])[:, 0], prev)
        negative = any_event & (se < 0)
        done = (negative & (te == near[rows])) | (~any_event & ~inside[:, -1])
        found = negative & fine & ~done
        hit[rows[found]] = (te - small * before / (se - before))[found]
        done |= found
        begin = any_event & ~fine & ~done
        base = torch.where(begin, torch.where(negative, te - mu, te), base)
        prev = torch.where(negative, before, se)
        idx = torch.where(begin, torch.ones_like(idx), idx + ahead)
        fine = fine | begin
        keep = ~done
        rows, base, idx, prev, fine = rows[keep], base[keep], idx[keep], prev[keep], fine[keep]
    p = o + dirs * hit[:, None]
    x, step = p * (n / width) + (0.5 * n - 0.5), mu * 0.5 / width
    g = torch.stack([_sample64(f, x - s) - _sample64(f, x + s)
                     for s in torch.eye(3, device=x.device, dtype=x.dtype) * step * n], -1) / step
    length = g.norm(dim=-1)
    ok = (hit != 0) & _valid(length)
    tag = torch.where(ok, -1.0, torch.where(met, -2.0, outside)).double()[:, None]
    zero = torch.zeros_like(p)
    v = torch.cat([torch.where(ok[:, None], p, zero), tag], -1).reshape(h, w, 4)
    return v, torch.cat([torch.where(ok[:, None], g / length[:, None], zero), tag], -1).reshape(h, w, 4)


def _rows64(v, tv, tn, K, before, R, t):
    """Point-to-plane rows A (h w x 6) and b of one ICP iteration; zero rows where rejected."""
    h, w = v.shape[:2]
    Rp, tp = _t(before[:3, :3]), _t(before[:3, 3])
    s = v[..., :3] @ R.T + t
    q = (s - tp) @ (_t(K) @ Rp.T).T
    u, r = (q[..., 0] / q[..., 2]).floor(), (q[..., 1] / q[..., 2]).floor()
    ok = (v[..., 3] == -1) & (u >= 0) & (r >= 0) & (u < w) & (r < h)
    at = torch.where(ok, r * w + u, torch.zeros_like(u)).long()
    d, m = tv.reshape(-1, 4)[at], tn.reshape(-1, 4)[at]
    src = _normals64(v)
    ok &= (d[..., 3] == -1) & (m[..., 3] == -1) & (src[..., 3] == -1)
    ok &= ~((s - d[..., :3]).norm(dim=-1) > float(np.float32(DIST_THRESH)))
    ok &= ~(((src[..., :3] @ R.T) * m[..., :3]).sum(-1) < math.cos(float(np.float32(ANGLE_THRESH))))
    A = torch.cat([torch.cross(m[..., :3], s, dim=-1), m[..., :3]], -1)
    b = ((d[..., :3] - s) * m[..., :3]).sum(-1)
    return torch.where(ok[..., None], A, torch.zeros_like(A)).reshape(-1, 6), torch.where(ok, b, torch.zeros_like(b)).reshape(-1)


def _least64(A, b):
    return torch.linalg.solve(A.T @ A, A.T @ b)


def _pose64(case, vmaps, tv, tn, pose):
    R, t = _t(pose[:3, :3]), _t(pose[:3, 3])
    one = torch.full_like(t, 1 / math.sqrt(3))
    for level in reversed(range(case["levels"])):
        for _ in range(ICP_ITERS[level]):
            x = _least64(*_rows64(vmaps[level], tv[level], tn[level], _matrix(case, level), pose, R, t))
            (sx, sy, sz), (cx, cy, cz) = x[:3].sin().tolist(), x[:3].cos().tolist()
            turn = _t([[cy, 0, sy], [0, 1, 0], [-sy, 0, cy]]) @ _t([[1, 0, 0], [0, cx, -sx], [0, sx, cx]]) @ \
                _t([[cz, -sz, 0], [sz, cz, 0], [0, 0, 1]])
            R1, t1 = turn.T @ R, turn.T @ t + x[3:]
            angle, dist = ((R1 - R) @ one).norm(), (t1 - t).norm()
            R, t = R1, t1
            if angle < float(np.float32(STOP_ANGLE)) and dist < float(np.float32(STOP_DIST)):
                break
    out = np.eye(4)
    out[:3, :3], out[:3, 3] = R.cpu().numpy(), t.cpu().numpy()
    return out


class _Session64:
    """The per-frame pipeline in 64 bits."""

    def __init__(self, case, pose):
        self.case, self.pose, self.first = case, np.asarray(pose, np.float64), True
        self.grids = [(_empty64(case["n"]), case["width"], case["mu"])]
        if case["vis_n"]:
            self.grids.append((_empty64(case["vis_n"]), 5.0, 2 * 5.0 / (case["vis_n"] - 1)))

    def frame(self, raw):
        case = self.case
        metres, _, vmaps = _pyramid64(case, raw)
        if not self.first:
            (F, _), width, mu = self.grids[0]
            maps = [_raycast64(F, width, mu, self.pose, np.linalg.inv(_matrix(case, lv).astype(np.float64)), *v.shape[:2])
                    for lv, v in enumerate(vmaps)]
            self.pose = _pose64(case, vmaps, [m[0] for m in maps], [m[1] for m in maps], self.pose)
        self.first = False
        for (F, W), width, mu in self.grids:
            _fuse64(F, W, width, mu, metres, _matrix(case), self.pose)
        return self.pose

    def state(self):
        grids = []
        for (F, W), _, _ in self.grids:
            grids += [F, None if self.case["f16"] else W]
        return grids


# ------------------------------------------------------------------------------------------
# prepare, run, exact
# ------------------------------------------------------------------------------------------
def _next(state):
    """The index of the next frame, back and forth over the LOOP frames."""
    at = state["at"] % (2 * LOOP - 2)
    state["at"] += 1
    return at if at < LOOP else 2 * LOOP - 2 - at


def _volume_before(case, seed):
    """A volume that holds two frames (in the case's storage), the third frame's depth and poses."""
    frames, poses = _frames(case, seed, 3)
    F, W = _empty64(case["n"])
    metres = [torch.as_tensor(f.astype(np.float32), device=_device()).half().float() * np.float32(SCALE) for f in frames]
    for k in (0, 1):
        _fuse64(F, W, case["width"], case["mu"], metres[k].double(), _matrix(case), poses[k])
    if case["f16"]:
        return F.half(), (W * 1024).round().clamp(max=65535).int(), metres[2], poses
    return F.float(), W.float(), metres[2], poses


def _maps_before(case, seed):
    """Vertex pyramid of a frame, the predicted pyramids of the one before, and its pose."""
    levels = range(case["levels"])
    poses = _poses(case, seed, 3)
    raw = _render(case, seed, poses[2], 2)[0]
    vmaps = [v.float() for v in _pyramid64(case, raw)[2]]
    tv = [_vertices64(case, _t(_render(case, seed, poses[1], 1, lv, noise=False)[1]), lv, poses[1]) for lv in levels]
    return vmaps, [v.float() for v in tv], [_normals64(v).float() for v in tv], poses[1]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "stream", "view"):
        frames, poses = _frames(case, seed)
        if case["device"]:
            frames = [_gpu(f) for f in frames]
        s = kfb200.KinectFusion(_config(case, poses[0]))
        for f in frames[:WARM]:
            s.process_frame(f)
        return {"kind": kind, "s": s, "frames": frames, "at": WARM, "view": poses[0],
                "grids": _grid(s.volume(), s) + (_grid(s.vis_volume(), s) if case["vis_n"] else [])}
    if kind in ("batch", "serve"):
        members = _members(case)
        rendered, frames, configs = {}, [], []
        for i, m in enumerate(members):   # four sequences of each frame size
            key = (m["w"], m["h"], m["width"], i % 4 if not case["mix"] else (i // 2) % 4)
            if key not in rendered:
                rendered[key] = _frames(m, seed + 101 * key[3])
            frames.append(rendered[key][0])
            configs.append(_config(m, rendered[key][1][0]))
        if kind == "batch":
            b = kfb200.Batch(configs)
            for k in range(WARM):
                b.step([f[k] for f in frames])
            sessions = [b.session(i) for i in range(len(members))]
            return {"kind": kind, "b": b, "frames": frames, "at": WARM,
                    "grids": [g for s in sessions for g in _grid(s.volume(), s)]}
        srv = kfb200.Server(len(members), 100 << 30)
        ids = [srv.open(c) for c in configs]
        for k in range(WARM):
            for i, f in zip(ids, frames):
                srv.submit(i, f[k])
            srv.step()
        sessions = [srv.session(i) for i in ids]
        return {"kind": kind, "srv": srv, "ids": ids, "frames": frames, "at": 2 * WARM,
                "grids": [g for s in sessions for g in _grid(s.volume(), s)]}
    if kind == "pyramid":
        frames, _ = _frames(case, seed, 1)
        sizes = [(case["h"] >> lv, case["w"] >> lv) for lv in range(case["levels"])]
        new = lambda shape: torch.zeros(shape, device="cuda")   # noqa: E731
        return {"kind": kind, "raw": _gpu(frames[0]), "filter": (case["sigma_s"], case["sigma_r"], case["radius"]),
                "metres": new(sizes[0]), "depth": [new(z) for z in sizes], "vertex": [new(z + (4,)) for z in sizes],
                "normal": [new(z + (4,)) for z in sizes], "inverse": [_inverse(case, lv) for lv in range(case["levels"])]}
    fmt = kfb200.KF_TSDF_F16U16 if case["f16"] else kfb200.KF_TSDF_F32F32
    if kind in ("raycast", "fuse"):
        F, W, metres, poses = _volume_before(case, seed)
        if case["f16"]:   # 16-bit weights, held as the bits of int16
            W = torch.where(W > 32767, W - 65536, W).short()
        vol = kfb200.kernel.volume(F, W, case["width"], case["mu"], fmt)
        state = {"kind": kind, "vol": vol, "F": F, "W": W, "metres": metres, "pose": poses[2], "K": _matrix(case),
                 "inverse": _inverse(case)}
        if kind == "raycast":
            state.update(v=torch.zeros((case["h"], case["w"], 4), device="cuda"),
                         n=torch.zeros((case["h"], case["w"], 4), device="cuda"))
        return state
    vmaps, tv, tn, pose = _maps_before(case, seed)
    state = {"kind": kind, "v": [v.contiguous() for v in vmaps], "tv": tv, "tn": tn, "pose": pose}
    if kind == "pose":
        state["icp"] = kfb200.ICP(_config(dict(case, n=64), pose))
    else:
        rows = case["w"] * case["h"]
        state.update(K=_matrix(case), A=torch.zeros((rows, 6), device="cuda"), b=torch.zeros(rows, device="cuda"), rows=rows,
                     lls=kfb200.LinearLeastSquares())
    return state


def run(state):
    kind = state["kind"]
    if kind == "frame":
        status, pose = state["s"].process_frame(state["frames"][_next(state)])
        return {"status": status, "pose": pose, "grids": state["grids"]}
    if kind == "stream":
        s, poses, flying = state["s"], [], 0
        for _ in range(BURST):
            s.submit_frame(state["frames"][_next(state)])
            flying += 1
            if flying == 2:
                poses.append(s.wait_frame()[1])
                flying -= 1
        while flying:
            poses.append(s.wait_frame()[1])
            flying -= 1
        return {"poses": poses, "grids": state["grids"]}
    if kind == "view":
        status, pose = state["s"].process_frame(state["frames"][_next(state)])
        return {"status": status, "pose": pose, "image": state["s"].render(kfb200.KF_RENDER_NORMALS, state["view"]),
                "grids": state["grids"]}
    if kind == "batch":
        k = _next(state)
        status, poses = state["b"].step([f[k] for f in state["frames"]])
        return {"status": status, "poses": poses, "grids": state["grids"]}
    if kind == "serve":
        srv, half = state["srv"], state["at"] % 2
        k = (state["at"] // 2) % (2 * LOOP - 2)
        k = k if k < LOOP else 2 * LOOP - 2 - k
        state["at"] += 1
        mine = [x for i, x in enumerate(zip(state["ids"], state["frames"])) if i // 2 % 2 == half]
        for i, f in mine:
            srv.submit(i, f[k])
        srv.step()
        return {"poses": [srv.result(i)[0] for i, _ in mine], "grids": state["grids"]}
    kernel = kfb200.kernel
    if kind == "pyramid":
        sigma_s, sigma_r, radius = state["filter"]
        depth, vertex, normal = state["depth"], state["vertex"], state["normal"]
        kernel.convertToDepthMeters(state["raw"], state["metres"], SCALE)
        kernel.applyBilateralFilter(state["metres"], depth[0], sigma_s, sigma_r, radius)
        for lv in range(1, len(depth)):
            kernel.downSample(depth[lv - 1], depth[lv], sigma_r)
        for lv, inverse in enumerate(state["inverse"]):
            kernel.createVertexMap(depth[lv], vertex[lv], inverse)
            kernel.createNormalMap(vertex[lv], normal[lv])
        return {"metres": state["metres"], "depth": depth, "vertex": vertex, "normal": normal}
    if kind == "raycast":
        kernel.raycast(state["vol"], state["pose"], state["inverse"], state["v"], state["n"])
        return {"vertex": state["v"], "normal": state["n"]}
    if kind == "fuse":
        kernel.fuse(state["metres"], state["vol"], state["pose"], state["K"])
        return {"grids": [state["F"], state["W"]]}
    if kind == "pose":
        status, pose, iters = state["icp"].computePose(state["v"], state["tv"], state["tn"], state["pose"])
        return {"status": status, "pose": pose, "iters": iters}
    pose = state["pose"]
    kernel.constructIcpResiduals(state["v"][0], state["tv"][0], state["tn"][0], pose[:3, :3], pose[:3, 3], pose[:3, :3],
                                 pose[:3, 3], state["K"], DIST_THRESH, ANGLE_THRESH, state["A"], state["b"])
    return {"A": state["A"], "b": state["b"], "x": state["lls"].solve(state["A"], state["b"], state["rows"])}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        return None   # dozens of sessions' frames in 64 bits take too long
    if kind in ("frame", "stream", "view"):
        frames, poses = _frames(case, seed)
        s = _Session64(case, poses[0])
        for f in frames[:WARM]:
            s.frame(f)
        state = {"at": WARM}
        if kind == "stream":
            return {"poses": [s.frame(frames[_next(state)]) for _ in range(BURST)], "grids": s.state()}
        out = {"status": None, "pose": s.frame(frames[_next(state)]), "grids": s.state()}
        return dict(out, image=None) if kind == "view" else out
    if kind == "pyramid":
        metres, depths, vmaps = _pyramid64(case, _frames(case, seed, 1)[0][0])
        return {"metres": metres, "depth": depths, "vertex": vmaps, "normal": [_normals64(v) for v in vmaps]}
    if kind in ("raycast", "fuse"):
        F, W, metres, poses = _volume_before(case, seed)
        if kind == "raycast":
            v, n = _raycast64(F, case["width"], case["mu"], poses[2], _inverse(case), case["h"], case["w"], outside=0.0)
            return {"vertex": v, "normal": n}
        F, W = F.double(), W.double() / 1024 if case["f16"] else W.double()
        _fuse64(F, W, case["width"], case["mu"], metres.double(), _matrix(case), poses[2])
        return {"grids": [F, None if case["f16"] else W]}
    vmaps, tv, tn, pose = _maps_before(case, seed)
    vmaps, tv, tn = ([m.double() for m in maps] for maps in (vmaps, tv, tn))
    if kind == "pose":
        return {"status": None, "pose": _pose64(case, vmaps, tv, tn, pose.astype(np.float64)), "iters": None}
    A, b = _rows64(vmaps[0], tv[0], tn[0], _matrix(case), pose, _t(pose[:3, :3]), _t(pose[:3, 3]))
    return {"A": A, "b": b, "x": _least64(A, b)}


# ------------------------------------------------------------------------------------------
# work
# ------------------------------------------------------------------------------------------
def _updated(case, n, width, mu):
    """Voxels of an n^3 volume that a frame updates, counted on a coarse grid."""
    coarse = 48
    pose = _poses(case, 1, 1)[0].astype(np.float64)
    depth = _render(dict(case, unmirror=False), 1, pose.astype(np.float32), 0, noise=False)[1]
    x = (np.arange(coarse) + 0.5) / coarse * width - width / 2
    z, y, x = np.meshgrid(x, x, x, indexing="ij")
    p = np.stack([x, y, z], -1).reshape(-1, 3)
    e = (p - pose[:3, 3]) @ pose[:3, :3]
    fx, fy, cx, cy = (float(v) for v in _camera(case))
    front = e[:, 2] > MIN_DEPTH
    e = e[front]
    u, v = np.floor(fx * e[:, 0] / e[:, 2] + cx), np.floor(fy * e[:, 1] / e[:, 2] + cy)
    ok = (u >= 0) & (v >= 0) & (u < case["w"]) & (v < case["h"])
    d = depth[v[ok].astype(int), u[ok].astype(int)]
    return n ** 3 * float(np.mean(np.concatenate([(d > 0) & (d < 4) & (d - e[ok, 2] >= -mu), np.zeros(p.shape[0] - ok.sum())])))


def work(case):
    """A frame reads its 16-bit image once and reads and writes each voxel that it updates (the
    raycast's voxels are among them); pyramids and predicted maps can stay on the chip.  Per-stage
    calls read and write whole maps.  Operations: about 8 per filter tap, 60 per pixel and level of
    the march's surface samples, 90 per pixel and ICP iteration (two a level), 40 per voxel."""
    kind, px = case["kind"], case["w"] * case["h"]
    pyramid = sum(0.25 ** lv for lv in range(case["levels"]))
    if kind in ("batch", "serve"):
        parts = [work(dict(m, kind="frame")) for m in _members(case)]
        share = 0.5 if kind == "serve" else 1.0
        return {k: share * sum(p[k] for p in parts) for k in ("bytes", "flops")}
    taps = 8.0 * px * (2 * case["radius"] + 1) ** 2
    icp = 2 * 90.0 * px * pyramid
    voxel = 4 if case["f16"] else 8
    if kind in ("frame", "stream", "view"):
        voxels = _updated(case, case["n"], case["width"], case["mu"])
        if case["vis_n"]:
            voxels += _updated(case, case["vis_n"], 5.0, 0.02)
        image = 4.0 * px if kind == "view" else 0.0
        times = BURST if kind == "stream" else 1
        return {"bytes": times * (2.0 * px + 2 * voxel * voxels + image),
                "flops": times * (taps + 600.0 * px * pyramid + icp + 40.0 * voxels)}
    if kind == "pyramid":
        return {"bytes": px * (2 + 4) + px * pyramid * (4 + 16 + 16), "flops": taps + 40.0 * px * pyramid}
    if kind == "raycast":   # at least the eight taps of the samples either side of each hit, once
        return {"bytes": 32.0 * px + 2 * 8 * (voxel / 2) * px, "flops": 600.0 * px}
    if kind == "fuse":
        voxels = _updated(case, case["n"], case["width"], case["mu"])
        return {"bytes": 4.0 * px + 2 * voxel * voxels, "flops": 40.0 * voxels}
    if kind == "pose":
        return {"bytes": 48.0 * px * pyramid, "flops": icp}
    return {"bytes": 48.0 * px + 28.0 * px, "flops": 140.0 * px}
