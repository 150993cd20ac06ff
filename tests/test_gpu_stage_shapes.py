"""Per-stage calls at the sizes where their work splits can go wrong -- the smallest and ragged
volumes, frames that no tile divides, non-finite depths -- against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dev(torch, a):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).cuda()


def depth_frames(kf, orc, w, h, unit):
    """Two metre maps (times unit) of the synthetic loop with their poses, and K; the second map
    holds zeros, a NaN and infinities too."""
    from kfb200 import synth
    cfg = kf.config_small(width=w, height=h, fx=262.5 * w / 320, fy=262.5 * w / 320, cx=w / 2 - 0.5, cy=h / 2 - 0.5)
    imgs, poses = synth.sequence(cfg, 42, seed=9, kind=synth.LOOP)
    maps, out = [], []
    for i in (38, 41):
        maps.append(orc.convert(imgs[i], 1e-3) * np.float32(unit))
        p = poses[i].copy()
        p[:3, 3] *= unit
        out.append(p)
    maps[1][h // 2, :3] = [np.nan, np.inf, -np.inf]
    return cfg, maps, out, kf.level_intrinsics(cfg, 0)


@pytest.mark.parametrize("n,w,h,fmt,unit", [(8, 33, 17, 0, 1.0), (40, 161, 119, 0, 1.0), (72, 160, 120, 1, 1.0),
                                            (136, 321, 241, 0, 1.0), (136, 320, 240, 1, 1.0), (64, 320, 240, 0, 1000.0)])
def test_fuse_shapes(kf, orc, cuda, n, w, h, fmt, unit):
    """Two frames fused, at the oracle's state.  The second frame's values agree to 1e-3 of the
    truncation distance (f16: plus the storage rounding 2^-10 of a value up to 1 and of the
    weights' steps) except where a projection within float rounding of a pixel edge, the depth
    range or the update limit picks otherwise: at most 0.5 % of the touched voxels, or three
    voxels of the smallest volumes."""
    _, maps, poses, k = depth_frames(kf, orc, w, h, unit)
    width, mu = 2.0 * unit, max(0.03, 3.0 / n) * unit
    f = np.full((n, n, n), 2.0, np.float32)
    wt = np.zeros((n, n, n), np.float32)
    rng = dict(min_d=0.4 * unit, max_d=6.0 * unit)
    orc.fuse(maps[0], k, f, wt, width, mu, poses[0], prec=1, **rng)
    if fmt:
        f = f.astype(np.float16).astype(np.float32)
        wq = np.minimum(np.rint(wt * kf.KF_WEIGHT_SCALE), 65535).astype(np.uint16)
        wt = wq.astype(np.float32) / np.float32(kf.KF_WEIGHT_SCALE)
        ft, wd = dev(cuda, f.astype(np.float16)), dev(cuda, wq)
    else:
        ft, wd = dev(cuda, f), dev(cuda, wt)
    vol = kf.kernel.volume(ft, wd, width, mu, fmt=fmt)
    kf.kernel.fuse(dev(cuda, maps[1]), vol, poses[1], k, min_depth=rng["min_d"], max_depth=rng["max_d"])
    fo, wo = f.copy(), wt.copy()
    orc.fuse(maps[1], k, fo, wo, width, mu, poses[1], prec=1, **rng)
    gf = ft.cpu().numpy().astype(np.float32)
    gw = wd.cpu().numpy()
    gw = gw.view(np.uint16).astype(np.float32) / np.float32(kf.KF_WEIGHT_SCALE) if fmt else gw
    touched = (wo != wt) | (gw != wt)
    tol_f, tol_w = (2e-3, 0.5 / kf.KF_WEIGHT_SCALE + 1e-6) if fmt else (1e-3, 1e-5 * max(1.0, float(wo.max())))
    bad = touched & ((np.abs(gf - fo) > tol_f) | (np.abs(gw - wo) > tol_w))
    assert int(bad.sum()) <= max(3, 0.005 * int(touched.sum())), (int(bad.sum()), int(touched.sum()))
    assert n == 8 or touched.sum() > 100


def plain_raycast(kf, cuda, vol, pose, ik, v, n, step, depths):
    """kf_raycast under stream capture, replayed once: a captured call marches every ray in its own
    thread, without bounds, scratch or queue."""
    import ctypes
    h, w = v.shape[:2]
    s = cuda.cuda.Stream()
    cuda.cuda.synchronize()
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g, stream=s):
        st = kf.lib.kf_raycast(ctypes.byref(vol), kf.to_colmajor(pose), kf.to_colmajor(ik),
                               ctypes.c_void_p(v.data_ptr()), w, h, ctypes.c_void_p(n.data_ptr()), w, h, depths[0],
                               depths[1], step[0], step[1], ctypes.c_void_p(s.cuda_stream), None)
        assert st == kf.KF_OK
    g.replay()
    cuda.cuda.synchronize()


SKEW = np.array([[1.02, 0.01, 0], [-0.02, 0.97, 0.03], [0, 0.01, 1.05]], np.float32)   # not a rotation
VIEWS = {"loop": None, "inside": (0.1, 0.1, 0.35), "away": (3.0, 0.0, 4.0), "mirrored": None}


@pytest.mark.parametrize("n,w,h,fmt,view", [(8, 33, 17, 0, "loop"), (40, 161, 119, 1, "loop"), (72, 401, 401, 0, "loop"),
                                            (136, 500, 330, 1, "loop"), (136, 500, 330, 0, "inside"),
                                            (136, 500, 330, 0, "away"), (136, 500, 330, 0, "mirrored"),
                                            (136, 500, 331, 0, "unaligned"), (512, 640, 480, 0, "loop"),
                                            (256, 160, 120, 1, "inside"), (200, 500, 330, 0, "inside"),
                                            (200, 500, 330, 1, "away"), (200, 500, 330, 0, "mirrored"),
                                            (264, 501, 331, 0, "loop"), (200, 500, 330, 0, "skewed")])
def test_raycast_paths_agree(kf, orc, cuda, n, w, h, fmt, view):
    """A call with scratch (bounds from one read of the visible volume, or none; ray tiles; long
    rays by warps) gives the maps of the call without any, bit for bit: skipping and queueing
    change which samples are evaluated where, not a sample's value or its test."""
    _, maps, poses, k = depth_frames(kf, orc, w, h, 1.0)
    width, mu = 2.0, max(0.01, 3.0 / n)
    f = cuda.full((n, n, n), 2.0, device="cuda")
    wt = cuda.zeros((n, n, n), device="cuda")
    vol = kf.kernel.volume(f, wt, width, mu)
    for m, p in zip(maps, poses):
        kf.kernel.fuse(dev(cuda, m), vol, p, k)
    if fmt:
        f, wt = f.half(), wt.short()
        vol = kf.kernel.volume(f, wt, width, mu, fmt=fmt)
    if view == "unaligned":
        room = cuda.zeros(n ** 3 + 1, device="cuda")
        room[1:] = f.reshape(-1)
        vol.f = room.data_ptr() + 4
    pose, depths = poses[1].copy(), (0.4, 6.0)
    if view == "inside":
        pose[:3, 3] = VIEWS[view]
        depths = (0.0, 6.0)
    elif view == "away":
        pose[:3, 3] = VIEWS[view]
    ik = np.linalg.inv(k.astype(np.float64)).astype(np.float32)
    if view == "skewed":
        pose[:3, :3] = pose[:3, :3] @ SKEW
    if view == "mirrored":
        ik = ik @ np.array([[-1, 0, w], [0, 1, 0], [0, 0, 1]], np.float32)
    out = [[cuda.full((h, w, 4), 7.0, device="cuda") for _ in range(2)] for _ in range(2)]
    kf.kernel.raycast(vol, pose, ik, *out[0], min_depth=depths[0], max_depth=depths[1])
    plain_raycast(kf, cuda, vol, pose, ik, *out[1], (1.99, 0.1), depths)
    for a, b in zip(*out):
        assert cuda.equal(a.view(cuda.int32), b.view(cuda.int32))
    hits = float((out[0][0][..., 3] == -1).float().mean())
    assert hits > 0.05 or n == 8 or view in ("away", "inside"), hits


@pytest.mark.parametrize("n,w,h,fmt,levels", [(192, 320, 240, 0, 3), (200, 164, 124, 1, 3), (264, 500, 330, 0, 2)])
def test_session_depth_ranges_change_nothing(kf, cuda, n, w, h, fmt, levels):
    """A session's raycast, whose rays start and end by their tile's depth range, equals the march
    of every sample (plain_raycast) bit for bit at every level: at the tracked pose, at one that is
    not exactly a rotation, looking across the volume from inside it, and looking away."""
    from kfb200 import synth
    cfg = kf.config_small(width=w, height=h, fx=262.5 * w / 320, fy=262.5 * w / 320, cx=w / 2 - 0.5, cy=h / 2 - 0.5,
                          levels=levels, volume_n=n, mu=0.03, tsdf_format=fmt, keep_on_miss=0, min_depth=0.05)
    imgs, _ = synth.sequence(cfg, 4, seed=5, kind=synth.LOOP)
    s = kf.KinectFusion(cfg)
    for img in imgs[:3]:
        s.process_frame(img)
    tracked = s.pose()
    poses = [tracked, tracked.copy(), tracked.copy(), tracked.copy()]
    poses[1][:3, :3] = poses[1][:3, :3] @ SKEW
    poses[2][:3, 3] = (0.1, 0.1, 0.0)
    poses[2][:3, :3] = np.array([[0, 0, 1], [0, 1, 0], [-1, 0, 0]], np.float32)
    poses[3][:3, 3] = (3.0, 0.0, 4.0)
    for pose in poses:
        f, wt = s.tsdf()
        ft = cuda.from_numpy(f).cuda()
        ft = ft.half() if fmt else ft
        vol = kf.kernel.volume(ft, cuda.zeros_like(ft), cfg.volume_width, cfg.mu, fmt=fmt)
        s.set_pose(pose)
        s.process_frame(imgs[3])
        for level in range(levels):
            wl, hl = w >> level, h >> level
            want = [cuda.zeros((hl, wl, 4), device="cuda") for _ in range(2)]
            for m in want:
                m[..., 3] = -2
            plain_raycast(kf, cuda, vol, pose, kf.level_inverse_intrinsics(cfg, level), *want,
                          (cfg.step_large, cfg.step_small), (cfg.min_depth, cfg.max_depth))
            for a, b in zip(s.raycast_maps(level), want):
                np.testing.assert_array_equal(a.view(np.int32), b.cpu().numpy().view(np.int32))
    s.close()


@pytest.mark.parametrize("sizes", [(8, 40, 72), (136, 24, 200)])
def test_session_fusion_equals_the_stage(kf, cuda, sizes):
    """The first frame of sessions of both formats stepped together, alone and through kf_fuse on the
    same depth map, at a pose without rotation (so the three form the same world-to-camera floats):
    the same volumes bit for bit, in sizes that no unit of fusion divides."""
    from kfb200 import synth
    cfgs = [kf.config_small(width=164, height=124, fx=134.0, fy=134.0, cx=81.5, cy=61.5, volume_n=n,
                            mu=max(0.03, 3.0 / n), tsdf_format=i % 2) for i, n in enumerate(sizes)]
    imgs = [synth.sequence(c, 1, seed=3 + i)[0][0] for i, c in enumerate(cfgs)]
    b = kf.Batch(cfgs)
    b.step(imgs)
    for i, (c, img) in enumerate(zip(cfgs, imgs)):
        alone = kf.KinectFusion(c)
        alone.process_frame(img)
        n = c.volume_n
        f = cuda.empty((n, n, n), dtype=cuda.float16 if c.tsdf_format else cuda.float32, device="cuda")
        wt = cuda.empty((n, n, n), dtype=cuda.int16 if c.tsdf_format else cuda.float32, device="cuda")
        vol = kf.kernel.volume(f, wt, c.volume_width, c.mu, fmt=c.tsdf_format)
        kf.kernel.initializeGrid(vol)
        pose = np.array(list(c.initial_pose), np.float32).reshape(4, 4).T
        kf.kernel.fuse(dev(cuda, alone.depth(-1)), vol, pose, kf.level_intrinsics(c, 0))
        w = wt.cpu().numpy()
        w = w.view(np.uint16).astype(np.float32) / np.float32(kf.KF_WEIGHT_SCALE) if c.tsdf_format else w
        for s in (alone, b.session(i)):
            sf, sw = s.tsdf()
            np.testing.assert_array_equal(sf, f.float().cpu().numpy())
            np.testing.assert_array_equal(sw, w)
        assert n == 8 or (w > 0).any()
        alone.close()
    b.close()


@pytest.mark.parametrize("w,h", [(1, 1), (31, 7), (33, 9), (161, 119), (64, 8)])
def test_icp_rows_shapes(kf, orc, cuda, w, h):
    """Residual rows in sizes that the kernel's 32 x 8-pixel blocks do not divide: the float oracle's
    rows to a relative 1e-5 of the largest entry (both in float, a few fused roundings apart), the
    same zero rows but for pixels within rounding of a rejection (at most 1 %), nothing written past
    the end."""
    from kfb200 import synth
    cfg = kf.config_small(width=max(w, 2), height=max(h, 2), fx=262.5 * w / 320, fy=262.5 * w / 320, cx=w / 2 - 0.5,
                          cy=h / 2 - 0.5, levels=1)
    poses = synth.trajectory(synth.LOOP, 6, 4, cfg.volume_width)
    k = kf.level_intrinsics(cfg, 0)
    ik = np.linalg.inv(k.astype(np.float64)).astype(np.float32)
    vm = []
    for i in (4, 5):
        img = synth.render(synth.scene(cfg.volume_width), poses[i], w, h, float(cfg.fx), float(cfg.fy), float(cfg.cx),
                           float(cfg.cy), 4, i, noise=False)
        vm.append(orc.vertex_map(orc.convert(img, 1e-3), ik))
    tv, tn = vm[0].copy(), orc.normal_map(vm[0])
    R, t = poses[4][:3, :3], poses[4][:3, 3]
    tv[..., :3] = np.where(tv[..., 3:] == -1, tv[..., :3] @ R.T + t, 0)
    tn[..., :3] = np.where(tn[..., 3:] == -1, tn[..., :3] @ R.T, 0)
    rows = w * h
    A = cuda.full((rows * 6 + 8,), 7.0, device="cuda")
    b = cuda.full((rows + 8,), 7.0, device="cuda")
    kf.kernel.constructIcpResiduals(dev(cuda, vm[1]), dev(cuda, tv), dev(cuda, tn), R, t, R, t, k, 0.1, 0.35, A, b)
    oa, ob = orc.icp_residuals(vm[1], tv, tn, R, t, R, t, k, 0.1, 0.35)[:2]
    ga, gb = A[:rows * 6].cpu().numpy().reshape(-1, 6), b[:rows].cpu().numpy()
    assert float((A[rows * 6:] - 7).abs().max()) == 0 and float((b[rows:] - 7).abs().max()) == 0
    oa, ob = np.asarray(oa).reshape(-1, 6), np.asarray(ob).reshape(-1)
    flips = (np.abs(ga).sum(1) == 0) != (np.abs(oa).sum(1) == 0)
    assert flips.sum() <= 0.01 * rows
    scale = max(1.0, float(np.abs(oa).max(initial=0)))
    assert np.abs(ga - oa)[~flips].max(initial=0) <= 1e-5 * scale
    assert np.abs(gb - ob)[~flips].max(initial=0) <= 1e-5 * scale


@pytest.mark.parametrize("n", [1, 6, 255, 256, 257, 2047, 2049, 8193, 148 * 4 * 2048 + 5])
def test_least_squares_alignments_agree(kf, cuda, n):
    """A that starts on 8 bytes (read in pairs) and the same rows 4 bytes further: the same sums in
    the same order, so the same x bit for bit (or the same failure, for too few rows)."""
    import ctypes
    g = cuda.Generator(device="cuda").manual_seed(n)
    rows = cuda.randn((n, 6), device="cuda", generator=g)
    b = cuda.randn((n,), device="cuda", generator=g)
    room = cuda.zeros(6 * n + 1, device="cuda")
    room[1:] = rows.reshape(-1)
    got = []
    for at in (rows.data_ptr(), room.data_ptr() + 4):
        x = (ctypes.c_float * 6)()
        st = kf.lib.kf_solve_linear_least_squares(ctypes.c_void_p(at), ctypes.c_void_p(b.data_ptr()), n, x, None)
        got.append((st, np.array(x[:], np.float32).view(np.int32).tolist()))
    assert got[0] == got[1]
    if n >= 255:
        a64, b64 = rows.double().cpu().numpy(), b.double().cpu().numpy()
        want = np.linalg.solve(a64.T @ a64, a64.T @ b64)
        np.testing.assert_allclose(np.array(got[0][1], np.int32).view(np.float32), want, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("w,h,levels,side", [(32, 24, 1, False), (36, 28, 3, False), (164, 124, 2, True),
                                             (320, 240, 3, False), (640, 480, 3, True)])
def test_compute_pose_equals_the_session(kf, cuda, w, h, levels, side):
    """ICP.computePose on a session's own maps gives the session's pose and iterations bit for bit
    (its second frame: the start pose is the configuration's), on the default stream and on another,
    with calls that follow one another and calls of two threads at once."""
    import threading
    from kfb200 import synth
    cfg = kf.config_small(width=w, height=h, fx=262.5 * w / 320, fy=262.5 * w / 320, cx=w / 2 - 0.5, cy=h / 2 - 0.5,
                          levels=levels, iters=(6, 4, 3)[:levels], volume_n=64, mu=0.06)
    imgs, _ = synth.sequence(cfg, 2, seed=3, kind=synth.LOOP)
    s = kf.KinectFusion(cfg)
    s.process_frame(imgs[0])
    status, pose = s.process_frame(imgs[1])
    iters = s.frame_stats()["icp_iters"]
    maps = [[dev(cuda, m) for m in (s.vertex_map(lv), *s.raycast_maps(lv))] for lv in range(levels)]
    start = np.array(list(cfg.initial_pose), np.float32).reshape(4, 4).T
    out = []

    def call():
        stream = cuda.cuda.Stream() if side else None
        for _ in range(3):
            out.append(kf.ICP(cfg).computePose(*[[m[k] for m in maps] for k in range(3)], start, stream=stream))
    call()
    threads = [threading.Thread(target=call) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(out) == 9
    for st, p, it in out:
        assert st == status and it == iters
        if st == 0:
            np.testing.assert_array_equal(p.view(np.int32), np.asarray(pose, np.float32).view(np.int32))
    s.close()


@pytest.mark.parametrize("w,h,n,vis", [(32, 24, 64, 0), (164, 124, 200, 48), (640, 480, 256, 0)])
def test_frames_from_any_memory_agree(kf, cuda, w, h, n, vis):
    """Frames from pageable memory (the raycast is launched before their copy), pinned memory and the
    device give the same poses and volumes, blocking and two in flight, in a session, a profiled
    session and a batch; the kinds may follow one another in one session."""
    from kfb200 import synth
    cfg = kf.config_small(width=w, height=h, fx=262.5 * w / 320, fy=262.5 * w / 320, cx=w / 2 - 0.5, cy=h / 2 - 0.5,
                          volume_n=n, mu=max(0.03, 6.0 / n), vis_volume_n=vis, vis_volume_width=5.0, vis_mu=0.2)
    imgs, _ = synth.sequence(cfg, 5, seed=6, kind=synth.LOOP)
    pinned = [cuda.from_numpy(i.copy()).pin_memory() for i in imgs]
    kinds = {"pageable": list(imgs), "pinned": [p.numpy() for p in pinned], "device": [dev(cuda, i) for i in imgs]}
    kinds["mixed"] = [kinds[("pageable", "device", "pinned")[i % 3]][i] for i in range(5)]
    wants = {}
    for name, frames in kinds.items():
        runs = ["blocking", "profiled", "flying"] + (["batch"] if name in ("pageable", "pinned") else [])
        for how in runs:
            b = kf.Batch([cfg, cfg]) if how == "batch" else None
            s = b.session(1) if b else kf.KinectFusion(cfg)
            if how == "profiled":
                s.set_profiling(True)
            poses = []
            if b:
                poses = [b.step([f, f])[1][1] for f in frames]
            elif how == "flying":
                for i, f in enumerate(frames):
                    s.submit_frame(f)
                    if i:
                        poses.append(s.wait_frame()[1])
                poses.append(s.wait_frame()[1])
            else:
                poses = [s.process_frame(f)[1] for f in frames]
            got = [np.asarray(poses, np.float32).reshape(5, 16), *s.tsdf(), *(s.vis_tsdf() if vis else ())]
            for a, c in zip(wants.setdefault("batch" if b else "alone", got), got):
                np.testing.assert_array_equal(a, c, err_msg=name + " " + how)
            (b or s).close()


@pytest.mark.parametrize("w,h,radius", [(1, 1, 3), (31, 7, 0), (33, 9, 2), (64, 8, 3), (161, 119, 1), (97, 65, 7),
                                        (161, 119, 3)])
def test_bilateral_shapes(kf, orc, cuda, w, h, radius):
    """Blocks that overhang the image and halos that clamp, at every kind of radius; a filtered depth
    is a mean of values up to 6 m with weights of the fast exponential (2e-6 relative), so it agrees
    with the FP64 oracle to 2e-5 m."""
    rng = np.random.default_rng(w * 31 + h)
    d = (rng.uniform(0.5, 6.0) + 0.05 * rng.standard_normal((h, w))).astype(np.float32)
    out = cuda.zeros((h, w), device="cuda")
    kf.kernel.applyBilateralFilter(dev(cuda, d), out, 4.0, 0.25, radius)
    want = orc.bilateral(d, 4.0, 0.25, radius, prec=1)
    np.testing.assert_allclose(out.cpu().numpy(), want, atol=2e-5, rtol=0)


@pytest.mark.parametrize("n,w,h,fmt", [(136, 500, 330, 0), (200, 500, 331, 0), (200, 501, 330, 1)])
@pytest.mark.parametrize("depths", [(-1.5, 6.0), (-0.9, -0.05)])
def test_raycast_behind_the_camera(kf, cuda, n, w, h, fmt, depths):
    """A depth range that begins (or lies) behind the camera is a march like any other: from the middle
    of a volume with a sphere ahead and one behind, the maps of the march of every sample, bit for
    bit, and hits on both sides."""
    width, mu = 2.0, max(0.02, 3.0 / n)
    x = (cuda.arange(n, device="cuda", dtype=cuda.float32) + 0.5) * (width / n) - width / 2
    z, y, x = cuda.meshgrid(x, x, x, indexing="ij")
    d = [cuda.sqrt(x * x + y * y + (z - c) ** 2) - 0.25 for c in (0.6, -0.6)]
    f = cuda.clamp(cuda.minimum(*d) / mu, -1.0, 1.0)
    f = (f.half() if fmt else f).contiguous()
    vol = kf.kernel.volume(f, cuda.zeros_like(f), width, mu, fmt=fmt)
    ik = np.linalg.inv(np.array([[300, 0, w / 2], [0, 300, h / 2], [0, 0, 1]], np.float64)).astype(np.float32)
    pose = np.eye(4, dtype=np.float32)
    pose[:3, 3] = (0.02, -0.01, 0.03)
    out = [[cuda.full((h, w, 4), 7.0, device="cuda") for _ in range(2)] for _ in range(2)]
    kf.kernel.raycast(vol, pose, ik, *out[0], min_depth=depths[0], max_depth=depths[1])
    plain_raycast(kf, cuda, vol, pose, ik, *out[1], (1.99, 0.1), depths)
    for a, b in zip(*out):
        assert cuda.equal(a.view(cuda.int32), b.view(cuda.int32))
    hit = out[1][0][out[1][0][..., 3] == -1]
    assert (hit[:, 2] < 0).sum() > 1000


@pytest.mark.parametrize("radius", [2, 3])
@pytest.mark.parametrize("sigma_s,sigma_r", [(4.5, 0.03), (4.0, 0.25), (3.3, 0.11)])
def test_bilateral_radii_agree(kf, cuda, radius, sigma_s, sigma_r):
    """A filtered depth does not depend on how the filter is built for its radius: patches as wide as the
    window, each ringed by depths so far off that their weights are zero, give their middles the same
    bits at every radius -- the ring adds zeros, in the same order."""
    cells, side = 40, 9
    rng = np.random.default_rng(radius)
    d = np.full((cells * side, cells * side), 900.0, np.float32)
    inner = slice(4 - radius, 5 + radius)
    for i in range(cells):
        for j in range(cells):
            patch = rng.uniform(0.5, 6.0) + sigma_r * rng.standard_normal((2 * radius + 1, 2 * radius + 1))
            d[i * side:(i + 1) * side, j * side:(j + 1) * side][inner, inner] = patch
    mid = []
    for r in (radius, 4):
        out = cuda.zeros(d.shape, device="cuda")
        kf.kernel.applyBilateralFilter(dev(cuda, d), out, sigma_s, sigma_r, r)
        mid.append(out.cpu().numpy()[4::side, 4::side])
    np.testing.assert_array_equal(mid[0].view(np.int32), mid[1].view(np.int32))


def test_fuse_refuses_a_captured_stream(kf, cuda):
    """kf_fuse waits for its stream, so a stream that is being captured is refused with an error, before
    anything is recorded: the capture goes on and the volume is untouched."""
    import ctypes
    n, w, h = 64, 64, 48
    f, wt = cuda.full((n, n, n), 2.0, device="cuda"), cuda.zeros((n, n, n), device="cuda")
    vol = kf.kernel.volume(f, wt, 2.0, 0.1)
    depth, other = cuda.full((h, w), 1.0, device="cuda"), cuda.zeros(1, device="cuda")
    k = np.array([[60, 0, w / 2], [0, 60, h / 2], [0, 0, 1]], np.float32)
    pose = np.eye(4, dtype=np.float32)
    pose[2, 3] = -1.0
    s = cuda.cuda.Stream()
    ms = ctypes.c_float()
    cuda.cuda.synchronize()
    g, got = cuda.cuda.CUDAGraph(), []
    with cuda.cuda.graph(g, stream=s):
        for elapsed in (None, ctypes.byref(ms)):
            got.append(kf.lib.kf_fuse(ctypes.c_void_p(depth.data_ptr()), w, h, kf.to_colmajor(k), ctypes.byref(vol),
                                      kf.to_colmajor(pose), 0.4, 6.0, ctypes.c_void_p(s.cuda_stream), elapsed))
        other.add_(1)
    assert got == [kf.KF_ERR_CUDA] * 2
    g.replay()
    cuda.cuda.synchronize()
    assert float(other) == 1 and float(wt.max()) == 0
    kf.kernel.fuse(depth, vol, pose, k)
    assert float(wt.max()) > 0


@pytest.mark.parametrize("w,h", [(1, 524281), (3, 1048560)])
def test_icp_rows_of_tall_maps(kf, orc, cuda, w, h):
    """More rows than a grid's second dimension holds blocks of eight: every row is written, the residual
    of the one pixel near the bottom that has a normal and zeros for the others."""
    maps = [cuda.zeros((h, w, 4), device="cuda") for _ in range(3)]
    for m in maps:
        m[..., 3] = -2
    corner = np.array([[[0, 0, 1.01, -1], [0.01, 0, 1.01, -1]], [[0, 0.01, 1.01, -1], [0, 0, 0, -2]]], np.float32)
    normal = orc.normal_map(corner)[0, 0]
    if w > 1:
        maps[0][h - 2:, :2] = dev(cuda, corner)
        maps[1][h - 2, 0] = cuda.tensor([0.0, 0.0, 1.0, -1.0])
        maps[2][h - 2, 0] = dev(cuda, normal)
    k = np.array([[1, 0, 0.5], [0, 1, h - 1.5], [0, 0, 1]], np.float32)
    eye, zero = np.eye(3, dtype=np.float32), np.zeros(3, np.float32)
    A, b = cuda.full((w * h, 6), 7.0, device="cuda"), cuda.full((w * h,), 7.0, device="cuda")
    kf.kernel.constructIcpResiduals(*maps, eye, zero, eye, zero, k, 0.1, 0.35, A, b)
    if w > 1:
        at = (h - 2) * w
        np.testing.assert_allclose(A[at].cpu().numpy(), [0, 0, 0, 0, 0, normal[2]], atol=1e-6)
        np.testing.assert_allclose(float(b[at]), -0.01 * normal[2], atol=1e-6)
        A[at] = 0
        b[at] = 0
    assert float(A.abs().max()) == 0 and float(b.abs().max()) == 0


@pytest.mark.parametrize("mode", ["global", "thread_local"])
def test_raycast_beside_a_capture(kf, orc, cuda, mode):
    """A raycast on one stream while another is captured: the capture goes on and replays, and the maps are
    those of a call without one.  In a process of its own, whose first scratch this call takes."""
    import os
    import subprocess
    import sys
    prog = ("import sys, ctypes; sys.path[:0] = %r\n"
            "import numpy as np, torch, kfb200 as kf\n"
            "n, w, h = 64, 480, 360\n"
            "r = (torch.arange(n, device='cuda') + 0.5) / n * 2 - 1\n"
            "z, y, x = torch.meshgrid(r, r, r, indexing='ij')\n"
            "f = torch.clamp((torch.sqrt(x * x + y * y + z * z) - 0.5) / 0.1, -1, 1).contiguous()\n"
            "vol = kf.kernel.volume(f, torch.zeros_like(f), 2.0, 0.1)\n"
            "ik = np.linalg.inv(np.array([[400, 0, w / 2], [0, 400, h / 2], [0, 0, 1]], float)).astype(np.float32)\n"
            "pose = np.eye(4, dtype=np.float32)\npose[2, 3] = -2\n"
            "out = [[torch.full((h, w, 4), 7.0, device='cuda') for _ in range(2)] for _ in range(2)]\n"
            "side, other, hit = torch.cuda.Stream(), torch.cuda.Stream(), torch.zeros(1, device='cuda')\n"
            "def cast(maps, stream):\n"
            "    p = [ctypes.c_void_p(m.data_ptr()) for m in maps]\n"
            "    return kf.lib.kf_raycast(ctypes.byref(vol), kf.to_colmajor(pose), kf.to_colmajor(ik), p[0], w, h, p[1],\n"
            "                             w, h, 0.4, 6.0, 1.99, 0.1, ctypes.c_void_p(stream), None)\n"
            "torch.cuda.synchronize()\ng = torch.cuda.CUDAGraph()\n"
            "with torch.cuda.graph(g, stream=side, capture_error_mode=%r):\n"
            "    hit.add_(1)\n    assert cast(out[0], other.cuda_stream) == 0\n"
            "g.replay()\nassert cast(out[1], 0) == 0\ntorch.cuda.synchronize()\n"
            "assert float(hit) == 1 and all(torch.equal(a, b) for a, b in zip(*out))\n"
            "assert float((out[0][0][..., 3] == -1).float().mean()) > 0.05\n"
            % ([os.path.dirname(os.path.dirname(os.path.abspath(kf.__file__)))], mode))
    r = subprocess.run([sys.executable, "-c", prog], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
