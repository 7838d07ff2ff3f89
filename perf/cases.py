"""The work a user of this library has it do, as cases that can be timed and compared.

Seven kinds, each through the public calls (the C ABI and its ctypes mirror):

  front   the kernel-level calls of one RGB-D frame on device buffers: depth filtering, depth
          pyramid, reference maps, colour pyramid with gradients
  track   one step-wise frame against given reference maps: upload and ICP
  locate  rendering the model from a pose, then upload and ICP against it (the step-wise frame
          without the integration; relocalisation does the same)
  fuse    depth frames with known poses into an empty scene (step-wise upload, pose,
          integration); a dense scene is meshed, a voxel-hash scene is rendered and tracked
          against once, so that what was fused comes back
  mesh    marching cubes of a scanned dense volume into device buffers
  stream  a live stream of one session: whole frames from host memory, poses back
  batch   many sessions, one frame each a tick: whole ticks on device frames, poses back

Frames come from the package's seeded synthetic scenes (Kinect-like noise, 2 degrees of orbit a
frame); sizes are those of the configurations, tests and benchmark of this repository (640x480
frames; dense volumes of 128 to 512 voxels a side over 3 or 4 m; voxel-hash scenes of 5 mm voxels
with 2^20 buckets; 10/5/4 ICP iterations) or generic ones (QQVGA to HD images, odd volumes).
"""
import ctypes as C

import numpy as np
import torch

from natureuserinterfacestudio_b200 import _lib as L
from natureuserinterfacestudio_b200 import synth as S

FORMATS = {"i16": L.TSDF_I16, "f32": L.TSDF_F32, "f16u8": L.TSDF_F16_U8, "f16f16": L.TSDF_F16_F16}
VOXEL_BYTES = {"i16": 4, "f32": 8, "f16u8": 3, "f16f16": 4}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a gesture camera's small frames: kernel-level calls whose time is launches and waits
        {"name": "front_160x120", "kind": "front", "w": 160, "h": 120, "levels": 3, "radius": 3},
        # the default frame through the kernel-level calls
        {"name": "front_640x480", "kind": "front", "w": 640, "h": 480, "levels": 3, "radius": 3},
        # the tracker alone on one stream (the latency an interactive program sees)
        {"name": "track_640x480", "kind": "track", "w": 640, "h": 480, "volume": "dense", "fmt": "f32",
         "rx": 256, "ry": 256, "rz": 256, "dim": 3.0, "color": False},
        # raycast and ICP on the large serving volume
        {"name": "locate_dense512_f16u8", "kind": "locate", "w": 640, "h": 480, "volume": "dense", "fmt": "f16u8",
         "rx": 512, "ry": 512, "rz": 512, "dim": 4.0, "color": False},
        # raycast and colour ICP on a voxel-hash scene
        {"name": "locate_hash_color", "kind": "locate", "w": 640, "h": 480, "volume": "hash", "fmt": "f16u8",
         "voxel": 0.005, "buckets": 1 << 20, "excess": 1 << 16, "pool": 1 << 16, "color": True},
        # fusion with known poses in the reference's format, then its mesh
        {"name": "fuse_dense256_i16", "kind": "fuse", "w": 640, "h": 480, "volume": "dense", "fmt": "i16",
         "rx": 256, "ry": 256, "rz": 256, "dim": 3.0, "color": False, "frames": 4},
        # the same on small frames and a ragged FP32 volume
        {"name": "fuse_dense_ragged_f32", "kind": "fuse", "w": 320, "h": 240, "volume": "dense", "fmt": "f32",
         "rx": 250, "ry": 231, "rz": 173, "dim": 3.0, "color": False, "frames": 3},
        # fusion with known poses into a voxel-hash scene (allocation, visible list, integration)
        {"name": "fuse_hash_color", "kind": "fuse", "w": 640, "h": 480, "volume": "hash", "fmt": "i16",
         "voxel": 0.005, "buckets": 1 << 20, "excess": 1 << 16, "pool": 1 << 16, "color": True, "frames": 4},
        # meshing a scan
        {"name": "mesh_dense256_f32", "kind": "mesh", "fmt": "f32", "rx": 256, "ry": 256, "rz": 256, "color": False},
        {"name": "mesh_dense512_f16u8", "kind": "mesh", "fmt": "f16u8", "rx": 512, "ry": 512, "rz": 512,
         "color": True},
        # one live stream, whole frames: depth and colour in, pose out
        {"name": "stream_dense384_f16u8", "kind": "stream", "w": 640, "h": 480, "volume": "dense", "fmt": "f16u8",
         "rx": 384, "ry": 384, "rz": 384, "dim": 4.0, "color": True, "frames": 5},
        # the serving mix: 64 streams, 3 of 5 dense, 2 of 5 voxel-hash RGB-D
        {"name": "batch_64_640x480", "kind": "batch", "n": 64, "w": 640, "h": 480, "fmt": "f16u8",
         "buckets": 1 << 20, "pool": 1 << 16, "frames": 4},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _image(rng, lo, hi, levels=3):
    """A width x height with `levels` pyramid levels, 4:3 to 16:9, odd multiples among them."""
    m = 1 << (levels - 1)
    w = max(m * 8, _log(rng, lo, hi) // m * m)
    h = max(m * 8, int(w / rng.uniform(1.2, 1.8)) // m * m)
    return w, h


def _dense(rng, lo, hi):
    r = _log(rng, lo, hi)
    sides = [max(24, int(r * rng.uniform(0.7, 1.0))) for _ in range(3)]
    if rng.random() < 0.4:
        sides = [r // 16 * 16 + 16] * 3
    return {"rx": sides[0], "ry": sides[1], "rz": sides[2], "dim": round(rng.uniform(2.5, 4.0), 2)}


def _hash(rng):
    return {"voxel": round(rng.uniform(0.005, 0.01), 4), "buckets": 1 << rng.randint(17, 20),
            "excess": rng.randint(20000, 70000), "pool": 1 << 16}


def draw(rng):
    kind = rng.choice(["front", "front", "track", "locate", "locate", "fuse", "fuse", "mesh", "mesh", "stream", "batch"])
    if kind == "front":
        levels = rng.randint(1, 3)
        w, h = _image(rng, 100, 1920, levels)
        return {"kind": kind, "w": w, "h": h, "levels": levels, "radius": rng.choice([2, 3, 3, 3, 4])}
    if kind == "mesh":
        d = _dense(rng, 48, 448)
        d.pop("dim")
        return {"kind": kind, "fmt": rng.choice(sorted(FORMATS)), "color": rng.random() < 0.4, **d}
    w, h = _image(rng, 160, 640)
    if kind == "batch":
        return {"kind": kind, "n": _log(rng, 2, 40), "w": w, "h": h, "fmt": rng.choice(["f16u8", "f16f16", "i16"]),
                "buckets": 1 << rng.randint(17, 20), "pool": 1 << 16, "frames": rng.randint(3, 4)}
    volume = "hash" if kind != "track" and rng.random() < 0.4 else "dense"
    fmt = rng.choice(sorted(FORMATS))
    if volume == "hash":
        fmt = rng.choice(["i16", "f16u8"])
    elif kind == "fuse":  # the exact formats: a rounding elsewhere cannot move a mesh's vertices
        fmt = rng.choice(["i16", "f32"])
    case = {"kind": kind, "w": w, "h": h, "volume": volume, "fmt": fmt, "color": rng.random() < 0.5,
            **(_hash(rng) if volume == "hash" else _dense(rng, 96, 448))}
    if kind in ("fuse", "stream"):
        case["frames"] = rng.randint(3, 6)
    return case


# ------------------------------------------------------------------ inputs
def _camera(w, h):
    f = float(np.float32(525.0 * w / 640.0))
    return f, (w - 1) / 2.0, (h - 1) / 2.0


def _frames(seed, n, w, h, color):
    """n frames of an orbit: (depth uint16, bgra uint8 or None, R, t), poses relative to the first."""
    f, cx, cy = _camera(w, h)
    scene = S.SynthScene(S.SYNTH_TABLETOP, seed=1000 + seed % 1000003, extent=3.0)
    out, first = [], None
    for i in range(n):
        R, t = scene.pose(i, radius=1.5, deg_per_frame=2.0)
        d, c = scene.render(R, t, w, h, fx=f, fy=f, cx=cx, cy=cy, noise_seed=seed % 65521 + 7, frame=i, color=color)
        R, t = np.asarray(R, np.float64), np.asarray(t, np.float64)
        first = first or (R, t)
        out.append((d, c, first[0].T @ R, first[0].T @ (t - first[1])))
    return out


def _config(case):
    f, cx, cy = _camera(case["w"], case["h"])
    common = dict(width=case["w"], height=case["h"], fx=f, fy=f, cx=cx, cy=cy, tsdf_format=FORMATS[case["fmt"]],
                  iterations=[10, 5, 4, 0], integration_threshold=0.0, color_volume=int(case["color"]),
                  photometric_weight=0.1 if case["color"] else 0.0)
    if case["volume"] == "hash":
        return L.default_cfg(volume_kind=L.VOLUME_HASH, voxel_size=case["voxel"], trunc_scale=4 * case["voxel"],
                             hash_buckets=case["buckets"], hash_excess=case["excess"], hash_pool_blocks=case["pool"],
                             depth_min=0.4, **common)
    return L.default_cfg(res=(case["rx"], case["ry"], case["rz"]), dim=(case["dim"],) * 3, trunc_dist=0.03, **common)


def _scan(case, seed, device):
    """A scanned volume in the reference layout (short2, z fastest): a room with ellipsoids, free
    space weighted with tsdf 1, noise in the truncation band, no weight inside the surfaces."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    r = (case["rx"], case["ry"], case["rz"])
    x, y, z = (((torch.arange(n, device=device, dtype=torch.float32) + 0.5) / n - 0.5) for n in r)
    p = torch.rand((6, 6), generator=g, device=device)
    sdf = torch.full((r[1], r[0], r[2]), 1.0, device=device)
    X, Y, Z = x[None, :, None], y[:, None, None], z[None, None, :]
    for k in range(6):
        c, a = (p[k, :3] - 0.5) * 0.7, 0.06 + 0.12 * p[k, 3:]
        q = (((X - c[0]) / a[0]) ** 2 + ((Y - c[1]) / a[1]) ** 2 + ((Z - c[2]) / a[2]) ** 2).sqrt_()
        torch.minimum(sdf, q.sub_(1.0).mul_(float(a.min())), out=sdf)
    torch.minimum(sdf, 0.42 - 0.02 * torch.sin(14 * X) * torch.cos(11 * Z) - Y, out=sdf)
    trunc = 2.1 / max(r) * 1.3
    sdf += torch.randn(sdf.shape, generator=g, device=device) * (0.08 * trunc)
    weight = torch.randint(1, 65, sdf.shape, generator=g, device=device, dtype=torch.int16)
    weight[sdf < -trunc] = 0
    tsdf = (sdf.div_(trunc).clamp_(-1, 1) * 32766).to(torch.int16)
    return torch.stack((tsdf, weight), dim=-1).cpu().numpy()


def _pose12(R, t):
    return np.concatenate([np.asarray(R, np.float32).reshape(9), np.asarray(t, np.float32).reshape(3)])


def _session_pose(s):
    R, t = s.get_pose()
    return _pose12(R, t)


def _address(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _mesh(s, pos, col):
    """Vertex count, with the vertices (as many as fit) written to the given device buffers."""
    n = C.c_uint64()
    r = L.lib().nui_mesh_device_noalloc(s.h, _address(pos), _address(col), pos.shape[0], C.byref(n))
    if r not in (L.NUI_OK, L.NUI_ERR_MESH_OVERFLOW):
        L.check(r)
    return n.value


def _mesh_buffers(case):
    # room for some ten layers of surface across the volume (an indoor scan fills a part of it)
    n = int(60 * (case["rx"] * case["ry"] * case["rz"]) ** (2 / 3))
    color = case["color"]
    pos = torch.zeros((n, 3), dtype=torch.float32, device="cuda")
    return pos, torch.zeros((n, 4), dtype=torch.float32, device="cuda") if color else None


def _pingpong(k, n):
    k %= 2 * n - 2
    return k if k < n else 2 * n - 2 - k


# ------------------------------------------------------------------ preparation
def prepare(case, seed):
    return {"case": case, **globals()["_prepare_" + case["kind"]](case, seed)}


def _prepare_front(case, seed):
    w, h, levels = case["w"], case["h"], case["levels"]
    (d, c, _, _), (_, _, R, t) = _frames(seed, 2, w, h, True)

    def maps(dtype, channels):
        return [torch.zeros(((h >> l), (w >> l)) + channels, dtype=dtype, device="cuda") for l in range(levels)]

    bgra, gx, gy = maps(torch.uint8, (4,)), maps(torch.uint8, (4,)), maps(torch.uint8, (4,))
    bgra[0].copy_(torch.from_numpy(c))
    return {"ctx": L.Context(0), "raw": torch.from_numpy(d.view(np.int16)).cuda(), "pose": _pose12(R, t),
            "depth": maps(torch.float32, ()), "vertex": maps(torch.float32, (4,)),
            "scaled": torch.zeros((h, w), dtype=torch.float32, device="cuda"),
            "vref": torch.zeros((h, w, 4), dtype=torch.float32, device="cuda"),
            "nref": torch.zeros((h, w, 4), dtype=torch.float32, device="cuda"),
            "bgra": bgra, "gx": gx, "gy": gy,
            "levels": [(C.c_void_p * levels)(*[x.data_ptr() for x in m]) for m in (bgra, gx, gy)]}


def _prepare_track(case, seed):
    frames = _frames(seed, 3, case["w"], case["h"], case["color"])
    s = L.Session(L.Context(0), _config(case))
    for d, c, _, _ in frames[:2]:
        s.process(d, c)
    return {"s": s, "frame": frames[2][:2], "pose": s.get_pose()}


_prepare_locate = _prepare_track


def _prepare_fuse(case, seed):
    frames = _frames(seed, case["frames"] + 1, case["w"], case["h"], case["color"])
    state = {"s": L.Session(L.Context(0), _config(case)), "frames": frames}
    if case["volume"] == "dense":
        state["pos"], state["col"] = _mesh_buffers(case)
    return state


def _prepare_mesh(case, seed):
    cfg = L.default_cfg(width=160, height=120, fx=131.25, fy=131.25, cx=79.5, cy=59.5,
                        res=(case["rx"], case["ry"], case["rz"]), tsdf_format=FORMATS[case["fmt"]],
                        color_volume=int(case["color"]))
    s = L.Session(L.Context(0), cfg)
    s.upload_volume(_scan(case, seed, "cuda"))
    pos, col = _mesh_buffers(case)
    return {"s": s, "pos": pos, "col": col}


def _prepare_stream(case, seed):
    frames = _frames(seed, case["frames"], case["w"], case["h"], case["color"])
    return {"s": L.Session(L.Context(0), _config(case)), "frames": [f[:2] for f in frames]}


def _prepare_batch(case, seed):
    n, kinds = case["n"], min(3, case["n"])
    dense = ((256, 3.0), (384, 4.0), (512, 4.0))
    small = case["w"] < 480  # smaller frames go with smaller volumes
    seqs = [_frames(seed + 17 * k, case["frames"], case["w"], case["h"], True) for k in range(kinds)]
    depth = [[torch.from_numpy(d.view(np.int16)).cuda() for d, _, _, _ in q] for q in seqs]
    color = [[torch.from_numpy(c).cuda() for _, c, _, _ in q] for q in seqs]
    ctx = L.Context(0)
    sessions, is_hash = [], []
    for i in range(n):
        shape = {"w": case["w"], "h": case["h"], "fmt": case["fmt"], "color": False}
        if i % 5 < 3:
            r, dim = dense[i % 3]
            r = r // 2 if small else r
            shape.update(volume="dense", rx=r, ry=r, rz=r, dim=dim)
        else:
            shape.update(volume="hash", voxel=0.01 if small else 0.005, buckets=case["buckets"], excess=1 << 16,
                         pool=case["pool"], color=True)
        sessions.append(L.Session(ctx, _config(shape)))
        is_hash.append(i % 5 >= 3)
    return {"ctx": ctx, "sessions": sessions, "is_hash": is_hash, "depth": depth, "color": color}


# ------------------------------------------------------------------ one pass
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_front(s):
    c, k, h = s["case"], L.lib(), s["ctx"].h
    f, cx, cy = _camera(c["w"], c["h"])
    L.check(k.nui_k_preprocess(h, _address(s["raw"]), c["w"], c["h"], f, f, cx, cy, 0.5, 4.5, c["radius"], 0.08, 50.0,
                               0.3, _address(s["depth"][0]), _address(s["vertex"][0]), _address(s["scaled"])))
    for l in range(1, c["levels"]):
        L.check(k.nui_k_pyramid_level(h, _address(s["depth"][l - 1]), c["w"] >> l, c["h"] >> l, f, f, cx, cy, 1 << l,
                                      0.3, _address(s["depth"][l]), _address(s["vertex"][l])))
    L.check(k.nui_k_feedback_maps(h, _address(s["vertex"][0]), c["w"], c["h"], 0.3, L.ptr(s["pose"]),
                                  _address(s["vref"]), _address(s["nref"])))
    L.check(k.nui_k_color_pyramid(h, _address(s["bgra"][0]), c["w"], c["h"], c["levels"], *s["levels"]))
    return {name: s[name] for name in ("depth", "vertex", "scaled", "vref", "nref", "bgra", "gx", "gy")}


def _run_track(s):
    s["s"].set_pose(*s["pose"])
    s["s"].upload(*s["frame"])
    ok, error, _ = s["s"].track()
    return {"ok": ok, "error": error, "pose": _session_pose(s["s"])}


def _run_locate(s):
    s["s"].set_pose(*s["pose"])
    s["s"].raycast()
    s["s"].upload(*s["frame"])
    ok, error, _ = s["s"].track()
    return {"ok": ok, "error": error, "pose": _session_pose(s["s"])}


def _fuse(s):
    s["s"].reset()
    for d, c, R, t in s["frames"][:-1]:
        s["s"].upload(d, c)
        s["s"].set_pose(R, t)
        s["s"].integrate()


def _run_fuse(s):
    _fuse(s)
    if s["case"]["volume"] == "dense":
        n = _mesh(s["s"], s["pos"], s["col"])
        return {"vertices": n, "updated": s["s"].touched(), "pos": s["pos"], "col": s["col"]}
    updated, blocks = s["s"].touched(), s["s"].hash_stats()
    s["s"].raycast()
    s["s"].upload(*s["frames"][-1][:2])
    ok, error, _ = s["s"].track()
    out = {"blocks": list(blocks), "ok": ok, "error": error, "pose": _session_pose(s["s"])}
    if s["case"]["fmt"] == "i16":  # (the half format may take another side of a pixel's edge)
        out["updated"] = updated
    return out


def _run_mesh(s):
    return {"vertices": _mesh(s["s"], s["pos"], s["col"]), "pos": s["pos"], "col": s["col"]}


def _run_stream(s):
    n = len(s["frames"])
    ok, poses = [], []
    for k in range(2 * n - 2):  # forth and back: the next pass goes on from here
        good, pose = s["s"].process(*s["frames"][_pingpong(k, n)])
        ok.append(good)
        poses.append(pose)
    return {"ok": np.array(ok), "poses": np.stack(poses)}


def _run_batch(s):
    n, nf, kinds = len(s["sessions"]), s["case"]["frames"], len(s["depth"])
    status, poses = [], []
    for k in range(2 * nf - 2):
        at = [_pingpong(7 * i + k, nf) for i in range(n)]
        st, p = s["ctx"].batch_tick(
            s["sessions"], [s["depth"][i % kinds][at[i]].data_ptr() for i in range(n)],
            [s["color"][i % kinds][at[i]].data_ptr() if s["is_hash"][i] else None for i in range(n)], device=True)
        status.append(st)
        poses.append(p)
    return {"status": np.stack(status), "poses": np.stack(poses)}


# ------------------------------------------------------------------ work of one pass
def _icp_flops(pixels):
    # one iteration of each of the three levels: ~60 operations to match a pixel, ~58 to add its row
    return pixels * (1 + 1 / 4 + 1 / 16) * 118


def _scene_bytes(case):
    """Voxels one frame cannot help updating, read and written: those in front of the surfaces, about
    a tenth of a volume that the frame sees whole; a hash scene's visible blocks, about one block for
    every 32 pixels of 5 mm voxels at 640x480."""
    if case["volume"] == "hash":
        return (0.005 / case["voxel"]) ** 2 * 9600 * 512 * 2 * (3 + 4 * case["color"])
    return 0.1 * case["rx"] * case["ry"] * case["rz"] * 2 * (VOXEL_BYTES[case["fmt"]] + 4 * case["color"])


def work(case):
    kind = case["kind"]
    if kind == "mesh":
        n = case["rx"] * case["ry"] * case["rz"]
        faces = 6 * (n ** (2 / 3))
        return {"bytes": n * VOXEL_BYTES[case["fmt"]] + faces * 2 * 3 * (12 + 16 * case["color"]), "flops": 10 * faces}
    px = case["w"] * case["h"]
    if kind == "front":
        taps = (2 * case["radius"] + 1) ** 2
        pyramid = sum(px / 4 ** l for l in range(case["levels"]))
        return {"bytes": px * (2 + 4 + 4 + 32) + pyramid * (4 + 16 + 4 + 8), "flops": px * (taps * 14 + 100)}
    if kind == "track":
        return {"bytes": px * (2 + 32), "flops": px * 49 * 14 + _icp_flops(px)}
    if kind == "locate":
        return {"bytes": px * (2 + 4 * case["color"] + 32), "flops": px * (49 * 14 + 400) + _icp_flops(px)}
    if kind == "fuse":
        frame = px * (2 + 4 * case["color"]) + _scene_bytes(case)
        return {"bytes": case["frames"] * frame, "flops": case["frames"] * px * 49 * 14}
    passes = 2 * case["frames"] - 2
    if kind == "stream":
        frame = px * (2 + 4 * case["color"] + 32) + _scene_bytes(case)
        return {"bytes": passes * frame, "flops": passes * (px * (49 * 14 + 400) + _icp_flops(px))}
    scale = 0.125 if case["w"] < 480 else 1.0
    dense = scale * 0.1 * (256 ** 3 + 384 ** 3 + 512 ** 3) / 3 * 2 * VOXEL_BYTES[case["fmt"]]
    blocks = (0.25 if case["w"] < 480 else 1.0) * 9600 * 512 * 2 * 7
    n, nd = case["n"], sum(i % 5 < 3 for i in range(case["n"]))
    total = n * px * 34 + (n - nd) * (px * 4 + blocks) + nd * dense
    return {"bytes": passes * total, "flops": passes * n * (px * (49 * 14 + 400) + _icp_flops(px))}


# ------------------------------------------------------------------ 64-bit results
def _shifted(a, dy, dx, fill):
    out = torch.full_like(a, fill)
    h, w = a.shape[:2]
    out[max(0, -dy):h - max(0, dy), max(0, -dx):w - max(0, dx)] = a[max(0, dy):h + min(0, dy), max(0, dx):w + min(0, dx)]
    return out


def _vertices(depth, w, h, level):
    f, cx, cy = _camera(w, h)
    div = 1 << level
    x, y = (torch.arange(n, dtype=torch.float64) for n in (depth.shape[1], depth.shape[0]))
    v = torch.stack((depth * ((x - cx / div) * div / f)[None, :], depth * ((y - cy / div) * div / f)[:, None], depth,
                     torch.zeros_like(depth)), dim=-1)
    v[..., 3] = 0.0
    return v


def exact(case, seed):
    """The filtered depths, vertices and reference maps of a front case.  The other kinds return
    poses that an iteration reaches, or vertices in the order of a scan: no closed form."""
    if case["kind"] != "front":
        return None
    w, h, nan = case["w"], case["h"], float("nan")
    (d, _, _, _), (_, _, R, t) = _frames(seed, 2, w, h, True)
    raw = torch.from_numpy(d.astype(np.float32)) * np.float32(0.001)  # the path's input is float metres
    raw[~((raw > 0.5) & (raw < 4.5))] = nan
    c = raw.double()
    top, bottom = torch.zeros_like(c), torch.zeros_like(c)
    r = case["radius"]
    for dy in range(-r, r + 1):
        for dx in range(-r, r + 1):
            q = _shifted(raw, dy, dx, nan)
            near = (q > 0) & ((raw - q).abs() < np.float32(0.3))
            q = q.double()
            wt = torch.where(near, torch.exp(-0.08 * (dx * dx + dy * dy) - 50.0 * (c - q) ** 2), torch.zeros_like(c))
            top += torch.where(near, q * wt, torch.zeros_like(c))
            bottom += wt
    depth = [torch.where(torch.isnan(c), torch.full_like(c, nan), top / bottom)]
    for l in range(1, case["levels"]):
        src = depth[-1]
        mid = src[::2, ::2]
        total, n = torch.zeros_like(mid), torch.zeros_like(mid)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                q = _shifted(src, dy, dx, nan)[::2, ::2]
                ok = ~torch.isnan(q) & (torch.isnan(mid) | ((mid - q).abs() < 0.3))
                total += torch.where(ok, q, torch.zeros_like(q))
                n += ok
        depth.append(torch.where(n > 0, total / n, torch.full_like(mid, nan)))
    vertex = [_vertices(x, w, h, l) for l, x in enumerate(depth)]
    f, cx, cy = _camera(w, h)
    xl, yl = ((torch.arange(n, dtype=torch.float64) - m) / f for n, m in ((w, cx), (h, cy)))
    scaled = c * (xl[None, :] ** 2 + yl[:, None] ** 2 + 1).sqrt()
    v = vertex[0][..., :3]

    def neighbour(dy, dx):
        q = _shifted(v, dy, dx, nan)
        ok = ~torch.isnan(q[..., 2]) & ((v[..., 2] - q[..., 2]).abs() <= 0.3)
        return torch.where(ok[..., None], q, v)

    n = torch.linalg.cross(neighbour(0, 1) - neighbour(0, -1), neighbour(1, 0) - neighbour(-1, 0))
    length = n.norm(dim=-1, keepdim=True)
    n = torch.where(length > 0, n / length, n)
    R = torch.from_numpy(np.float32(R).astype(np.float64))
    t = torch.from_numpy(np.float32(t).astype(np.float64))
    pad = torch.zeros((h, w, 1), dtype=torch.float64)
    return {"depth": depth, "vertex": vertex, "scaled": scaled, "vref": torch.cat((v @ R.T + t, pad), -1),
            "nref": torch.cat((n @ R.T, pad), -1), "bgra": None, "gx": None, "gy": None}
