"""Skipping by brick distances against the plain march: volumes of odd sizes (rows of bricks
that are no multiple of 16 or 32, less than the blocks' tiles, up to the largest) with surfaces
at every distance from the bricks' and words' edges, raycast from several poses, exact and
tolerance formats, against the oracle's maps; and a snapshot, whose distances are rebuilt."""
import ctypes as C

import numpy as np
import pytest

from natureuserinterfacestudio_b200 import _lib as L
from oracle import oracle as O

from _util import cfg_for, same_bits

pytestmark = pytest.mark.gpu


def _volume(res, seed):
    """Free space with a far wall, floating blobs and pockets without weight; reference layout."""
    rng = np.random.default_rng(seed)
    rx, ry, rz = res
    x, y, z = np.meshgrid(np.arange(rx), np.arange(ry), np.arange(rz), indexing="ij")
    f = (rz - 4.0 - z) + 2.0 * np.sin(x / 9.0) + 1.5 * np.cos(y / 7.0)
    for _ in range(7):
        c, r = rng.random(3) * res, 1.5 + rng.random() * min(res) / 6
        f = np.minimum(f, np.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) - r)
    v = np.zeros(res + (2,), np.int16)
    v[..., 0] = np.clip(f / 3, -1, 1) * 32766
    v[..., 1] = np.where(f > -2.5, 5, 0)
    c = rng.integers(0, np.array(res) - 4, (6, 3))
    for i in c:
        v[i[0]:i[0] + 4, i[1]:i[1] + 4, i[2]:i[2] + 4, 1] = 0
    return np.ascontiguousarray(v.transpose(1, 0, 2, 3).reshape(-1, 2))


POSES = [((0, 0, 0), (0.0, 0.0, 0.0)), ((0.0, 0.3, 0.0), (-0.4, 0.1, 0.2)), ((0.2, -0.25, 0.1), (0.3, -0.2, 0.5)),
         ((0.0, 0.0, 0.0), (0.0, 0.0, 1.5))]


def _rot(a):
    cx, sx, cy, sy, cz, sz = np.cos(a[0]), np.sin(a[0]), np.cos(a[1]), np.sin(a[1]), np.cos(a[2]), np.sin(a[2])
    rx = np.array([[1, 0, 0], [0, cx, -sx], [0, sx, cx]])
    ry = np.array([[cy, 0, sy], [0, 1, 0], [-sy, 0, cy]])
    rz = np.array([[cz, -sz, 0], [sz, cz, 0], [0, 0, 1]])
    return (rz @ ry @ rx).astype(np.float32)


@pytest.mark.parametrize("res", [(8, 8, 8), (40, 24, 56), (129, 65, 33), (256, 72, 40), (264, 48, 130), (520, 40, 48),
                                 (1024, 16, 24)])
def test_raycast_skips_no_surface(gpu_ctx, res):
    vol = _volume(res, sum(res))
    cfgs = [cfg_for(W=96, H=72, res=res, fmt=f, trunc=0.1) for f in (L.TSDF_I16, L.TSDF_F32, L.TSDF_F16_U8, L.TSDF_F16_F16)]
    ss = [L.Session(gpu_ctx, c) for c in cfgs]
    for s in ss:
        s.upload_volume(vol)
    tsdf = O.OrcTsdf.make(res, tuple(cfgs[0].dim), cfgs[0].trunc_dist)
    cam = O.OrcCam.make(96, 72, cfgs[0].fx, cfgs[0].fy, cfgs[0].cx, cfgs[0].cy, cfgs[0].depth_min, cfgs[0].depth_max)
    for a, t in POSES:
        R = _rot(a)
        t = np.array(t, np.float32)
        v = np.zeros((72 * 96, 3), np.float32)
        n = np.zeros((72 * 96, 3), np.float32)
        xf = O.make_xform(R, t)
        O.oracle().orc_raycast(O.p(vol), None, C.byref(tsdf), C.byref(cam), C.byref(xf), 96, 72, O.p(v), O.p(n), None, None)
        for s in ss:
            s.set_pose(R, t)
            s.raycast()
            g = s.download(3).reshape(-1, 4)[:, :3]
            if s.cfg.tsdf_format in (L.TSDF_I16, L.TSDF_F32):  # (both hold v / 32766)
                assert same_bits(g, v)
                assert same_bits(s.download(4).reshape(-1, 4)[:, :3], n)
            else:
                # a skipped surface would lose its pixels (a blob's are several per cent); those whose
                # crossing lies within a rounding of a voxel or step edge may differ
                both = ~np.isnan(g[:, 0]) & ~np.isnan(v[:, 0])
                assert np.mean(np.isnan(g[:, 0]) != np.isnan(v[:, 0])) < 0.01
                if both.any():
                    assert np.quantile(np.abs(g[both] - v[both]), 0.98) < 1e-3
    for s in ss[:3:2]:  # a restored session's distances are its own
        s.raycast()
        want = s.download(3)
        other = L.Session(gpu_ctx, s.cfg)
        other.restore(s.snapshot())
        other.raycast()
        assert same_bits(other.download(3), want)
        other.close()
    for s in ss:
        s.close()
