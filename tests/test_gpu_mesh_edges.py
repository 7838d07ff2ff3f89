"""Marching cubes at the edges of its tiling (128 columns a block, 32 columns and 32 slices a
warp's chunk, 8 slices a step): volumes one below, at and one above them, of every storage
format, against the oracle's extraction; and a scene whose surfaces lie on the chunk borders."""
import ctypes as C

import numpy as np
import pytest

from natureuserinterfacestudio_b200 import _lib as L
from oracle import oracle as O

from _util import cfg_for, same_bits

pytestmark = pytest.mark.gpu


def _volume(res, seed):
    """Blobs, planes on multiples of 8 and 32, noise, unweighted voxels; reference layout."""
    rng = np.random.default_rng(seed)
    rx, ry, rz = res
    x, y, z = np.meshgrid(np.arange(rx), np.arange(ry), np.arange(rz), indexing="ij")
    f = np.minimum(np.abs((z % 32) - 31.5) - 1.2, np.abs((x % 32) - 31.5) - 0.9)
    f = np.minimum(f, np.sqrt((x - rx / 2) ** 2 + (y - ry / 2) ** 2 + (z - rz / 2) ** 2) - min(res) / 3)
    f = f + rng.normal(0, 0.1, f.shape)
    v = np.zeros(res + (2,), np.int16)
    v[..., 0] = np.clip(f / 3, -1, 1) * 32766
    v[..., 1] = rng.integers(0, 40, f.shape) * ((f > -2.5) & (rng.random(f.shape) > 0.01))
    return np.ascontiguousarray(v.transpose(1, 0, 2, 3).reshape(-1, 2))  # (x + y rx) rz + z


@pytest.mark.parametrize("res", [(8, 8, 8), (33, 9, 33), (32, 17, 32), (34, 8, 65), (128, 10, 64), (129, 12, 97),
                                 (130, 9, 10), (200, 31, 1024), (9, 40, 257)])
@pytest.mark.parametrize("fmt", [L.TSDF_I16, L.TSDF_F32, L.TSDF_F16_U8, L.TSDF_F16_F16])
def test_edges(gpu_ctx, res, fmt):
    import torch
    cfg = cfg_for(W=64, H=48, res=res, fmt=fmt)
    s = L.Session(gpu_ctx, cfg)
    vol = _volume(res, seed=sum(res))
    s.upload_volume(vol)
    rx, ry, rz = res
    cases_o = np.zeros((rx - 1) * (ry - 1) * (rz - 1), np.uint8)
    tsdf = O.OrcTsdf.make(res, tuple(cfg.dim), cfg.trunc_dist)
    count = lambda c, p, cap: O.oracle().orc_marching_cubes(O.p(vol), None, C.byref(tsdf), c, p, None, cap)
    n = count(O.p(cases_o), None, 0)
    pos_o = np.zeros((n, 3), np.float32)
    assert n > 0 and count(None, O.p(pos_o), n) == n
    cases, k = s.mesh_cases()
    assert k == n and np.array_equal(cases, cases_o)  # every format keeps the signs
    cap = n + 7
    pos = torch.full((cap, 3), -9.0, device="cuda")
    k = C.c_uint64()
    torch.cuda.synchronize()
    assert L.lib().nui_mesh_device_noalloc(s.h, C.c_void_p(pos.data_ptr()), None, cap, C.byref(k)) == L.NUI_OK
    pos = pos.cpu().numpy()
    assert k.value == n and np.all(pos[n:] == -9.0)
    if fmt in (L.TSDF_I16, L.TSDF_F32):
        assert same_bits(pos[:n], pos_o)
    else:
        # a half holds each corner's tsdf within 2^-11 (1e-3 for the smallest, near 1 / 32766):
        # the crossing a / (a - b) moves by less than 4e-3 of an edge
        assert np.max(np.abs(pos[:n] - pos_o)) < 4e-3 * 3.0 / min(res)
    s.close()
