"""Integration where its splits can go wrong.  Tolerance mode (tiles of 32 x 8 x 8 voxels, two z
slices a warp): single tiles, x sizes whose rows are not whole or not 16-byte aligned, y and z
remainders that leave a warp one slice or none, several sessions of unlike sizes in one launch.
The exact formats (32 columns a block, chunks of z a warp): columns that do not fill a block, z
sizes below, at and past a chunk's and the largest."""
import numpy as np
import pytest

from natureuserinterfacestudio_b200 import _lib as L
from oracle import oracle as O

from _util import cfg_for, frames, integration_near_ties, oracle_preprocess
from test_gpu_parity import _brick_states

pytestmark = pytest.mark.gpu

SIZES = [(32, 8, 8), (33, 9, 9), (40, 17, 15), (48, 8, 10), (80, 23, 11), (96, 40, 29), (130, 64, 63)]


@pytest.mark.parametrize("fmt", [L.TSDF_F16_U8, L.TSDF_F16_F16])
@pytest.mark.parametrize("res", SIZES)
def test_edges_of_tiles(gpu_ctx, res, fmt):
    """Tolerance: that of the larger volumes' comparison with the oracle -- 1e-3 truncation units
    (half precision rounds to 2.4e-4 near 1) and equal weights outside near ties; brick states
    exactly those of the voxels; nothing written outside the volume's voxels (the planes end with
    the volume, so the last brick's states would show it)."""
    W, H = 96, 72
    seq = frames(3, W=W, H=H, seed=4)
    cfg, ref = (cfg_for(W=W, H=H, res=res, fmt=f, trunc=0.2) for f in (fmt, L.TSDF_I16))
    eng = O.Engine(ref)
    s = L.Session(gpu_ctx, cfg)
    exact = L.Session(gpu_ctx, ref)  # the exact kernel of the int16 format, at the same poses
    amb = np.zeros(res[0] * res[1] * res[2], bool)
    for i, (d, _, R, t) in enumerate(seq):
        amb |= integration_near_ties(ref, eng.tsdf, R, t, oracle_preprocess(d, ref)["scaled"], eps_px=3e-3)
        for k in (s, exact):
            k.upload(d)
            k.set_pose(R, t)
            k.integrate()
        vg, vo = s.volume_ref_layout().astype(np.float64), exact.volume_ref_layout().astype(np.float64)
        bad = vg[:, 1] != vo[:, 1]
        both = (vg[:, 1] > 0) & (vo[:, 1] > 0)
        bad |= both & (np.abs(vg[:, 0] - vo[:, 0]) / 32766.0 > 1e-3)
        assert not np.any(bad & ~amb), (i, int(np.sum(bad & ~amb)), int(np.sum(bad)))
        assert exact.touched() > 0 and np.array_equal(s.download(13), _brick_states(s, res)), i
    s.close()
    exact.close()


def test_unlike_sizes_in_one_launch(gpu_ctx):
    """Each session of a batch integrates what it does alone, bit for bit (the roundings of a
    voxel do not depend on the split)."""
    W, H = 96, 72
    seq = frames(3, W=W, H=H, seed=4)
    cfgs = [cfg_for(W=W, H=H, res=r, fmt=L.TSDF_F16_U8, trunc=0.2) for r in SIZES]
    solo, both = ([L.Session(gpu_ctx, c) for c in cfgs] for _ in range(2))
    for i, (d, _, _, _) in enumerate(seq):
        for s in solo:
            s.process(d)
        gpu_ctx.batch_tick(both, [d] * len(both))
        for a, b, r in zip(solo, both, SIZES):
            assert np.array_equal(a.download(6).view(np.uint16), b.download(6).view(np.uint16)), (i, r)
            assert np.array_equal(a.download(14), b.download(14)) and np.array_equal(a.download(13), b.download(13)), (i, r)


@pytest.mark.parametrize("res", [(8, 8, 8), (33, 9, 15), (31, 33, 17), (64, 40, 129), (24, 20, 1024), (9, 8, 1023)])
def test_exact_columns(gpu_ctx, res):
    """The first frame's int16 volume equals the oracle's, the FP32 one its values' twin: the
    same voxels with the same weights."""
    d = frames(1, W=96, H=72, seed=4)[0][0]
    cfg, c32 = (cfg_for(W=96, H=72, res=res, fmt=f, trunc=0.2) for f in (L.TSDF_I16, L.TSDF_F32))
    eng = O.Engine(cfg)
    s, f = L.Session(gpu_ctx, cfg), L.Session(gpu_ctx, c32)
    assert s.process(d)[0] and f.process(d)[0] and eng.frame(d)
    assert s.touched() == f.touched() == eng.touched() > 0
    v = eng.volume().reshape(-1, 2)
    assert np.array_equal(s.volume_ref_layout().reshape(-1, 2), v)
    w = f.volume_ref_layout().reshape(-1, 2)
    assert np.array_equal(w[:, 1], v[:, 1]) and np.max(np.abs(w[:, 0] - v[:, 0].astype(np.int32))) <= 1
    s.close()
    f.close()


@pytest.mark.parametrize("fmt", [L.TSDF_F16_U8, L.TSDF_F16_F16])
@pytest.mark.parametrize("res", [(40, 160, 160), (8, 160, 200)])
def test_rows_of_more_tiles_than_a_quarter_of_their_bricks(gpu_ctx, res, fmt):
    """Rows that end with a tile of one to three bricks: the volume's last tiles, hundreds past a
    quarter of its bricks, are integrated like the others (same comparison)."""
    ntx, nbx, n = (res[0] + 31) // 32, (res[0] + 7) // 8, (res[1] // 8) * (res[2] // 8)
    first = -(-(nbx * n // 4 + 1) // 256) * 256  # tiles from here on had no thread in the cull
    assert first < ntx * n
    d, _, R, t = frames(1, W=96, H=72, seed=4)[0]
    ref = L.Session(gpu_ctx, cfg_for(W=96, H=72, res=res, fmt=L.TSDF_I16, trunc=0.2))
    ref.upload(d)
    ref.set_pose(R, t)
    ref.integrate()
    w = ref.volume_ref_layout().reshape(res[1], res[0], res[2], 2)[..., 1]
    assert np.sum(w[:, :, 8 * -(-first // (ntx * (res[1] // 8))):] > 0) > 100  # in view
    ref.close()
    test_edges_of_tiles(gpu_ctx, res, fmt)
