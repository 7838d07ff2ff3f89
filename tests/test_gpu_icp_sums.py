"""The ICP's FP64 sums are formed in an order that the image size alone fixes: a session's state --
the accepted normal equations in FP64 among it -- is the same bytes whether it is tracked alone or in
a batch, over the whole device or by clusters of any size and width, and whatever its neighbours do."""
import numpy as np
import pytest

from natureuserinterfacestudio_b200 import _lib as L

from _util import cfg_for, cfg_hash, frames

pytestmark = pytest.mark.gpu

STATE = 4096  # bytes of a snapshot that hold the tracker's state (and the first points of a map)
DEFAULT = (18, 4, 8, 8, 12)


def _cfg(W, H, color, iters=(4, 3, 3)):
    cfg = cfg_for(W=W, H=H, res=(64, 64, 64), color=color, trunc=0.1, iters=iters)
    cfg.photometric_weight = 0.1 if color else 0.0
    return cfg


def _hash(color=True):
    cfg = cfg_hash(W=160, H=120, color=color, buckets=1 << 12, excess=1 << 10, pool=1 << 12, voxel=0.02, mu=0.08,
                   fmt=L.TSDF_F16_U8, iters=(4, 3, 3))
    cfg.photometric_weight = 0.1 if color else 0.0
    return cfg


def _alone(ctx, cfg, seq):
    """The state after every frame of a session that is the only one of its ticks."""
    s = L.Session(ctx, cfg)
    out = []
    for d, c, _, _ in seq:
        ctx.batch_tick([s], [d], [c] if c is not None else None)
        out.append(s.snapshot()[:STATE].copy())
    s.close()
    return out


def _together(ctx, cfgs, seqs):
    ss = [L.Session(ctx, c) for c in cfgs]
    out = [[] for _ in ss]
    for f in range(len(seqs[0])):
        ctx.batch_tick(ss, [q[f][0] for q in seqs], [q[f][1] if q[f][1] is not None else None for q in seqs])
        for s, o in zip(ss, out):
            o.append(s.snapshot()[:STATE].copy())
    for s in ss:
        s.close()
    return out


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("W,H,color", [(64, 48, False), (188, 132, False), (320, 240, False), (640, 480, False),
                                       (1280, 720, False), (64, 48, True), (188, 132, True), (640, 480, True)])
def test_state_does_not_depend_on_the_number_of_sessions(gpu_ctx, W, H, color):
    """n = 1 .. 4 (shares of the whole device), 5 .. 8 and 9 (clusters of wider and narrower blocks),
    each tick between the same frames."""
    cfg, seq = _cfg(W, H, color), frames(4, W=W, H=H, seed=5, color=color)
    ref = _alone(gpu_ctx, cfg, seq)
    for n in (2, 3, 4, 5, 6, 8, 9):
        for i, o in enumerate(_together(gpu_ctx, [cfg] * n, [seq] * n)):
            assert _same(o, ref), (n, i)


def test_state_does_not_depend_on_the_neighbours(gpu_ctx):
    """A depth session beside a colour-tracked one, beside one of a larger image, and beside
    voxel-hash sessions (tracked on a second stream, each launch over half the device), few and
    many of them."""
    seq = {c: frames(4, W=160, H=120, seed=5, color=c) for c in (False, True)}
    big = frames(4, W=640, H=480, seed=3)
    kinds = {"depth": (_cfg(160, 120, False), seq[False]), "color": (_cfg(160, 120, True), seq[True]),
             "big": (_cfg(640, 480, False), big), "hash": (_hash(), seq[True]), "hashd": (_hash(False), seq[False])}
    ref = {k: _alone(gpu_ctx, *v) for k, v in kinds.items()}
    for mix in (["depth", "color"], ["depth", "big"], ["depth", "hash"], ["depth", "depth", "depth", "hash", "hashd"],
                ["depth", "color", "hash"], ["depth"] * 5 + ["hash"] * 2, ["depth"] * 9 + ["color"],
                ["depth"] * 5 + ["big"] + ["hash"] * 9):
        for k, o in zip(mix, _together(gpu_ctx, [kinds[k][0] for k in mix], [kinds[k][1] for k in mix])):
            assert _same(o, ref[k]), (mix, k)


@pytest.mark.parametrize("W,H,color", [(188, 132, False), (640, 480, False), (188, 132, True)])
def test_state_does_not_depend_on_the_cluster(gpu_ctx, W, H, color):
    """Every cluster size, two sessions past the whole-device launch, and the pixels a thread."""
    cfg, seq = _cfg(W, H, color), frames(3, W=W, H=H, seed=5, color=color)
    gpu_ctx.set_tuning(L.Tuning(*DEFAULT))
    ref = _alone(gpu_ctx, cfg, seq)
    try:
        for cl in range(2, 17):
            gpu_ctx.set_tuning(L.Tuning(18, (2, 4, 8, 16)[cl % 4], 8, 8, cl))
            for n in (5, 10):
                for o in _together(gpu_ctx, [cfg] * n, [seq] * n):
                    assert _same(o, ref), (cl, n)
    finally:
        gpu_ctx.set_tuning(L.Tuning(*DEFAULT))
