"""Session snapshot / restore: a session restored from a snapshot continues exactly as the
snapshotted one -- the same poses bit for bit, the same volume -- for a dense colour volume,
a voxel hash and a shifting volume; a snapshot does not load into another configuration."""
import numpy as np
import pytest

from natureuserinterfacestudio_b200 import _lib as L

from _util import cfg_for, cfg_hash, frames

pytestmark = pytest.mark.gpu


def _cases():
    shift = cfg_for(W=320, H=240, res=(96, 80, 112), dim=3.0, color=True)
    shift.voxel_shift = 3
    return [
        ("dense colour", cfg_for(W=320, H=240, res=(128, 128, 128), color=True), True),
        ("hash", cfg_hash(), False),
        ("shifting", shift, True),
    ]


@pytest.mark.parametrize("name,cfg,color", _cases(), ids=[c[0] for c in _cases()])
def test_restored_session_continues_identically(gpu_ctx, name, cfg, color):
    seq = frames(7, W=320, H=240, seed=5, deg=1.0, color=True, kind=L.SYNTH_ROOM)
    a = L.Session(gpu_ctx, cfg)
    for d, c, _, _ in seq[:4]:
        assert a.process(d, np.ascontiguousarray(c) if color else None)[0]
    snap = a.snapshot()
    first = [a.process(d, np.ascontiguousarray(c) if color else None)[1] for d, c, _, _ in seq[4:]]
    b = L.Session(gpu_ctx, cfg)
    b.restore(snap)
    second = [b.process(d, np.ascontiguousarray(c) if color else None)[1] for d, c, _, _ in seq[4:]]
    for p1, p2 in zip(first, second):
        assert np.array_equal(p1, p2), name
    if cfg.volume_kind == L.VOLUME_DENSE:
        assert np.array_equal(a.volume_ref_layout(), b.volume_ref_layout())
        assert np.array_equal(a.shift_state()[0], b.shift_state()[0])
    else:
        assert np.array_equal(a.hash_download(22), b.hash_download(22))
    other = L.Session(gpu_ctx, cfg_for(W=320, H=240, res=(64, 64, 64)))
    with pytest.raises(L.NuiError):
        other.restore(snap)
    for s in (a, b, other):
        s.close()


def test_pose_and_restore_while_another_device_is_current(gpu_ctx):
    """nui_set_pose and nui_session_restore work on the session's device whatever the calling
    thread's current one is, and leave that as it was."""
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    cfg = cfg_for(W=320, H=240, res=(64, 64, 64), trunc=0.1)
    d, _, R, t = frames(1, W=320, H=240, seed=5)[0]
    s = L.Session(gpu_ctx, cfg)
    assert s.process(d)[0]
    snap = s.snapshot()
    with torch.cuda.device(1):
        s.set_pose(R, t)
        r2, t2 = s.get_pose()
        s.restore(snap)
        assert torch.cuda.current_device() == 1
    assert np.array_equal(r2, np.asarray(R, np.float32)) and np.array_equal(t2, np.asarray(t, np.float32))
    assert np.array_equal(s.snapshot(), snap)
    s.close()
