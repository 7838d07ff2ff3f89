"""A wait of the whole-device tracking that runs out (a missing arrival, put there from the host, and
a limit of a thousand polls): the frame reports a device error and not lost tracking, the session
stays where it was, and the context goes on by clusters with the poses it would have had."""
import numpy as np
import pytest

from natureuserinterfacestudio_b200 import _lib as L

from _util import cfg_for, cfg_hash, frames

pytestmark = pytest.mark.gpu

W, H = 320, 240


def _cfg():
    return cfg_for(W=W, H=H, res=(64, 64, 64), trunc=0.1)


def _stall(ctx, polls=1000):
    L.check(L.lib().nui_debug_stall_icp(ctx.h, polls))


def _raises_device(call):
    with pytest.raises(L.NuiError) as e:
        call()
    assert e.value.status == L.NUI_ERR_DEVICE


def _same(a, b):
    return a[0] == b[0] and np.array_equal(a[1], b[1])


@pytest.fixture
def ctx():
    c = L.Context(0)
    yield c
    c.close()


def test_frames(ctx, gpu_ctx):
    seq = frames(5, W=W, H=H, seed=5)
    ref = L.Session(gpu_ctx, _cfg())
    want = [ref.process(d) for d, _, _, _ in seq]
    s = L.Session(ctx, _cfg())
    for i in (0, 1):
        assert _same(s.process(seq[i][0]), want[i])
    _stall(ctx)
    _raises_device(lambda: s.process(seq[2][0]))
    R, t = s.get_pose()
    assert np.array_equal(np.concatenate([R.reshape(9), t]), want[1][1])
    for i in (2, 3, 4):  # the same frame again, then the next ones; other sessions of the context too
        assert _same(s.process(seq[i][0]), want[i])
    other = L.Session(ctx, _cfg())
    for i in (0, 1, 2):
        assert _same(other.process(seq[i][0]), want[i])
    for x in (ref, s, other):
        x.close()


def test_step_wise(ctx, gpu_ctx):
    seq = frames(2, W=W, H=H, seed=5)
    poses = []
    for c in (gpu_ctx, ctx):
        s = L.Session(c, _cfg())
        s.upload(seq[0][0])
        s.feedback_update()
        s.integrate()
        s.upload(seq[1][0])
        if c is ctx:
            _stall(c)
            _raises_device(s.track)
        s.track()
        poses.append(s.get_pose())
        s.close()
    assert all(np.array_equal(a, b) for a, b in zip(*poses))


def test_graphed_batch_of_both_families(ctx, gpu_ctx):
    seq = frames(4, W=W, H=H, seed=5)
    want = None
    for c in (gpu_ctx, ctx):
        ss = [L.Session(c, k) for k in (_cfg(), cfg_hash(), _cfg())]
        got = []
        for i, (d, _, _, _) in enumerate(seq):
            if c is ctx and i == 2:
                _stall(c)
                _raises_device(lambda: c.batch_tick(ss, [d] * 3))
            got.append(np.concatenate([x.reshape(-1) for x in c.batch_tick(ss, [d] * 3)]))
        want = got if want is None else want
        for s in ss:
            s.close()
    assert all(np.array_equal(a, b) for a, b in zip(want, got))


def test_server_delivers_the_frame_as_a_device_error(ctx):
    seq = frames(6, W=W, H=H, seed=5)
    srv = L.Server(ctx, 8 << 30, max_streams=2)
    k = srv.admit(_cfg())
    for i in (0, 1):
        srv.submit(k, seq[i][0], tag=i)
        srv.step()
    srv.drain()
    _stall(ctx)
    for i in (2, 3, 4, 5):
        srv.submit(k, seq[i][0], tag=i)
        srv.step()
    srv.drain()
    st = {r.tag: r.status for r in srv.poll()}
    # (the tick queued behind the stalled one is on the same workspace)
    assert [st[i] == L.NUI_ERR_DEVICE for i in range(6)] == [False, False, True, True, False, False]
    srv.close()
