"""The launch routes of the ICP: few sessions over the whole device (k_icp_wide), clusters with
and without the photometric rows, block sizes by image size -- the same poses by
every route, at the edges of the rules -- and the shared-reciprocal quotients of the
photometric rows against the division they replace."""
import ctypes as C
import random
import threading
from fractions import Fraction

import numpy as np
import pytest

from natureuserinterfacestudio_b200 import _lib as L
from oracle import oracle as O

from _util import cfg_for, frames, rot_angle


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,color", [(512, 512, False), (508, 512, False), (516, 508, False), (128, 128, True),
                                       (124, 128, True), (132, 124, True), (64, 48, False)])
def test_one_session_and_many_agree(gpu_ctx, W, H, color):
    """n = 1 (the whole-device route) against the same
    stream nine times in a batch (clusters only): the routes regroup FP64 sums, so poses agree
    within the 1e-5 that the ICP shapes are held to; depth poses agree with the oracle's."""
    cfg = cfg_for(W=W, H=H, res=(64, 64, 64), color=color, trunc=0.1)
    cfg.photometric_weight = 0.1 if color else 0.0
    seq = frames(4, W=W, H=H, seed=5, color=color)
    one = L.Session(gpu_ctx, cfg)
    many = [L.Session(gpu_ctx, cfg) for _ in range(9)]
    eng = None if color else O.Engine(cfg)
    for d, c, _, _ in seq:
        ok, p = one.process(d, c)
        st, q = gpu_ctx.batch_tick(many, [d] * 9, [c] * 9 if color else None)
        assert np.all((st == 0) == ok)  # (the smallest image loses tracking, by every route)
        assert np.array_equal(q, np.repeat(q[:1], 9, axis=0))
        assert rot_angle(p[:9].reshape(3, 3), q[0, :9].reshape(3, 3)) < 1e-5
        assert np.max(np.abs(p[9:] - q[0, 9:])) < 1e-5
        if eng is not None:
            assert bool(eng.frame(d)) == ok
            R, t = eng.pose()
            assert rot_angle(p[:9].reshape(3, 3), R) < 1e-4 and np.max(np.abs(p[9:] - t)) < 1e-4
    for s in [one] + many:
        s.close()


@pytest.mark.gpu
def test_lost_at_a_coarse_level_stays_lost(gpu_ctx):
    """A frame that loses tracking in the clusters' levels does not go on at level 0 from what
    an earlier frame (of another session) left in the whole-device route's workspace: the flat
    wall of test_gpu_lost after a frame whose single iteration ends level 0 undone."""
    W = H = 512
    other = L.Session(gpu_ctx, cfg_for(W=W, H=H, res=(64, 64, 64), trunc=0.1, iters=(1, 0, 0)))
    wall = L.Session(gpu_ctx, cfg_for(W=W, H=H, res=(64, 64, 64)))
    flat = np.full((H, W), 1500, np.uint16)
    ok, first = wall.process(flat)
    assert ok
    for d, _, _, _ in frames(3, W=W, H=H, seed=5, deg=4.0):
        assert other.process(d)[0]
        ok, p = wall.process(flat)
        assert not ok and np.array_equal(p, first)
        assert wall.work_counters()["icp_iters"][:3] == [0, 0, 1]  # lost by the first iteration of the coarsest level
    for s in (other, wall):
        s.close()


@pytest.mark.gpu
def test_contexts_on_threads_track_at_once():
    """Each context's whole-device launch fills the device, and several may be launched at once
    (threads, each with a context and its streams): every one runs to its end, with the poses it
    gives alone."""
    W, H = 320, 240
    seq = frames(6, W=W, H=H, seed=5)
    cfg = cfg_for(W=W, H=H, res=(64, 64, 64), trunc=0.1)

    def run(out, laps):
        ctx = L.Context(0)
        for _ in range(laps):
            s = L.Session(ctx, cfg)
            out.append([s.process(d) for d, _, _, _ in seq])
            s.close()

    alone, many = [], [[] for _ in range(4)]
    run(alone, 1)
    ts = [threading.Thread(target=run, args=(o, 12)) for o in many]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for o in many:
        assert len(o) == 12
        for lap in o:
            for (ok, p), (ok0, p0) in zip(lap, alone[0]):
                assert ok == ok0 and np.array_equal(p, p0)


@pytest.mark.gpu
def test_first_trackings_of_a_context_on_threads(gpu_ctx):
    """Sessions of one context may be called from several threads, its first trackings too: the
    workspace is allocated once, and every thread tracks to the poses of a context that one uses."""
    W, H, N = 160, 120, 6
    cfg, seq = cfg_for(W=W, H=H, res=(64, 64, 64), trunc=0.1, iters=(4, 3, 3)), frames(2, W=W, H=H, seed=5)

    def count():
        n = C.c_uint64()
        L.check(L.lib().nui_debug_allocation_count(C.byref(n)))
        return n.value

    def track(s, bar, out):
        s.upload(seq[0][0])
        s.feedback_update()
        s.upload(seq[1][0])
        if bar:
            bar.wait()
        s.track()
        out.append(s.get_pose())

    want, allocations = [], []
    for threads in (1, N, N, N, N):
        ctx = L.Context(0)
        ss = [L.Session(ctx, cfg) for _ in range(N)]
        L.check(L.lib().nui_ctx_synchronize(ctx.h))
        n0, out, bar = count(), [], threading.Barrier(N) if threads > 1 else None
        if threads == 1:
            for s in ss:
                track(s, None, out)
        else:
            ts = [threading.Thread(target=track, args=(s, bar, out)) for s in ss]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
        assert len(out) == N
        want = want or out[0]
        assert all(np.array_equal(a, b) for p in out for a, b in zip(p, want))
        allocations.append(count() - n0)
        for s in ss:
            s.close()
        ctx.close()
    assert len(set(allocations)) == 1, allocations


def _f32(x):
    """The float32 nearest to a rational (ties to even), as a Fraction; normal range."""
    if x == 0:
        return Fraction(0)
    s, x, e = (-1, -x, 0) if x < 0 else (1, x, 0)
    while x >= 1 << 24:
        x, e = x / 2, e + 1
    while x < 1 << 23:
        x, e = x * 2, e - 1
    n, r = divmod(x.numerator, x.denominator)
    r = Fraction(r, x.denominator)
    n += 1 if r > Fraction(1, 2) or (r == Fraction(1, 2) and n & 1) else 0
    return s * n * Fraction(2) ** e


def test_shared_reciprocal_quotient_is_the_division():
    """div_shared's steps in exact arithmetic with one rounding each, against the rounded
    quotient: random and extreme mantissas over the range it is used in."""
    rng = random.Random(7)

    def value(lo, hi):
        m = rng.choice([rng.randrange(1 << 23, 1 << 24), (1 << 24) - 1 - rng.randrange(4), (1 << 23) + rng.randrange(4)])
        return Fraction(m) * Fraction(2) ** (rng.randint(lo, hi) - 23)

    for _ in range(3000):
        a, b = value(-60, 59) * rng.choice([-1, 1]), value(-40, 39)
        r = _f32(1 / b)
        q = _f32(a * r)
        for _ in range(2):
            q = _f32(q + _f32(a - q * b) * r)
        assert q == _f32(a / b), (a, b)


def _quotients(ctx, a, b):
    torch = pytest.importorskip("torch")
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    q = torch.empty_like(ta)
    torch.cuda.synchronize()
    L.check(L.lib().nui_debug_quotients(ctx.h, ta.data_ptr(), tb.data_ptr(), q.data_ptr(), a.size))
    return q.cpu().numpy()


def _random(rng, n, lo, hi):
    """Floats of 2^lo .. 2^(hi + 1), a third of them with mantissas at the ends of the binade."""
    m = rng.integers(1 << 23, 1 << 24, n)
    k = rng.integers(0, 6, n)
    m = np.where(k == 0, (1 << 23) + rng.integers(0, 4, n), np.where(k == 1, (1 << 24) - 1 - rng.integers(0, 4, n), m))
    return np.ldexp(m.astype(np.float64), rng.integers(lo, hi + 1, n) - 23).astype(np.float32)


@pytest.mark.gpu
def test_device_quotients_are_the_division(gpu_ctx):
    """The rows' quotients over the whole range they claim (numerators of 2^-80 .. 2^80 and zero,
    denominators of 2^-40 .. 2^40), bit for bit; below it, where a numerator cancels, two ulps."""
    rng, n = np.random.default_rng(11), 1 << 20
    b = _random(rng, n, -40, 39)
    a = _random(rng, n, -80, 79) * rng.choice(np.array([-1, 1], np.float32), n)
    a[:64] = 0
    want = (a.astype(np.float64) / b.astype(np.float64)).astype(np.float32)  # (53 bits: no double rounding)
    assert np.array_equal(_quotients(gpu_ctx, a, b), want)
    a = _random(rng, n, -126, -81) * rng.choice(np.array([-1, 1], np.float32), n)
    exact = a.astype(np.float64) / b.astype(np.float64)
    ulp = np.maximum(np.spacing(np.abs(exact).astype(np.float32)).astype(np.float64), 2.0 ** -149)
    assert np.max(np.abs(_quotients(gpu_ctx, a, b).astype(np.float64) - exact) / ulp) <= 2.0
