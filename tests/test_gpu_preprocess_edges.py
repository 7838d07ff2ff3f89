"""The paired bilateral of k_preprocess (radius 3) at the edges of its 32 x 16 tiles, and the
thresholds at which it hands over to the general taps, against the oracle bit for bit; raw
depths of 0 that the range admits (negative minimum) count for no tap but keep their pixel."""
import ctypes as C

import numpy as np
import pytest

from natureuserinterfacestudio_b200 import _lib as L
from oracle import oracle as O

from _util import same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 1), (2, 3), (31, 15), (32, 16), (33, 17), (65, 49), (160, 120)])
@pytest.mark.parametrize("radius,sd2,thr,dmin", [(3, 50.0, 0.3, 0.5), (3, 50.0, 0.3, -1.0), (3, 0.0, 5.0, 0.5),
                                                 (3, 966.0, 0.3, 0.5), (3, 970.0, 0.3, 0.5), (2, 50.0, 0.3, 0.5),
                                                 (3, 0.0, 3e29, 0.5)])
def test_preprocess_edges(gpu_ctx, W, H, radius, sd2, thr, dmin):
    import torch
    rng = np.random.default_rng(W * 131 + H)
    raw = (1200 + 400 * rng.standard_normal((H, W)).cumsum(axis=1) * 0.02).clip(0, 5000)
    raw = np.where(rng.random((H, W)) < 0.1, 0, raw).astype(np.uint16)
    f = 525.0
    cx, cy = (W - 1) / 2.0, (H - 1) / 2.0
    d = torch.from_numpy(raw.view(np.int16)).cuda()
    out, vert, sc = (torch.zeros(s, device="cuda") for s in ((H, W), (H, W, 4), (H, W)))
    torch.cuda.synchronize()
    p = lambda t: C.c_void_p(t.data_ptr())
    L.check(L.lib().nui_k_preprocess(gpu_ctx.h, p(d), W, H, f, f, cx, cy, dmin, 4.5, radius, 0.08, sd2, thr, p(out),
                                     p(vert), p(sc)))
    orc, N = O.oracle(), W * H
    a, g, want, scaled = (np.zeros(n, np.float32) for n in (N, 2 * radius + 1, N, N))
    cam = O.OrcCam.make(W, H, f, f, cx, cy, dmin, 4.5)
    orc.orc_pass_filter(O.p(raw.reshape(-1)), N, dmin, 4.5, O.p(a))
    orc.orc_gaussian_table(radius, 0.08, O.p(g))
    orc.orc_bilateral(O.p(a), W, H, O.p(g), radius, sd2, thr, O.p(want))
    scaled[:] = a
    orc.orc_scale_depths(O.p(scaled), W, H, C.byref(cam))
    assert same_bits(out.cpu().numpy().reshape(-1), want)
    assert same_bits(sc.cpu().numpy().reshape(-1), scaled)
