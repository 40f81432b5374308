"""The adjoint's gather over patch shapes around its limits: 8, 16, 32 and 128
ticks side by side and one more, more than 128 impacts, zero widths in time, in
pitch and in both; a depo's gradient of a weighted sum of the frame against the
FP64 gradient, at the tolerance of the adjoint's own tests (1e-4 per
coordinate), for the widths at ten times that: theirs are second differences of
weights of up to a hundred, known to single precision."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("long_mm,tran_mm", [
    (0.9, 1.0), (1.05, 1.0),     # about 8 and 9 ticks
    (2.0, 3.0), (2.15, 3.0),     # 16, 17
    (4.1, 1.5), (4.3, 1.5),      # 32, 33
    (17.0, 1.0), (17.3, 1.0),    # 128, 129
    (2.0, 10.5), (20.0, 12.0),   # 135 and 154 impacts, the latter with 150 ticks
    (0.0, 1.0), (1.0, 0.0), (0.0, 0.0),
])
def test_shapes(wct, oracle, synth, long_mm, tran_mm):
    import adjoint as A
    cfg = synth.plane1_config(nticks=2000, nwire_half=10)
    cfg["drifter"] = None  # the depo's own widths reach the plane
    d = np.array([[412.3 * synth.us, -5000.0, synth.RESPONSE_X, 0.0, 37.1, long_mm, tran_mm]])
    m = A.FrozenModel(cfg, d)
    F = m.base_frames[0]
    # weights that every coordinate moves without cancellation: a slope and a
    # parabola about the centre of the frame's charge, in time and across wires
    w, t = (np.arange(n, dtype=np.float64) for n in F.shape)
    wc, tc = (F.sum(axis=1) @ w) / F.sum(), (F.sum(axis=0) @ t) / F.sum()
    x, y = (w - wc)[:, None] / 8.0, (t - tc)[None, :] / 40.0
    g = (1.0 + x + y + x * x + y * y).astype(np.float32)
    gd, _ = wct.from_config(cfg).adjoint(d, g)
    ref, _ = m.gradient([g.astype(np.float64)])
    for k in range(7):
        tol = 1e-3 if k >= 5 else 1e-4
        assert abs(gd[0, k] - ref[0, k]) <= tol * abs(ref[0, k]), (k, gd[0, k], ref[0, k])
