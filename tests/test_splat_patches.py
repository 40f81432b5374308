"""DepoFluxSplat patch shapes around the warp's limits: more than 31 ticks or
wires, both edges in one warp's lanes or not, zero widths, and patches cut by
the window and by the first and last wire; against the oracle's restatement.
Tolerance as the truth frame's own tests: float cells, rel-L2 1e-6."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _depos(synth, n, long_mm, tran_mm, seed):
    rng = np.random.default_rng(seed)
    d = np.zeros((n, 7))
    d[:, 0] = rng.uniform(-50.0, 1050.0, n) * synth.us  # some before, some past the window of 1 ms
    d[:, 1] = -rng.uniform(1000.0, 9000.0, n)
    d[:, 2] = synth.RESPONSE_X
    d[:, 3] = rng.uniform(-1500.0, 1500.0, n)
    d[:, 4] = rng.uniform(-2290.0, 2290.0, n)
    d[:, 5] = long_mm
    d[:, 6] = tran_mm
    return d


@pytest.mark.parametrize("long_mm,tran_mm,smear", [
    (1.0, 1.5, True),     # 7 ticks x 3 wires: all edges in one warp
    (2.5, 12.0, False),   # about 28 edges
    (3.3, 14.0, False),   # about 33
    (26.0, 2.0, True),    # 100 ticks
    (4.0, 60.0, False),   # 75 wires
    (0.0, 2.0, False), (2.0, 0.0, False), (0.0, 0.0, False), (0.0, 0.0, True),
])
def test_patch_shapes(wct, oracle, synth, long_mm, tran_mm, smear):
    cfg = synth.apa_config(nticks=2000)
    d = _depos(synth, 400, long_mm, tran_mm, seed=int(10 * long_mm + tran_mm))
    sc = dict(tick=synth.TICK, window_start=0.0, window_duration=2000 * synth.TICK, nsigma=3.0,
              drift_speed=1.6 * synth.mm / synth.us, response_plane=synth.RESPONSE_X,
              time_offsets=[0.0, 3.0 * synth.TICK, -2.0 * synth.TICK])
    if smear:
        sc.update(smear_long=[2.0, 0.0, 3.0], smear_tran=[0.3, 0.6, 0.0])
    out = wct.from_config(cfg).splat(d, **sc)
    ref = oracle.splat(cfg, d, sc)
    assert np.count_nonzero(ref) > 100
    assert rel_l2(out, ref) < 1e-6
