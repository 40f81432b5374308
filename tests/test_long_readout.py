"""Readouts of more than 8192 ticks: the batched path's time-FFT lengths stay
close to the windows'.  The ladder's steps are 10 %, a length is rounded up by
at most 15 % of itself."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TICK = 500.0
NWIRES = 960


def _event(synth, nticks, span, n=60, seed=1, wires=(300.0, 460.0)):
    """Depos whose arrival spans about `span` ticks from tick 40 on."""
    rng = np.random.default_rng(seed)
    d = np.zeros((n, 7))
    d[:, 1] = -5000.0 * (0.5 + rng.random(n))
    d[:, 2] = synth.RESPONSE_X + 300.0
    drift = 300.0 / synth.DRIFT["drift_speed"]
    t = np.concatenate([[0.0, 1.0], rng.random(n - 2)])
    d[:, 0] = (40.0 + t * (span - 1)) * TICK - drift
    w = wires[0] + (wires[1] - wires[0]) * rng.random(n)
    d[:, 4] = (w - 0.5 * (NWIRES - 1)) * 4.79
    return d


@pytest.mark.parametrize("nticks", [6000, 8500, 9600, 12500])
def test_batch_lengths_follow_the_windows(wct, synth, nticks):
    dt = wct.from_config(synth.plane1_config(nticks=nticks))
    spans = [s for s in (500, 1300, 2400, 4200, 5000, 5900, 7000, 7700, 8300, 8900, 9400, 10200, 12300)
             if s <= nticks - 100]
    _, wins, _ = dt.forward_batch([_event(synth, nticks, s) for s in spans])
    for w in wins:
        assert w[0]["nt_fft"] <= w[0]["nt_gpu"] <= 1.155 * w[0]["nt_fft"], w[0]
