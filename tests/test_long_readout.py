"""Readouts of more than 8192 ticks: the batched path's time-FFT lengths stay
close to the windows', a short event takes the same kernels as in a component
of fewer ticks, and the forms that only long windows reach give the oracle's
frames.

The ladder's steps are 10 %, a length is rounded up by at most 15 % of itself.
Frames: rel-L2, 6e-8 a butterfly stage over about 15 + 10 stages, the
convolution's sums and the bin integrals' 1.2e-7, times four."""

import numpy as np
import pytest

from conftest import rel_l2

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


# a window of 8960 ticks (three-stage rows), of 12000 (the longest of those; its wire spectra are over the bound
# of a plane: direct convolution and adjoint), of 14336 (generic row transforms)
LONG = [(8500, 8300), (11950, 11700), (12500, 12400)]
TOL = 2e-6


@pytest.mark.parametrize("nticks,span", LONG)
def test_long_windows_against_oracle(wct, oracle, synth, nticks, span):
    cfg = synth.plane1_config(nticks=nticks)
    cfg["pir_nticks"] = 2000
    dt = wct.from_config(cfg)
    d = _event(synth, nticks, span)
    short = _event(synth, nticks, 900, seed=2)
    o = [oracle.run(cfg, e, fp64=True)["frames"][0] for e in (d, short)]
    frame, _, _ = dt(d)
    assert rel_l2(frame, o[0]) < TOL
    frames, _, _ = dt.forward_batch([d, short])
    for k in range(2):
        assert rel_l2(frames[k], o[k]) < TOL, k
    # the adjoint is the transpose: positive weights on a unipolar response, no cancellation
    G = np.random.default_rng(5).random(frame.shape).astype(np.float32)
    gd, _ = dt.adjoint(d, G)
    lhs = float(np.sum(G.astype(np.float64) * frame))
    assert abs(float(np.sum(d[:, 1] * gd[:, 1])) - lhs) < TOL * abs(lhs)


@pytest.mark.parametrize("nticks", [8500, 12500])
def test_short_event_as_in_a_short_readout(wct, synth, nticks):
    """The form of the convolution goes by the event's own length, not by the
    component's longest: the same bits as from a component of 6000 ticks."""
    ev = [_event(synth, 6000, s, seed=s) for s in (400, 1500, 3000)]
    out = []
    for n in (6000, nticks):
        cfg = synth.plane1_config(nticks=n)
        cfg["pir_nticks"] = 2000
        out.append(wct.from_config(cfg).forward_batch(ev)[0])
    assert np.array_equal(out[0], out[1][:, :, :6000])
    assert not np.any(out[1][:, :, 6000:])
