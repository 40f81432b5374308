"""Patch placement where a quotient is a whole number or next to one, and depos
on the border of the rejection cuts: a few steps of the last place to either
side.  Bins, counters and windows are whole numbers: equal to the oracle's."""

import numpy as np
import pytest

from test_gpu_forward import _records_match, _windows_match

pytestmark = pytest.mark.gpu


def _steps(v, k):
    """v moved by k units of its last place."""
    return v + k * np.spacing(np.abs(v))


def _on_edges(synth, n, sigma):
    rng = np.random.default_rng(n)
    tick, imp, speed = 500.0, 4.79 / 10, 1.6e-3
    pmin, end = -0.5 * 4.79 * 960, 1500 * tick
    d = np.zeros((n, 7))
    d[:, 1] = -1000.0
    d[:, 2] = synth.RESPONSE_X
    st = rng.integers(1, 12, n) * tick / 3 * sigma
    d[:, 5] = st * speed
    st = d[:, 5] / speed
    d[:, 6] = rng.integers(1, 8, n) * imp / 3 * sigma
    sp = d[:, 6]
    kind = np.arange(n) % 5  # inside, at the four borders of the cuts
    t = rng.integers(0, 1500, n) * tick
    p = pmin + rng.integers(0, 9600, n) * imp
    t = np.where(kind == 1, 0.0 - 3 * st, np.where(kind == 2, end + 3 * st, t))
    p = np.where(kind == 3, pmin - 3 * sp, np.where(kind == 4, -pmin + 3 * sp, p))
    d[:, 0] = _steps(t, rng.integers(-2, 3, n))
    d[:, 4] = _steps(p, rng.integers(-2, 3, n))
    return d


@pytest.mark.parametrize("sigma", [0.0, 1.0])
@pytest.mark.parametrize("n", [1, 33, 257, 5000])
def test_bins_on_edges(wct, oracle, synth, n, sigma):
    cfg = synth.plane1_config(nticks=1500)
    cfg.pop("drifter")
    d = _on_edges(synth, n, sigma)
    dt = wct.from_config(cfg)
    _, wins, _ = dt(d)
    o = oracle.run(cfg, d, fp64=True, records=True)
    _windows_match(wins, o["windows"])
    _records_match(dt, cfg, o["records"], n)
