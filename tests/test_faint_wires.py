"""Wires with little charge beside bright ones keep their own precision: rows one
by one against the 64-bit oracle, and a gradient that is not a number stays
within the response's width.

Tolerance, per row: the row transforms and the convolution's sums as for whole
frames, 6e-8 a butterfly stage over about 25 stages, plus the overlap-save
blocks' rounding of at most twice 1.5e-7 where a row keeps it; times three."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-6
NWIRES = 960


def _depos(synth, wires, q, seed, rows=NWIRES):
    rng = np.random.default_rng(seed)
    w = np.asarray(wires, dtype=np.float64)
    d = np.zeros((len(w), 7))
    d[:, 1] = q
    d[:, 2] = synth.RESPONSE_X + 200.0 + 300.0 * rng.random(len(w))
    d[:, 4] = (w - 0.5 * (rows - 1)) * 4.79
    return d


def _uneven(synth, ratio, seed=0):
    """A bright group of wires, faint ones before and after it, near and far."""
    rng = np.random.default_rng(seed)
    faint = np.concatenate([200 + 6 * rng.random(8), 380 + 5 * rng.random(8), 700 + 90 * rng.random(20)])
    return np.concatenate([_depos(synth, [300.2, 301.1], -5e7, 1), _depos(synth, faint, -5e7 / ratio, 2)])


def _row_errors(f, o):
    """Each live row's error over its norm, and the rows."""
    n = np.linalg.norm(o, axis=1)
    live = n > 0
    return np.linalg.norm(f[live].astype(np.float64) - o[live], axis=1) / n[live], np.nonzero(live)[0]


def _near(rows, wires, half):
    return np.min(np.abs(rows[:, None] - np.asarray(wires)[None, :]), axis=1) <= half


@pytest.mark.parametrize("half", [21, 10, 4])
@pytest.mark.parametrize("ratio", [1.0, 30.0, 1e3, 1e5])
def test_rows_against_oracle(wct, oracle, synth, ratio, half):
    cfg = synth.plane1_config(nticks=2000, nwire_half=half)
    d = _uneven(synth, ratio)
    o = oracle.run(cfg, d, fp64=True)["frames"][0].astype(np.float64)
    dt = wct.from_config(cfg)
    wires = d[:, 4] / 4.79 + 0.5 * (NWIRES - 1)
    frame, _, _ = dt(d)
    batch, _, _ = dt.forward_batch([d, d[:5]])
    for f in (frame, batch[0]):
        err, rows = _row_errors(f, o)
        # (past the response's edge the oracle's transform leaves rounding of its own)
        assert np.max(err[_near(rows, wires, half)]) < TOL


@pytest.mark.parametrize("half", [21, 40])
def test_gradient_rows_of_faint_weights(wct, synth, half):
    """dL/dq of faint depos where dL/dframe is 1e5 times larger some blocks of wires away: as without that."""
    cfg = synth.plane1_config(nticks=2000, nwire_half=half)
    rng = np.random.default_rng(3)
    d = _depos(synth, 200.0 + 500.0 * rng.random(60), -5000.0, 4)
    dt = wct.from_config(cfg)
    G = rng.random((NWIRES, 2000)).astype(np.float32)
    plain, _ = dt.adjoint(d, G)
    lo, hi = 420, 470
    bright = G.copy()
    bright[lo:hi] *= 1e5
    got, _ = dt.adjoint(d, bright)
    w = d[:, 4] / 4.79 + 0.5 * (NWIRES - 1)
    out = (w < lo - half - 4) | (w > hi + half + 4)
    assert out.sum() > 20
    a, b = got[out, 1], plain[out, 1]
    assert np.max(np.abs(a - b) / np.abs(b)) < TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_bad_gradient_stays_local(wct, synth, bad):
    half = 21
    cfg = synth.plane1_config(nticks=2000, nwire_half=half)
    rng = np.random.default_rng(6)
    d = _depos(synth, 200.0 + 500.0 * rng.random(80), -5000.0, 7)
    dt = wct.from_config(cfg)
    G = rng.random((NWIRES, 2000)).astype(np.float32)
    plain, _ = dt.adjoint(d, G)
    G[450, 700] = bad
    got, _ = dt.adjoint(d, G)
    w = d[:, 4] / 4.79 + 0.5 * (NWIRES - 1)
    out = np.abs(w - 450) > half + 4
    assert out.sum() > 40
    assert np.all(np.isfinite(got[out]))
    assert np.max(np.abs(got[out, 1] - plain[out, 1]) / np.abs(plain[out, 1])) < TOL
    assert not np.all(np.isfinite(got[~out]))
