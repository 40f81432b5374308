"""Charge grids with most tiles empty: the row transform reads no tile without
visits and the raster leaves those unwritten, so a workspace full of an
earlier event's charge must not show. First ticks of every remainder by four
(a 16-byte piece may span two tiles), tiles at both ends of the readout, one
depo, a whole-window spread, one event and batches, fixed and fluctuated
charges. The same bits as from a component that has held nothing before, and
the oracle's frame (tolerance: the frame's own, bin integrals 1.2e-7 and
transforms 4e-7 in rel-L2, times four)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 2e-6


def _depos(synth, t, z, ext=1.0, seed=1):
    rng = np.random.default_rng(seed)
    d = np.zeros((len(t), 7))
    d[:, 0] = t
    d[:, 1] = -rng.uniform(1000.0, 5000.0, len(t))
    d[:, 2] = synth.RESPONSE_X + 100.0
    d[:, 4] = z
    d[:, 5] = rng.uniform(0.0, ext, len(t))
    d[:, 6] = rng.uniform(0.0, 2.4, len(t))
    return d


def _full(synth, nticks):
    rng = np.random.default_rng(3)
    return _depos(synth, rng.uniform(0, (nticks - 300) * 500.0, 30000), rng.uniform(-2300, 2300, 30000))


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("case", ["one", "far apart", "diagonal", "readout ends"])
def test_against_oracle(wct, oracle, synth, case, shift):
    nticks = 3000
    cfg = synth.plane1_config(nticks=nticks)
    t0 = shift * 500.0
    rng = np.random.default_rng(7)
    if case == "one":
        d = _depos(synth, [400e3 + t0], [10.0])
    elif case == "far apart":
        d = _depos(synth, np.array([100e3, 600e3, 1300e3]) + t0, [-900.0, 0.0, 900.0], ext=8.0)
    elif case == "diagonal":
        u = np.linspace(0.0, 1.0, 400)
        d = _depos(synth, 50e3 + t0 + 1200e3 * u, -1500.0 + 3000.0 * u)
    else:
        d = _depos(synth, np.where(rng.random(40) < 0.5, -62e3, 1437e3) + t0, rng.uniform(-1000, 1000, 40), ext=8.0)
    dt = wct.from_config(cfg)
    full = _full(synth, nticks)
    dt(full)  # the workspace is full of charge
    frame, _, _ = dt(d)
    assert np.array_equal(frame, wct.from_config(cfg)(d)[0])
    assert rel_l2(frame, oracle.run(cfg, d, fp64=True)["frames"][0]) < TOL
    bt = wct.from_config(cfg)
    bt.forward_batch([full, full, full])
    batch, _, _ = bt.forward_batch([d, full, d])
    assert np.array_equal(batch[0], batch[2])
    assert rel_l2(batch[0], frame) < TOL


def test_fluctuated_charges(wct, synth):
    cfg = synth.plane1_config(nticks=3000)
    cfg["fluctuate"] = True
    u = np.linspace(0.0, 1.0, 300)
    d = _depos(synth, 50e3 + 1200e3 * u, -1500.0 + 3000.0 * u)
    full = _full(synth, 3000)
    used, fresh = wct.from_config(cfg), wct.from_config(cfg)
    used(full)
    fresh(d[:1])  # the random streams are keyed by the frame's ident
    assert np.array_equal(used(d)[0], fresh(d)[0])
