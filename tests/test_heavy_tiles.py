"""Raster tiles worked off in parts: long patches (over 16 ticks) in one part and
in several, more visits of short patches than a tile takes at once, both in one
tile, fewer impact groups than the usual eleven, patches cut by the
readout; against the oracle, and the same bits from run to run.

Tolerance: the grid's fixed point adds under 1e-8; the frame's own (bin
integrals 1.2e-7, transforms 4e-7 in rel-L2) times four."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 2e-6


def _blob(synth, n, seed, radius, ext, x=900.0, z=0.0, t0=0.0):
    rng = np.random.default_rng(seed)
    d = np.zeros((n, 7))
    d[:, 0] = t0
    d[:, 1] = -rng.uniform(100.0, 5000.0, n)
    d[:, 2] = x + rng.normal(0.0, radius, n)
    d[:, 4] = z + rng.normal(0.0, radius, n)
    d[:, 5] = rng.uniform(0.0, ext, n)
    d[:, 6] = rng.uniform(0.0, 2.4, n)
    return d


CASES = {
    "one part": lambda s: _blob(s, 60, 1, 5.0, 26.0),
    "parts of long patches": lambda s: _blob(s, 2500, 2, 15.0, 26.0),
    "a full part": lambda s: _blob(s, 256, 3, 0.5, 26.0),
    "short patches on one wire": lambda s: _blob(s, 9000, 4, 0.4, 0.0),
    "short and long": lambda s: np.concatenate([_blob(s, 5000, 5, 0.5, 0.0), _blob(s, 700, 6, 3.0, 26.0)]),
    "cut by the readout": lambda s: np.concatenate([_blob(s, 800, 7, 5.0, 26.0, t0=-490e3),
                                                    _blob(s, 800, 8, 5.0, 26.0, t0=990e3)]),
}


@pytest.mark.parametrize("name", CASES)
def test_against_oracle(wct, oracle, synth, name):
    cfg = synth.plane1_config(nticks=3000)
    d = CASES[name](synth)
    dt = wct.from_config(cfg)
    frame, _, _ = dt(d)
    again, _, _ = dt(d)
    assert np.array_equal(frame, again)
    shuffled, _, _ = dt(d[np.random.default_rng(9).permutation(len(d))])
    assert np.array_equal(frame, shuffled)  # integer sums: the order of the depos does not matter
    assert rel_l2(frame, oracle.run(cfg, d, fp64=True)["frames"][0]) < TOL
    batch, _, _ = wct.from_config(cfg).forward_batch([d, d[:50]])
    assert rel_l2(batch[0], frame) < TOL


@pytest.mark.parametrize("nimp", [2, 4])
def test_few_impact_groups(wct, synth, nimp):
    """3 and 5 groups of the 12 that a part holds: the frame stays additive."""
    pitch = 4.79
    dt = wct.DepoTransform(dict(tick=500.0, start_time=0.0, readout_time=2000 * 500.0, drift_speed=1.6e-3))
    f = dt.add_face()
    pl = dict(synth.plane1_config(nticks=2000)["planes"][0], nimp=nimp)
    dt.add_plane(f, pl)
    rng = np.random.default_rng(2)
    dt.set_response_table(f, 0, rng.random((nimp + 1, 7, 60)), pitch, pitch / nimp, 100)
    a, b = (_blob(synth, 600, k, 10.0, 26.0, t0=300e3) for k in (1, 2))
    frames = [dt(d)[0].astype(np.float64) for d in (a, b, np.concatenate([a, b]))]
    assert rel_l2(frames[2], frames[0] + frames[1]) < TOL
