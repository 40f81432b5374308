"""Fluctuated patches whose draws found no room in a batch are drawn again in the
raster: the same numbers as stored ones, so the same frames bit for bit.

The room of a first call is 160 cells a plane and depo; a call that was short
doubles it for the next.  Components that start at frame f draw the streams of
frame f, so a component's later calls and another's first one can be compared."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _events(synth, n=300, nev=3):
    rng = np.random.default_rng(4)
    return [synth.shower_depos(rng, n, center=np.array([900.0, 0.0, 100.0 * k]), ext_long_max=26.0)
            for k in range(nev)]


def _cells(wct, cfg, events):
    """Patch cells of the events, from the records of single calls."""
    total = 0
    dt = wct.from_config(cfg)
    for d in events:
        dt(d)
        r = dt.patch_records(0, 0, len(d)).astype(np.int64)
        total += int(np.sum(r[:, 2] * r[:, 3]))
    return total


def test_redrawn_patches_equal_stored_ones(wct, synth):
    events = _events(synth)
    cfg = synth.plane1_config(nticks=3000)
    cfg["fluctuate"], cfg["seed"] = True, 11
    ndepos = sum(len(d) for d in events)
    cells = _cells(wct, cfg, events)
    assert cells > 4 * 160 * ndepos  # two calls at least are short of room
    long = wct.from_config(cfg)
    for call in range(8):
        frames, _, ident = long.forward_batch(events)
        assert ident == 3 * call
        # the same frame numbers with the room of a first call
        c = dict(cfg, first_frame_number=ident)
        short, _, ident0 = wct.from_config(c).forward_batch(events)
        assert ident0 == ident
        assert np.array_equal(frames, short), call
    assert 160 * 2 ** 7 * ndepos > cells  # the last calls stored every draw
