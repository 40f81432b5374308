"""The forms of the wire convolution that an event chooses by its rows and visits:
blocks with their faint rows listed, or every row listed; rows one by one against
the 64-bit oracle, on either side of each line (few wires, few visits a row, few
taps).

Tolerance, per row: the row transforms and the convolution's sums, 6e-8 a
butterfly stage over about 25 stages, plus the blocks' rounding of at most twice
1.5e-7 where a row keeps it; times three."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-6
NWIRES = 960
BLOCKS, LISTED, DIRECT = 3, 2, 1  # launches: the blocks, the pick and the rows; without the blocks


def _event(synth, lo, span, n, depth, seed=0):
    """n depos over span wires from lo on, and a group 1e4 times brighter."""
    rng = np.random.default_rng(seed)
    w = np.concatenate([[lo, lo + span], lo + span * rng.random(n - 4), [lo + 0.3 * span, lo + 0.3 * span + 0.7]])
    d = np.zeros((n, 7))
    d[:, 1] = -5000.0 * (0.5 + rng.random(n))
    d[-2:, 1] = -5e7
    d[:, 2] = synth.RESPONSE_X + 200.0 + depth * rng.random(n)
    d[:, 4] = (w - 0.5 * (NWIRES - 1)) * 4.79
    return d


@pytest.mark.parametrize("half,span,n,form", [
    (21, 90, 1500, DIRECT), (21, 160, 1500, DIRECT), (21, 250, 3000, BLOCKS),  # resident blocks
    (21, 700, 3000, BLOCKS), (21, 700, 60, DIRECT),                            # visits a row
    (40, 300, 2000, BLOCKS), (40, 300, 20, LISTED),
    (30, 216, 1500, BLOCKS), (30, 160, 1500, LISTED),  # 256 output rows
    (64, 100, 1500, LISTED),
    (6, 300, 2000, BLOCKS), (5, 300, 2000, LISTED), (2, 700, 2000, LISTED), (2, 30, 8, LISTED)])
def test_rows_against_oracle(wct, oracle, synth, half, span, n, form):
    # long windows for the direct kernel of its own, so that not all of its blocks are resident
    nticks, depth = (6000, 2200.0) if half == 21 else (2000, 300.0)
    cfg = synth.plane1_config(nticks=nticks, nwire_half=half)
    d = _event(synth, 120.3, span, n, depth)
    o, faint, bright = (oracle.run(cfg, part, fp64=True)["frames"][0].astype(np.float64)
                        for part in (d, d[:-2], d[-2:]))
    dt = wct.from_config(cfg)
    dt.set_profiling(True)
    frame, wins, _ = dt(d)
    assert dt.stage_times()[0]["wire_conv"][1] == form, wins[0]["charge_rows"]
    wires = d[:, 4] / 4.79 + 0.5 * (NWIRES - 1)
    norm = np.linalg.norm(o, axis=1)
    near = np.min(np.abs(np.arange(NWIRES)[:, None] - wires[None, :]), axis=1) <= half
    # where the 64-bit transforms' own rounding is below it: 1e-16 of the bright rows lies in every row, and the
    # response falls to 2e-8 of its peak at 40 wires, 1e-13 at 64
    sure = np.linalg.norm(o - faint - bright, axis=1) < 0.05 * TOL * norm
    rows = np.nonzero((norm > 0) & near & sure)[0]
    assert len(rows) > min(span, NWIRES - 121) // 2
    err = np.linalg.norm(frame[rows].astype(np.float64) - o[rows], axis=1) / norm[rows]
    assert np.max(err) < TOL, rows[np.argmax(err)]
    live = np.nonzero(np.any(frame != 0, axis=1))[0]  # a patch spans a wire or two around its depo
    assert live.min() >= wires.min() - half - 4 and live.max() <= wires.max() + half + 4


def test_windows_whose_spectra_do_not_fit(wct, oracle, synth):
    """A window of 12000 ticks: no wire spectra are kept, every row is listed at a pad without a direct kernel."""
    cfg = synth.plane1_config(nticks=11950, nwire_half=16)
    cfg["pir_nticks"] = 2000
    d = _event(synth, 120.3, 260, 1200, 300.0)[:-2]
    d[:, 0] += 500.0 * 11500 * np.random.default_rng(1).random(len(d))
    o = oracle.run(cfg, d, fp64=True)["frames"][0].astype(np.float64)
    dt = wct.from_config(cfg)
    dt.set_profiling(True)
    frame, wins, _ = dt(d)
    assert wins[0]["nt_gpu"] == 12000 and dt.stage_times()[0]["wire_conv"][1] == LISTED
    norm = np.linalg.norm(o, axis=1)
    rows = np.nonzero(norm > 1e-6 * norm.max())[0]
    err = np.linalg.norm(frame[rows].astype(np.float64) - o[rows], axis=1) / norm[rows]
    assert len(rows) > 260 and np.max(err) < TOL


@pytest.mark.parametrize("half", [21, 10, 16])
def test_direct_sums_add_the_groups_apart(wct, oracle, synth, half):
    """A frame of directly convolved rows is as close to 64 bits as the row transforms leave it.

    Roundings of 6e-8 * 0.29 (rms) each: about 60 in the two transforms' butterflies (1.4e-7), 43 taps a group in sums
    of a sixth of the total added in quadrature with six group sums (0.7e-7), the bins' integrals and the charge grid
    (0.5e-7): 1.65e-7, times 1.5.  One sum over all groups adds 2.8e-7."""
    cfg = synth.plane1_config(nticks=6000, nwire_half=half)
    d = synth.plane1_depos(n=300, seed=1)
    o = oracle.run(cfg, d, fp64=True)["frames"][0].astype(np.float64)
    dt = wct.from_config(cfg)
    dt.set_profiling(True)
    frame, _, _ = dt(d)
    assert dt.stage_times()[0]["wire_conv"][1] < BLOCKS
    assert np.linalg.norm(frame - o) < 2.5e-7 * np.linalg.norm(o)
