"""The wire-direction convolution by blocks of 256 wires: window widths on
either side of one and two blocks, pads with and without a direct kernel, the
widest pad it takes and one beyond, the rows that no charge reaches, and the
adjoint as the transpose.

Tolerance: the two transforms of about 12 + 8 butterfly stages each add half
an ulp a stage, 6e-8 * sqrt(40) = 4e-7 in rel-L2 beside the bin integrals'
1.2e-7; times four."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 2e-6
PITCH = 4.79
NWIRES = 960


def _depos(synth, wires, seed):
    """Point depos at given (fractional) wires, near the response plane."""
    rng = np.random.default_rng(seed)
    w = np.asarray(wires, dtype=np.float64)
    d = np.zeros((len(w), 7))
    d[:, 1] = -5000.0 * (0.5 + rng.random(len(w)))
    d[:, 2] = synth.RESPONSE_X + 200.0 + 300.0 * rng.random(len(w))
    d[:, 4] = (w - 0.5 * (NWIRES - 1)) * PITCH
    return d


def _spans(half):
    """Window spans (wires) at the smallest, about one block, and two blocks."""
    valid = 256 - 2 * half if half <= 64 else 120
    return [0, max(2, valid - 2 * half - 4), max(4, valid - 2 * half), valid - 4, valid, 2 * valid - 2 * half]


@pytest.mark.parametrize("half", [1, 3, 10, 21, 64, 66])
def test_blocks_against_oracle(wct, oracle, synth, half):
    cfg = synth.plane1_config(nticks=2000, nwire_half=half)
    dt = wct.from_config(cfg)
    rng = np.random.default_rng(half)
    for k, span in enumerate(_spans(half)):
        lo = 100.0 + 0.31 * k
        d = _depos(synth, np.concatenate([[lo, lo + span], lo + span * rng.random(30)]), seed=k)
        frame, wins, _ = dt(d)
        o = oracle.run(cfg, d, fp64=True)
        assert wins[0]["start_ch"] == o["windows"][0]["start_ch"]
        assert rel_l2(frame, o["frames"][0]) < TOL, (half, span)


@pytest.mark.parametrize("half", [10, 21])
def test_rows_out_of_reach_are_zero(wct, synth, half):
    cfg = synth.plane1_config(nticks=2000, nwire_half=half)
    d = _depos(synth, [200.2, 201.4, 430.1, 431.9, 433.3], seed=2)
    frame, _, _ = wct.from_config(cfg)(d)
    live = np.nonzero(np.any(frame != 0, axis=1))[0]
    # a depo's patch spans a few wires around it (3 sigma of diffusion over half a metre, under 2 pitches)
    near = np.zeros(NWIRES, dtype=bool)
    for w in (200, 202, 430, 432, 433):
        near[max(0, w - half - 4):w + half + 5] = True
    assert len(live) and not np.any(~near[live])


@pytest.mark.parametrize("half,span", [(21, 0), (21, 170), (21, 214), (21, 600), (40, 300), (10, 300)])
def test_adjoint_is_the_transpose(wct, synth, half, span):
    """The frame is linear in the charges: <G, F(q)> = sum_i q_i dL/dq_i."""
    cfg = synth.plane1_config(nticks=2000, nwire_half=half)
    dt = wct.from_config(cfg)
    rng = np.random.default_rng(span)
    d = _depos(synth, np.concatenate([[150.0, 150.0 + span], 150.0 + span * rng.random(40)]), seed=span)
    frame, _, _ = dt(d)
    # positive weights and one charge sign on a unipolar response: no cancellation in the products
    G = rng.random(frame.shape).astype(np.float32)
    gd, _ = dt.adjoint(d, G)
    lhs = float(np.sum(G.astype(np.float64) * frame))
    assert abs(float(np.sum(d[:, 1] * gd[:, 1])) - lhs) < TOL * abs(lhs)
