"""Tiles by their number of visits: up to 64 the block of the first launch takes
the tile, over that a larger block, and an event with many visits a tile goes
in one launch. Both sides of the line, full and partial chunks, against the
oracle, the same bits in any order of the depos, and batches (tolerance: the
frame's own, bin integrals 1.2e-7 and transforms 4e-7 in rel-L2, times four)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 2e-6


def _depos(synth, counts, seed):
    """Clusters on one wire and tick tile each, counts[k] depos in the k-th."""
    rng = np.random.default_rng(seed)
    d = np.zeros((sum(counts), 7))
    at = np.repeat(np.arange(len(counts)), counts)
    d[:, 0] = 100e3 + 256 * 500.0 * (at % 5) + rng.uniform(0, 5e3, len(d))
    d[:, 1] = -rng.uniform(100.0, 5000.0, len(d))
    d[:, 2] = synth.RESPONSE_X + 100.0
    d[:, 4] = 4.79 * 7 * (at - len(counts) // 2) + rng.uniform(-0.3, 0.3, len(d))
    d[:, 6] = rng.uniform(0.0, 0.3, len(d))
    return d


@pytest.mark.parametrize("counts", [(64,), (65, 1), (63, 64, 65), (128, 129, 255, 256, 257), (1, 700, 3, 4200),
                                    (3000,) * 20])
def test_against_oracle(wct, oracle, synth, counts):
    cfg = synth.plane1_config(nticks=2000)
    d = _depos(synth, counts, 5)
    dt = wct.from_config(cfg)
    frame, _, _ = dt(d)
    shuffled, _, _ = dt(d[np.random.default_rng(9).permutation(len(d))])
    assert np.array_equal(frame, shuffled)
    assert rel_l2(frame, oracle.run(cfg, d, fp64=True)["frames"][0]) < TOL
    batch, _, _ = wct.from_config(cfg).forward_batch([d[:1], d, d])
    assert np.array_equal(batch[1], batch[2])
    assert rel_l2(batch[1], frame) < TOL
