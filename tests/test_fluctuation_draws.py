"""The sampler's single-precision decisions give the double-precision draws, and
patches whose draws found no room are drawn again with the same result.

The restatement below is inversion / BTRS in Python floats on the same Philox
streams; draws are whole numbers and compared exactly."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MASK = 0xFFFFFFFF
TAG = 0xFFFE


def _block(k0, k1, c):
    x0, x1, x2, x3 = c
    for _ in range(10):
        a, b = 0xD2511F53 * x0, 0xCD9E8D57 * x2
        x0, x1, x2, x3 = (b >> 32) ^ x1 ^ k0, b & MASK, (a >> 32) ^ x3 ^ k1, a & MASK
        k0, k1 = (k0 + 0x9E3779B9) & MASK, (k1 + 0xBB67AE85) & MASK
    return x0, x1, x2, x3


def _uniforms(k0, k1, i):
    block = 0
    while True:
        o = _block(k0, k1, (i, TAG, 0, block))
        for hi, lo in ((o[0], o[1]), (o[2], o[3])):
            yield ((((hi << 32) | lo) >> 11) + 0.5) * 2.0 ** -53
        block += 1


def _fc(x):
    if x < 10:
        return (0.08106146679532733, 0.041340695955409457, 0.027677925684997717, 0.020790672103765839,
                0.016644691189821259, 0.013876128823072875, 0.011896709945893313, 0.010411265261973668,
                0.0092554621827094508, 0.0083305634333594725)[x]
    r = 1.0 / (x + 1.0)
    return r * (1 / 12.0 - r * r * (1 / 360.0 - r * r * (1 / 1260.0)))


def _lf(x):
    return (x + 0.5) * math.log(x + 1.0) + _fc(x)


def _draw(n, p, us):
    if p > 0.5:
        return n - _draw(n, 1.0 - p, us)
    q, np_ = 1.0 - p, n * p
    if np_ < 10.0:
        u, x, f = next(us), 0, math.exp(n * math.log1p(-p))
        while u > f and x < n:
            u -= f
            f *= p / q * (n - x) / (x + 1)
            x += 1
        return x
    spq = math.sqrt(np_ * q)
    b = 1.15 + 2.53 * spq
    a = -0.0873 + 0.0248 * b + 0.01 * p
    m = math.floor((n + 1) * p)
    while True:
        u, v = next(us) - 0.5, next(us)
        r = 0.5 - abs(u)
        k = math.floor((2.0 * a / r + b) * u + np_ + 0.5)
        if k < 0 or k > n:
            continue
        if r >= 0.07 and v <= 0.92 - 4.2 / b:
            return k
        lv = math.log(v * (2.83 + 5.1 / b) * spq / (a / (r * r) + b))
        if lv <= _lf(m) + _lf(n - m) - _lf(k) - _lf(n - k) + (k - m) * math.log(p / q):
            return k


@pytest.mark.parametrize("n,p", [(1, 0.3), (3, 0.5), (7, 0.999), (620, 1e-4), (620, 0.016), (3100, 0.0033), (3100, 0.05),
                                 (25, 0.45), (20, 0.5), (5000, 0.31), (5000, 0.77), (200000, 0.003), (20000000, 0.1)])
def test_draws_equal_double_precision(wct, n, p):
    import torch
    count, seed, ident = 6000, 987654321012345, 5
    out = torch.zeros(count, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    wct.binomial_device(seed, ident, n, p, count, out.data_ptr())
    torch.cuda.synchronize()
    k0, k1 = seed & MASK, ((seed >> 32) + 0x9E3779B9 * ident) & MASK
    ref = np.array([_draw(n, p, _uniforms(k0, k1, i)) for i in range(count)])
    assert np.array_equal(out.cpu().numpy(), ref)


def test_patches_without_room_are_redrawn(wct, synth):
    """A batch of wide patches (about 3000 cells) exceeds the room of the first
    call; its frames are the per-event frames then and with more room."""
    cfg = synth.plane1_config(nticks=3000)
    cfg["fluctuate"], cfg["seed"] = True, 11
    rng = np.random.default_rng(4)
    events = [synth.shower_depos(rng, 300, center=np.array([900.0, 0.0, 100.0 * k]), ext_long_max=26.0)
              for k in range(3)]
    batch = wct.from_config(cfg)
    first, _, _ = batch.forward_batch(events)
    again = wct.from_config(cfg)
    for _ in range(2):
        more, _, ident = again.forward_batch(events)
        if ident == 0:
            assert np.array_equal(more, first)
    single = wct.from_config(cfg)
    for e, d in enumerate(events):
        f, _, _ = single(d)
        assert np.linalg.norm(f - first[e]) < 2e-6 * np.linalg.norm(f)
