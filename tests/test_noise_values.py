"""Noise waveforms value by value: the streams' normals and the transform
restated in float64, at lengths with and without a three-stage transform, rows
shorter and longer than the spectrum, aligned and not, some without a spectrum.

Tolerance: rel-L2 of the added waveform; single-precision transform 6e-8 *
sqrt(24) = 3e-7 and the rounding of the sums, times three."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-6
MASK = np.uint64(0xFFFFFFFF)


def _normals(key0, key1, stream, model, index):
    c = [np.full(index.shape, stream, np.uint64), np.full(index.shape, model, np.uint64), index.astype(np.uint64),
         np.zeros(index.shape, np.uint64)]
    k0, k1 = key0, key1
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        s = np.uint64(32)
        c = [(b >> s) ^ c[1] ^ np.uint64(k0), b & MASK, (a >> s) ^ c[3] ^ np.uint64(k1), a & MASK]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = [(((hi << np.uint64(32)) | lo) >> np.uint64(11)).astype(np.float64) for hi, lo in ((c[0], c[1]), (c[2], c[3]))]
    u = [(v + 0.5) * 2.0 ** -53 for v in u]
    return np.sqrt(-2.0 * np.log(u[0])) * np.cos(2.0 * np.pi * u[1])


@pytest.mark.parametrize("N,ncols,pad", [
    (512, 512, 0), (800, 800, 0), (3200, 3200, 0), (6000, 6000, 0), (8192, 8192, 0), (12000, 12000, 0),
    (1000, 1000, 0), (3240, 3240, 0),          # halves 500 and 1620: no three-stage transform
    (3200, 3001, 0), (3200, 3500, 4), (6000, 5999, 3), (4096, 4096, 1),
])
def test_waveforms(wct, N, ncols, pad):
    import torch
    rng = np.random.default_rng(N + ncols)
    rows, seed, ident, model = 37, 77, 3, 2
    spectra = (rng.random((3, N)) + 0.1).astype(np.float32)
    spec = rng.integers(-1, 3, rows).astype(np.int32)
    stream = rng.integers(0, 5000, rows).astype(np.int32)
    base = rng.standard_normal((rows, ncols + pad)).astype(np.float32)
    d = [torch.from_numpy(v.copy()).cuda() for v in (base, spectra, spec, stream)]
    torch.cuda.synchronize()
    wct.add_noise_device(d[0].data_ptr(), ncols + pad, rows, ncols, d[1].data_ptr(), N, d[2].data_ptr(),
                         d[3].data_ptr(), seed=seed, ident=ident, model=model)
    torch.cuda.synchronize()
    out = d[0].cpu().numpy()
    h, n = N // 2, min(N, ncols)
    key1 = (0x9E3779B9 * ident) & 0xFFFFFFFF
    for r in range(rows):
        want = np.zeros(ncols)
        if spec[r] >= 0:
            z = _normals(seed, key1, int(stream[r]), model, np.arange(N + 1))
            m = spectra[spec[r]].astype(np.float64)[:h + 1] * np.sqrt(2.0 / 3.141592)
            X = m * z[:h + 1] + 1j * m * z[h:]
            X[0], X[h] = abs(X[0]), abs(X[h])
            want[:n] = np.fft.irfft(X, N)[:n]
        got = out[r, :ncols].astype(np.float64) - base[r, :ncols]
        # what is left of the frame's own rounding: half an ulp of values up to about 5
        assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want) + 3e-7 * np.sqrt(ncols), r
        assert np.array_equal(out[r, ncols:], base[r, ncols:])
