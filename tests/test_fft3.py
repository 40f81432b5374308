"""The three-stage row transforms at every planned length: real rows through the
row convolution, complex rows through the IDFT, against numpy in float64, with
aligned and unaligned strides, odd row lengths and one to many rows a block.

Tolerance: a transform of M points is about 12 radix-2 levels of half an ulp
(6e-8) each, a convolution two of them: 6e-8 * sqrt(24) = 3e-7 in rel-L2, times
three."""

import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-6
HERE = os.path.dirname(os.path.abspath(__file__))


def _lengths():
    with open(os.path.join(HERE, "..", "wire-cell-toolkit_b200", "csrc", "fft3.cuh")) as f:
        text = f.read()
    text = text[text.index("#define WCT_FFT3_PLANS"):text.index("template <int R1_")]
    return sorted(int(a) * int(b) * int(c) for a, b, c in re.findall(r"X\((\d+), (\d+), (\d+)\)", text))


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("M", _lengths())
def test_real_rows(wct, M):
    import torch
    rng = np.random.default_rng(M)
    nfft = 2 * M
    for nrows, n_in, ld_in, n_out, ld_out in ((3, nfft - 40, nfft, nfft, nfft),
                                              (2, nfft // 2 + 1, nfft // 2 + 5, nfft - 1, nfft + 1),
                                              (1300, 37, 40, 101, 103)):
        k = rng.standard_normal(29)
        x = rng.standard_normal((nrows, n_in))
        d_x = torch.zeros((nrows, ld_in), dtype=torch.float32, device="cuda")
        d_x[:, :n_in] = torch.from_numpy(x)
        d_k = torch.from_numpy(k.astype(np.float32)).cuda()
        d_o = torch.full((nrows, ld_out), 7.0, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        wct.convolve_rows(d_x.data_ptr(), ld_in, nrows, n_in, d_k.data_ptr(), 29, d_o.data_ptr(), ld_out, n_out,
                          nfft=nfft)
        torch.cuda.synchronize()
        x32, k32 = x.astype(np.float32).astype(np.float64), k.astype(np.float32).astype(np.float64)
        ref = np.fft.irfft(np.fft.rfft(x32, nfft) * np.fft.rfft(k32, nfft), nfft)[:, :n_out]
        out = d_o.cpu().numpy()
        assert _rel(out[:, :n_out], ref) < TOL, (M, nrows)
        assert np.all(out[:, n_out:] == 7.0)


@pytest.mark.parametrize("M", _lengths())
@pytest.mark.parametrize("inverse", [False, True])
def test_complex_rows(wct, M, inverse):
    rng = np.random.default_rng(M + inverse)
    for nrows in (1, 1200):
        x = (rng.standard_normal((nrows, M)) + 1j * rng.standard_normal((nrows, M))).astype(np.complex64)
        y = (wct.IDFT().inv1b if inverse else wct.IDFT().fwd1b)(x, 1)
        ref = (np.fft.ifft if inverse else np.fft.fft)(x.astype(np.complex128), axis=1)
        assert _rel(y, ref) < TOL, (M, nrows)
