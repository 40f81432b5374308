"""The random streams' uniforms lie in (0, 1], and the noise normals are finite
and right up to the ends of that interval (CPU only: csrc/rng.cuh
compiled for the host).

Tolerance: 1e-10 of the chain, the rounding of the result to float (2^-24), and
the start of the root, which a Newton step squares: (2^-23)^2."""

import math
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "wire-cell-toolkit_b200", "csrc")
TOP = 0xFFFFFFFF


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    inc = next((d for d in (os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include",)
                if os.path.exists(os.path.join(d, "cuda_runtime.h"))), None)
    if shutil.which("g++") is None or inc is None:
        pytest.skip("g++ or the CUDA headers not available")
    out = str(tmp_path_factory.mktemp("rng") / "host_rng")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", CSRC, "-isystem", inc,
                        os.path.join(ROOT, "tests", "host_rng.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def _run(exe, words):
    text = "\n".join("%x %x %x %x" % tuple(w) for w in words)
    r = subprocess.run([exe], input=text, capture_output=True, text=True, check=True)
    return np.array([[float(v) for v in line.split()] for line in r.stdout.splitlines()])


def _words(x):
    """(hi, lo) of the 53-bit number x."""
    return x >> 21, (x & 0x1FFFFF) << 11


ENDS = [0, 1, 2, 1 << 26, (1 << 52) - 1, 1 << 52, (1 << 52) + 1, (1 << 53) - 3, (1 << 53) - 2, (1 << 53) - 1]


def test_uniforms(exe):
    words = [_words(x) + _words(y) for x in ENDS for y in ENDS]
    words += [(TOP, TOP, 0, 0), (TOP, 0xFFFFF800, TOP, 0xFFFFF7FF), (TOP - 1, TOP, TOP, 0x7FF)]
    o = _run(exe, words)
    assert np.all((o[:, :2] > 0.0) & (o[:, :2] <= 1.0))
    # (x + 1/2) 2^-53, rounded: the largest word's is 1
    for w, u in zip(words, o):
        for hi, lo, v in ((w[0], w[1], u[0]), (w[2], w[3], u[1])):
            x = ((hi << 32) | lo) >> 11
            assert v == (float(x) + 0.5) * 2.0 ** -53


def test_normals_at_the_ends(exe):
    rng = np.random.default_rng(3)
    rand = [tuple(int(v) for v in rng.integers(0, 1 << 32, 4)) for _ in range(2000)]
    words = [_words(x) + _words(y) for x in ENDS for y in ENDS] + rand
    for u1, u2, z in _run(exe, words):
        r = math.sqrt(abs(2.0 * math.log(u1)))
        assert math.isfinite(z)
        assert abs(z - r * math.cos(2.0 * math.pi * u2)) <= r * (1e-10 + 2.0 ** -24 + 2.0 ** -45)
