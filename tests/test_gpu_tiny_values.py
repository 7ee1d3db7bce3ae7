"""Double build: values far below a sequence's largest, down to the smallest
double, are cut off like any other small value; only a lane whose largest value
is that small leaves the fixed-point tiles."""
import math

import numpy as np
import pytest

import kfft_gb300 as K

pytestmark = pytest.mark.gpu

# compile-time and run-time tiles, one and more passes, Rader, Bluestein
SIZES = [3, 5, 8, 16, 45, 64, 100, 512, 1000, 4096, 8192, 59049, 257, 4099]


def noise(n, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(n) + 1j * rng.standard_normal(n)


@pytest.mark.parametrize("tiny", [2.0 ** -768, 1e-300, 5e-324])
@pytest.mark.parametrize("n", SIZES)
def test_tiny_values_among_ordinary_ones(lib, n, tiny):
    """They change nothing: the outputs are those of zeros in their place."""
    x = np.stack([noise(n, n + i) for i in range(5)])
    at = np.random.default_rng(n).random(x.shape) < 0.25
    at[:, n // 2] = False
    x[at] = 0
    zeros = lib.fft_cpx(x)
    x[at] = tiny * (1 - 1j)
    assert np.array_equal(lib.fft_cpx(x), zeros)
    back = lib.fft_cpx(x, K.FLAG_INVERSE)
    x[at] = 0
    assert np.array_equal(back, lib.fft_cpx(x, K.FLAG_INVERSE))


@pytest.mark.parametrize("sigma", [3.0, 40.0])
@pytest.mark.parametrize("n", [1000, 4096, 8192, 59049])
def test_gaussian(lib, n, sigma):
    """A tabulated Gaussian, whose tail runs through the smallest doubles."""
    i = np.arange(n) - n // 2
    x = np.exp(-(i / sigma) ** 2 / 2) + 0j
    ref = np.fft.fft(x.astype(np.clongdouble))
    y = lib.fft_cpx(np.stack([x, noise(n, 1), x]))
    tol = (3 * math.log2(n) + 4) * 2.0 ** -53
    for r in (0, 2):
        assert float(np.linalg.norm(y[r] - ref) / np.linalg.norm(ref)) <= tol


@pytest.mark.parametrize("n", SIZES)
def test_tiny_sequences_among_ordinary_ones(lib, n):
    """Sequences that are tiny as a whole keep their bits (scaled by a power of
    two the transform is the same one, scaled)."""
    x = np.stack([noise(n, n + i) for i in range(7)])
    ref = lib.fft_cpx(x)
    x[2] *= 2.0 ** -900
    x[5] *= 2.0 ** -800
    y = lib.fft_cpx(x)
    for r, s in ((2, 900), (5, 800)):
        got = y[r] * 2.0 ** (s // 2) * 2.0 ** (s - s // 2)
        assert np.linalg.norm(got - ref[r]) <= 2 * 3 * (3 * math.log2(n) + 4) * 2.0 ** -53 * np.linalg.norm(ref[r])


def test_queue(lib):
    lengths = np.array([16, 45, 64, 100, 512, 1000, 2048, 4096, 8192, 30030, 257, 4099], np.uint32)
    x = noise(int(lengths.sum()), 1)
    at = np.random.default_rng(2).random(x.size) < 0.25

    def run(v):
        y = np.empty_like(v)
        p = lib.L.kfft_config_cpx_uneven(len(lengths), lengths.ctypes.data, K.FLAG_NORMAL)
        assert p, lib.last_error()
        r = lib.L.kfft_eval_cpx_uneven(p, v.ctypes.data, y.ctypes.data)
        lib.L.kfft_release_uneven(p)
        assert r == 0, lib.last_error()
        return y

    x[at] = 0
    zeros = run(x)
    x[at] = 1e-300
    assert np.array_equal(run(x), zeros)
