"""The double build's fixed-point tiles: accuracy against long double
transforms, and the tiles that IEEE arithmetic has to take over."""
import numpy as np
import pytest

import kfft_gb300 as K
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

# Every pass rounds its results to doubles once (2^-53 relative at most); the
# integers between hold 2^-60 or so, well inside one rounding's worth.
ULP = 2.0 ** -53


def rounds(lib, n):
    """Roundings to double on the way of an n-point transform, plus two."""
    p = lib._plan("kfft_config_cpx", n, 0)
    text = lib.describe(p)
    lib.cleanup(p)
    passes = text.count("R=")
    # a convolution: forward, inverse and the spectrum it multiplies by
    return 2 + (passes if " direct" in text.split("[")[0] else 3 * passes)


def signal(kind, n):
    rng = np.random.default_rng(n)
    z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    if kind == "delta":
        d = np.zeros(n, complex)
        d[n // 3] = 1 - 0.3j
        return d
    if kind == "range":  # magnitudes from 1e-12 to 1e12 side by side
        return z * 10.0 ** rng.uniform(-12, 12, n)
    return z


# every radix alone and in the first, middle and last place; every power of
# two of the compile-time tiles and the lengths that split; Rader, Bluestein
SIZES = list(range(2, 17)) + [32, 64, 128, 169, 256, 405, 512, 1024, 1155, 2048, 2187, 2197, 3328,
                              4095, 4096, 8192, 16384, 30030, 32768, 65536, 97, 257, 1009, 2879, 4099]


@pytest.mark.parametrize("kind", ["normal", "delta", "range"])
@pytest.mark.parametrize("n", SIZES)
def test_against_long_double(lib, n, kind):
    x = signal(kind, n)
    tol = rounds(lib, n) * ULP
    ref = np.fft.fft(x.astype(np.clongdouble))
    y = lib.fft_cpx(x)
    assert float(np.linalg.norm(y - ref) / np.linalg.norm(ref)) <= tol
    ref = np.fft.ifft(x.astype(np.clongdouble))
    y = lib.fft_cpx(x, K.FLAG_INVERSE)
    assert float(np.linalg.norm(y - ref) / np.linalg.norm(ref)) <= tol


@pytest.mark.parametrize("n", [5, 16, 45, 100, 512, 4096, 8192])
def test_batch_lanes_keep_their_own_scale(lib, n):
    """Sequences of very different magnitude side by side, zeros among them."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((37, n)) + 1j * rng.standard_normal((37, n))
    x *= 10.0 ** rng.uniform(-90, 90, (37, 1))
    x[5] = 0
    y = lib.fft_cpx(x)
    tol = rounds(lib, n) * ULP
    assert np.all(y[5] == 0)
    for b in range(37):
        if b != 5:
            ref = np.fft.fft(x[b].astype(np.clongdouble))
            assert float(np.linalg.norm(y[b] - ref) / np.linalg.norm(ref)) <= tol


@pytest.mark.parametrize("n", [12, 64, 1000, 4096, 32768])
@pytest.mark.parametrize("what", [np.inf, -np.inf, np.nan])
def test_non_finite_values_stay_in_their_sequence(lib, n, what):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((3, n)) + 1j * rng.standard_normal((3, n))
    clean = lib.fft_cpx(x)
    x[1, n // 2] = what
    y = lib.fft_cpx(x)
    for b in (0, 2):
        assert rel_l2(y[b], clean[b]) <= rounds(lib, n) * 4 * ULP
    assert not np.any(np.isfinite(y[1]))


# (216 .. 720: middle stages of several small butterflies a thread)
@pytest.mark.parametrize("n", [9, 64, 216, 250, 343, 360, 720, 1000, 4096, 32768])
@pytest.mark.parametrize("e", [-1040, -900, -765, 765, 900])
def test_ends_of_the_exponent_range(lib, n, e):
    """Scaled by a power of two the transform is the same one, scaled."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((23, n)) + 1j * rng.standard_normal((23, n))
    got = lib.fft_cpx(x * 2.0 ** (e // 2) * 2.0 ** (e - e // 2))
    ref = lib.fft_cpx(x)
    # below 2^-1022 the inputs themselves lose bits
    lost = 2.0 ** (-1074 - e) * 4 if e < -1000 else 0.0
    assert rel_l2(got * 2.0 ** (-e // 2) * 2.0 ** (-e - (-e // 2)), ref) <= 1e-15 + lost


def test_queue_tiles(lib):
    """The queue kernel's tiles: every power of two it runs in one tile, and
    lengths whose stages take one round of its threads or more."""
    lengths = np.array([16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 1 << 17, 11, 1792, 1820, 1848,
                        1960, 2016, 2028, 2047, 1890, 1331, 2197, 30030, 4099, 65537, 9973, 504 * 488, 2016 * 45], np.uint32)
    rng = np.random.default_rng(3)
    x = rng.standard_normal(int(lengths.sum())) + 1j * rng.standard_normal(int(lengths.sum()))
    for flags, f in ((0, np.fft.fft), (K.FLAG_INVERSE, np.fft.ifft)):
        p = lib.L.kfft_config_cpx_uneven(len(lengths), lengths.ctypes.data, flags)
        assert p, lib.last_error()
        y = np.empty_like(x)
        r = lib.L.kfft_eval_cpx_uneven(p, x.ctypes.data, y.ctypes.data)
        lib.L.kfft_release_uneven(p)
        assert r == 0, lib.last_error()
        at = 0
        for n in lengths.tolist():
            ref = f(x[at:at + n].astype(np.clongdouble))
            # at most four passes a transform in the queue, and a convolution has three
            assert float(np.linalg.norm(y[at:at + n] - ref) / np.linalg.norm(ref)) <= 14 * ULP, n
            at += n
