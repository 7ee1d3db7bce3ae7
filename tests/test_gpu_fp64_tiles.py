"""Double build: the FP64 tiles that take over from the fixed-point ones, in
every layout and with every prologue and epilogue: both directions, columns,
real transforms, convolutions, Rader and Bluestein."""
import math

import numpy as np
import pytest

import kfft_gb300 as K

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -53
# compile-time tiles of every length, run-time ones of every first radix, several passes
SIZES = [16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 8192, 32768, 65536, 1 << 18,
         3, 5, 6, 7, 9, 10, 11, 12, 13, 14, 15, 45, 100, 1000, 4000, 59049, 257, 12289, 4099]
DOWN = 900  # 2^-900: every lane is too small for the fixed-point tiles


def noise(shape, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def scaled(x, e):
    return x * 2.0 ** (e // 2) * 2.0 ** (e - e // 2)


def close(got, ref, n, transforms=1):
    """Two results with the rounding errors of as many transforms of n points each."""
    tol = 2 * transforms * (3 * math.log2(n) + 4) * ULP
    return np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("flags", [K.FLAG_NORMAL, K.FLAG_INVERSE, K.FLAG_INVERSE | K.FLAG_DISABLE_NORM])
@pytest.mark.parametrize("n", SIZES)
def test_small_sequences(lib, n, flags):
    x = noise((3, n), n)
    assert close(scaled(lib.fft_cpx(scaled(x, -DOWN), flags), DOWN), lib.fft_cpx(x, flags), n, 3)


@pytest.mark.parametrize("n", SIZES)
def test_nearly_real_both_ways(lib, n):
    x = noise((3, n), n)
    x.imag *= 2.0 ** -30
    y = lib.fft_cpx(x)
    assert close(y, np.fft.fft(x.astype(np.clongdouble), axis=1).astype(complex), n, 3)
    z = lib.fft_cpx(x, K.FLAG_INVERSE)
    assert close(z, np.fft.ifft(x.astype(np.clongdouble), axis=1).astype(complex), n, 3)
    # bin 0 keeps the small parts by themselves (Bluestein's chirp turns every
    # value, so there it does not, in doubles either)
    p = lib._plan("kfft_config_cpx", n, K.FLAG_NORMAL)
    mixed = "bluestein" in lib.describe(p)
    lib.cleanup(p)
    for i in range(0 if mixed else 3):
        tol = 3 * (3 * math.log2(n) + 4) * ULP * np.abs(x[i].imag).sum()
        assert abs(y[i, 0].imag - math.fsum(x[i].imag)) <= tol
        assert abs(z[i, 0].imag * n - math.fsum(x[i].imag)) <= tol


# columns in tiles of 16 lanes and more, with a partly filled last one
@pytest.mark.parametrize("y,x", [(16, 100), (64, 77), (512, 33), (4096, 18), (8192, 17), (45, 100), (1000, 21), (6, 300)])
def test_columns(lib, y, x):
    a = noise((y, x), x)
    for flags in (K.FLAG_NORMAL, K.FLAG_INVERSE):
        got = scaled(lib.fft2_cpx(scaled(a, -DOWN), flags), DOWN)
        assert close(got, lib.fft2_cpx(a, flags), x * y, 2)
    a.imag *= 2.0 ** -30
    got = lib.fft2_cpx(a)
    assert close(got, np.fft.fft2(a.astype(np.clongdouble)).astype(complex), x * y)
    assert abs(got[0, 0].imag - math.fsum(a.imag.ravel())) <= (3 * math.log2(x * y) + 4) * ULP * np.abs(a.imag).sum()


@pytest.mark.parametrize("n", [16, 64, 1000, 4096, 8192, 30030, 255])
def test_real(lib, n):
    x = noise((2, n), n).real.copy()
    got = np.asarray(lib.rfft(scaled(x[0], -DOWN)))
    ref = np.asarray(lib.rfft(x[0]))
    assert close(scaled(got, DOWN), ref, n, 2)


# the second operand small: its forward transform's last pass multiplies by the
# first one's spectrum
@pytest.mark.parametrize("n", [64, 1000, 4096, 8192, 1009])
def test_convolution(lib, n):
    a, b = noise((2, n), n).real
    ref = lib.conv_scalar(a.copy(), b.copy())
    got = lib.conv_scalar(a.copy(), scaled(b, -DOWN))
    assert close(scaled(got, DOWN), ref, n, 3)


def test_in_place(lib):
    torch = pytest.importorskip("torch")
    for n in (64, 1000, 4096, 8192, 257):
        x = torch.from_numpy(scaled(noise((5, n), n), -DOWN)).cuda()
        y = torch.empty_like(x)
        p = lib._plan("kfft_config_cpx", n, K.FLAG_NORMAL)
        assert lib.L.kfft_eval_cpx_batch(p, x.data_ptr(), y.data_ptr(), 5) == 0
        assert lib.L.kfft_eval_cpx_batch(p, x.data_ptr(), x.data_ptr(), 5) == 0
        lib.cleanup(p)
        assert torch.equal(x, y), n


def test_queue(lib):
    lengths = np.array([16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 1 << 17, 2, 3, 4, 7, 8, 45, 100, 1000, 30030, 257,
                        4099], np.uint32)
    x = noise(int(lengths.sum()), 1)

    def run(v, flags):
        y = np.empty_like(v)
        p = lib.L.kfft_config_cpx_uneven(len(lengths), lengths.ctypes.data, flags)
        assert p, lib.last_error()
        r = lib.L.kfft_eval_cpx_uneven(p, v.ctypes.data, y.ctypes.data)
        lib.L.kfft_release_uneven(p)
        assert r == 0, lib.last_error()
        return np.split(y, np.cumsum(lengths)[:-1])

    for flags in (K.FLAG_NORMAL, K.FLAG_INVERSE):
        for n, got, ref in zip(lengths.tolist(), run(scaled(x, -DOWN), flags), run(x, flags)):
            assert close(scaled(got, DOWN), ref, max(n, 2), 3), n
