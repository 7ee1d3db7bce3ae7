"""Prime lengths by Rader's convolution: x_0 is in no part of the convolution,
so it reaches every output as it is: infinite, or far larger than the rest."""
import math

import numpy as np
import pytest

import kfft_gb300 as K

pytestmark = pytest.mark.gpu

# convolutions of one pass and of more, of every kind of tile
PRIMES = [37, 101, 257, 1009, 12289, 65537]


@pytest.fixture(params=["double", "float"])
def either(request, lib, libf):
    return (lib, 2.0 ** -53) if request.param == "double" else (libf, 2.0 ** -24)


def noise(lib, n, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(lib.cpx)


@pytest.mark.parametrize("flags", [K.FLAG_NORMAL, K.FLAG_INVERSE])
@pytest.mark.parametrize("n", PRIMES)
def test_infinite_first_value(either, n, flags):
    lib, _ = either
    p = lib._plan("kfft_config_cpx", n, flags)
    assert "rader" in lib.describe(p)
    lib.cleanup(p)
    x = np.stack([noise(lib, n, n + i) for i in range(3)])
    x.real[:, 0] = 0
    plain = lib.fft_cpx(x, flags)
    x.real[1, 0] = np.inf
    y = lib.fft_cpx(x, flags)
    assert np.all(y[1].real == np.inf)
    # (the parts that the infinity does not touch come from the same arithmetic)
    assert np.array_equal(y[1].imag, plain[1].imag)
    assert np.array_equal(y[[0, 2]], plain[[0, 2]])


@pytest.mark.parametrize("e", [-8, -12, -40, -70])
@pytest.mark.parametrize("n", PRIMES)
def test_large_first_value(either, n, e):
    """A real x_0 over noise of 2^e: the imaginary parts are the noise's."""
    lib, ulp = either
    x = noise(lib, n, n) * lib.real(2.0 ** e)
    rest = float(np.linalg.norm(x[1:]))
    x[0] = 1j * x[0].imag
    ref = np.fft.fft(x.astype(np.clongdouble)).imag  # (x_0's real part reaches none of these)
    x[0] += lib.real(1.25)
    y = lib.fft_cpx(x)
    # three roundings a radix-2 step or its like, in each of three transforms
    tol = 3 * (3 * math.log2(n) + 4) * ulp * rest * math.sqrt(n)
    assert np.linalg.norm((y.imag - ref).astype(float)) <= tol
