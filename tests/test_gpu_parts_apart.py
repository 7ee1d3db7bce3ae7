"""Double build: parts that arithmetic in doubles keeps apart from larger ones
are as accurate as in doubles (lanes of such parts run in FP64)."""
import math

import numpy as np
import pytest

import kfft_gb300 as K

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -53
# additions only; one and more passes; every first radix; primes (Rader)
SIZES = [2, 3, 4, 5, 8, 12, 15, 16, 32, 45, 64, 100, 256, 512, 1000, 1024, 2048, 4096, 8192, 30030, 65536]
PRIMES = [101, 257]


def noise(n, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(n) + 1j * rng.standard_normal(n)


def both_ways(lib, x):
    """The result of `x` alone and within a batch of ordinary sequences."""
    n = x.size
    batch = np.stack([noise(n, 1), x, noise(n, 2)])
    return lib.fft_cpx(x), lib.fft_cpx(batch)[1]


def bound(n, terms):
    """A transform's rounding errors on the way to a part, as a multiple of what
    is added up there: one an addition and product of each radix-2 step or its
    like, three transforms where it is a convolution."""
    return 3 * (3 * math.log2(n) + 4) * ULP * terms


@pytest.mark.parametrize("n", [2, 4, 8, 12, 15, 16, 64, 100, 1000, 2048, 4096, 8192, 65536])
def test_one_value_stays_itself(lib, n):
    """A value at index 0 alone: every bin is that value, to the last bit."""
    x = np.zeros(n, complex)
    x[0] = 1e18 + 1.25j
    for y in both_ways(lib, x):
        assert np.all(y == x[0])


@pytest.mark.parametrize("e", [-8, -20, -40, -70])
@pytest.mark.parametrize("n", SIZES + PRIMES)
def test_nearly_real(lib, n, e):
    """Imaginary parts 2^e of the real ones: bin 0 adds up each by itself."""
    z = noise(n, n)
    for x in (z.real + 1j * z.imag * 2.0 ** e, z.imag * 2.0 ** e + 1j * z.real):
        for y in both_ways(lib, x):
            assert abs(y[0].real - math.fsum(x.real)) <= bound(n, np.abs(x.real).sum())
            assert abs(y[0].imag - math.fsum(x.imag)) <= bound(n, np.abs(x.imag).sum())


@pytest.mark.parametrize("e", [-12, -40, -70])
@pytest.mark.parametrize("n", [s for s in SIZES if s > 2])
def test_impulse_over_noise(lib, n, e):
    """A real value at index 0 over complex noise: no imaginary part sees it."""
    x = noise(n, n) * 2.0 ** e
    rest = float(np.linalg.norm(x[1:]))
    x[0] = 1.3 + 1j * x[0].imag
    ref = np.fft.fft(x.astype(np.clongdouble))
    for y in both_ways(lib, x):
        err = np.linalg.norm((y.imag - ref.imag).astype(float))
        assert err <= bound(n, rest) * math.sqrt(n)
    x *= 1j  # the same for the real parts
    ref = ref * 1j
    for y in both_ways(lib, x):
        err = np.linalg.norm((y.real - ref.real).astype(float))
        assert err <= bound(n, rest) * math.sqrt(n)


@pytest.mark.parametrize("at", [1, 2, 3])
@pytest.mark.parametrize("n", [8, 16, 64, 512, 4096, 65536])
def test_impulse_on_an_axis(lib, n, at):
    """A real value at index n at / 4: it stays on an axis in every bin, so the
    other part of the bin is the noise's."""
    x = noise(n, n) * 2.0 ** -30
    rest = float(np.linalg.norm(x))
    x[n * at // 4] = 1.3
    ref = np.fft.fft(x.astype(np.clongdouble))
    k = np.arange(n) * at % 4  # the bin's turn of the value, in quarters
    for y in both_ways(lib, x):
        d = (y - ref).astype(complex)
        other = np.where(k % 2 == 0, d.imag, d.real)
        assert float(np.linalg.norm(other)) <= bound(n, rest) * math.sqrt(n)


@pytest.mark.parametrize("n", [8, 16, 64, 512, 4096])
@pytest.mark.parametrize("parity", [0, 1])
def test_real_values_of_two_sizes(lib, n, parity):
    """Real values, every second one tiny: bin n / 4 has them in a part each."""
    x = noise(n, n).real + 0j
    x[parity::2] *= 2.0 ** -30
    re = math.fsum(v * (1, 0, -1, 0)[i % 4] for i, v in enumerate(x.real))
    im = math.fsum(v * (0, -1, 0, 1)[i % 4] for i, v in enumerate(x.real))
    for y in both_ways(lib, x):
        assert abs(y[n // 4].real - re) <= bound(n, np.abs(x.real[0::2]).sum())
        assert abs(y[n // 4].imag - im) <= bound(n, np.abs(x.real[1::2]).sum())


def test_queue(lib):
    """The same in the queue kernel."""
    lengths = np.array([2, 3, 4, 8, 16, 45, 64, 100, 512, 1000, 2048, 4096, 30030], np.uint32)
    xs = []
    for n in lengths.tolist():
        x = noise(n, n) * 2.0 ** -40
        x[0] = 1.3
        xs.append(x)
    x = np.concatenate(xs)
    y = np.empty_like(x)
    p = lib.L.kfft_config_cpx_uneven(len(lengths), lengths.ctypes.data, K.FLAG_NORMAL)
    assert p, lib.last_error()
    r = lib.L.kfft_eval_cpx_uneven(p, x.ctypes.data, y.ctypes.data)
    lib.L.kfft_release_uneven(p)
    assert r == 0, lib.last_error()
    at = 0
    for n, v in zip(lengths.tolist(), xs):
        ref = np.fft.fft(v.astype(np.clongdouble))
        err = np.linalg.norm((y[at:at + n].imag - ref.imag).astype(float))
        assert err <= bound(n, float(np.linalg.norm(v[1:]))) * math.sqrt(n), n
        at += n
