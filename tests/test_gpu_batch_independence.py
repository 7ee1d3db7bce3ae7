"""Double build: what becomes of a sequence depends on its own values alone, to
the last bit: not on what else is in the batch, whichever of them need FP64."""
import numpy as np
import pytest

import kfft_gb300 as K

pytestmark = pytest.mark.gpu

SIZES = [3, 5, 8, 12, 16, 32, 45, 64, 100, 128, 256, 512, 1000, 1024, 2048, 4096, 8192, 30030, 65536, 101, 4099]


def noise(shape, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def odd_ones(n):
    """Sequences that leave the fixed-point tiles, or take the closer look."""
    z = noise((8, n), n)
    z[0, n // 2] = np.inf
    z[1, 0] = np.nan
    z[2] *= 2.0 ** -900
    z[3].imag *= 2.0 ** -30
    z[4, 1:] *= 2.0 ** -40
    z[5].imag = 0
    z[6, :] = 0
    z[6, n // 3] = 1
    z[7] *= 2.0 ** 800
    return z


@pytest.mark.parametrize("flags", [K.FLAG_NORMAL, K.FLAG_INVERSE])
@pytest.mark.parametrize("n", SIZES)
def test_sequences(lib, n, flags):
    plain, odd = noise((11, n), 3 * n), odd_ones(n)
    y = lib.fft_cpx(plain, flags)
    alone = [lib.fft_cpx(v, flags) for v in odd]
    mixed = plain.copy()
    at = [1, 2, 4, 5, 6, 8, 9, 10]
    mixed[at] = odd
    got = lib.fft_cpx(mixed, flags)
    rest = [i for i in range(11) if i not in at]
    assert np.array_equal(got[rest], y[rest])
    for i, a in zip(at, alone):
        assert np.array_equal(got[i], a, equal_nan=True), i
    assert np.array_equal(lib.fft_cpx(plain[3], flags), y[3])


@pytest.mark.parametrize("y", [12, 64, 512, 1000, 4096])
def test_columns(lib, y):
    """The columns of an array whose rows are copies of one value each: the row
    transforms leave column 0 with all of it, the others with zeros."""
    x = 36
    a = np.zeros((y, x), complex)
    a[:, 0] = noise(y, y)
    plain = lib.fft2_cpx(a)  # every column the same sequence
    b = a.copy()
    b[0, 5] = 1e-3  # spreads into every bin of row 0: columns differ, all ordinary
    c = lib.fft2_cpx(b)
    assert all(np.array_equal(plain[:, 0], plain[:, k]) for k in range(x))
    ref = np.fft.fft2(b.astype(np.clongdouble))
    assert float(np.linalg.norm(c - ref) / np.linalg.norm(ref)) <= 1e-15


def test_queue(lib):
    lengths = np.array([64, 100, 512, 1000, 4096, 8192, 45, 2048, 257, 16], np.uint32)

    def run(v):
        y = np.empty_like(v)
        p = lib.L.kfft_config_cpx_uneven(len(lengths), lengths.ctypes.data, K.FLAG_NORMAL)
        assert p, lib.last_error()
        r = lib.L.kfft_eval_cpx_uneven(p, v.ctypes.data, y.ctypes.data)
        lib.L.kfft_release_uneven(p)
        assert r == 0, lib.last_error()
        return np.split(y, np.cumsum(lengths)[:-1])

    x = noise(int(lengths.sum()), 5)
    ref = run(x)
    at = np.cumsum(lengths)
    x[at[0]:at[1]].imag *= 2.0 ** -40
    x[at[3]] = np.inf
    got = run(x)
    for i in range(len(lengths)):
        if i not in (1, 4):
            assert np.array_equal(got[i], ref[i]), i


@pytest.mark.parametrize("n", [8, 45, 64, 512, 1000, 2048, 8192, 257])
def test_in_place(lib, n):
    """The tiles that do some lanes after the others, on one buffer."""
    torch = pytest.importorskip("torch")
    mixed = noise((11, n), 3 * n)
    mixed[[1, 2, 4, 5, 6, 8, 9, 10]] = odd_ones(n)
    x = torch.from_numpy(mixed).cuda()
    y = torch.empty_like(x)
    for flags in (K.FLAG_NORMAL, K.FLAG_INVERSE):
        z = x.clone()
        p = lib._plan("kfft_config_cpx", n, flags)
        assert lib.L.kfft_eval_cpx_batch(p, x.data_ptr(), y.data_ptr(), 11) == 0
        assert lib.L.kfft_eval_cpx_batch(p, z.data_ptr(), z.data_ptr(), 11) == 0
        lib.cleanup(p)
        assert np.array_equal(y.cpu().numpy(), z.cpu().numpy(), equal_nan=True)


@pytest.mark.parametrize("y,x", [(64, 40), (512, 36), (45, 40), (4096, 20), (8192, 20)])
def test_columns_in_place(lib, y, x):
    """Likewise down columns, of which every fifth row-transforms to nearly real
    values."""
    torch = pytest.importorskip("torch")
    a = noise((y, x), x)
    cols = np.fft.fft(a, axis=1)
    cols[:, ::5].imag *= 2.0 ** -20
    t = torch.from_numpy(np.ascontiguousarray(np.fft.ifft(cols, axis=1))).cuda()
    out, z = torch.empty_like(t), t.clone()
    p = lib._plan("kfft_config2_cpx", x, y, K.FLAG_NORMAL)
    assert lib.L.kfft_eval2_cpx(p, t.data_ptr(), out.data_ptr()) == 0
    assert lib.L.kfft_eval2_cpx(p, z.data_ptr(), z.data_ptr()) == 0
    lib.cleanup(p)
    assert torch.equal(out, z)
    ref = torch.fft.fft2(t)
    assert float(torch.linalg.norm(out - ref) / torch.linalg.norm(ref)) <= 1e-15
