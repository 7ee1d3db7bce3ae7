"""FP32 power-of-two passes on resident grids: tiles that arrive by
asynchronous copies (two lanes at a time, or one where the rows do not pair up
on 16 bytes) and by bulk copies, against FP64."""
import numpy as np
import pytest

import kfft_gb300 as K
from tests.helpers import TOL32, rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# enough points for two tiles of 4096 per resident CTA (152 SMs x 3)
POINTS = 4 << 20


def device(a, off):
    """`a` on the GPU, `off` complex values past an aligned address."""
    t = torch.empty(a.size + off, dtype=torch.complex64, device="cuda")
    t[off:] = torch.from_numpy(a).cuda().reshape(-1)
    return t, t.data_ptr() + 8 * off


# lengths whose passes cover 16..1024 points, with even and odd lane counts
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n", [1 << 13, 1 << 15, 1 << 18, 1 << 20, 1 << 21, 16 * 375, 45 * 1024, 512 * 13, 256 * 27])
def test_batches_at_any_alignment(libf, n, off):
    batch = -(-POINTS // n) + 1
    rng = np.random.default_rng(n)
    x = rng.standard_normal((batch, n), np.float32) + 1j * rng.standard_normal((batch, n), np.float32)
    tx, px = device(x.astype(np.complex64), off)
    ty, py = device(np.zeros_like(x, np.complex64), off)
    for flags, f in ((0, np.fft.fft), (K.FLAG_INVERSE, np.fft.ifft)):
        p = libf._plan("kfft_config_cpx", n, flags)
        assert libf.L.kfft_eval_cpx_batch(p, px, py, batch) == 0, libf.last_error()
        libf.cleanup(p)
        y = ty[off:].cpu().numpy().reshape(batch, n)
        rows = [0, 1, batch // 2, batch - 1]
        ref = f(x[rows].astype(np.complex128), axis=1)
        for i, r in enumerate(rows):
            assert rel_l2(y[r], ref[i]) <= TOL32, (flags, r)


# columns: even and odd counts of them
@pytest.mark.parametrize("x", [2048, 2049, 2050])
@pytest.mark.parametrize("y", [2048, 8192])
def test_columns(libf, x, y):
    rng = np.random.default_rng(x)
    a = (rng.standard_normal((y, x), np.float32) + 1j * rng.standard_normal((y, x), np.float32)).astype(np.complex64)
    got = libf.fft2_cpx(a)
    assert rel_l2(got, np.fft.fft2(a.astype(np.complex128))) <= TOL32
    back = libf.fft2_cpx(got, K.FLAG_INVERSE)
    assert rel_l2(back, a) <= 2 * TOL32


# single-pass batches, a last tile that is not full among them
@pytest.mark.parametrize("n", [16, 64, 128, 512, 1024, 2048, 4096])
def test_contiguous_batches(libf, n):
    batch = POINTS // n + 3
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((batch, n), np.float32) + 1j * rng.standard_normal((batch, n), np.float32)).astype(np.complex64)
    y = libf.fft_cpx(x)
    ref = np.fft.fft(x[-8:].astype(np.complex128), axis=1)
    assert rel_l2(y[-8:], ref) <= TOL32
    assert rel_l2(y[:8], np.fft.fft(x[:8].astype(np.complex128), axis=1)) <= TOL32


# run-time tiles: every radix in the first place and behind others, one, two
# and more stages, and (through Bluestein and a convolution) the product stores
@pytest.mark.parametrize("n", [3, 5, 6, 7, 9, 10, 11, 12, 13, 14, 15, 24, 36, 60, 105, 169, 196, 225, 240,
                               1000, 1080, 1155, 1728, 1920, 2016, 2187, 2197, 2310, 3003, 3375, 4000, 4095,
                               4160, 59049, 100000, 1009, 4111])
def test_run_time_tiles(libf, n):
    batch = max(3, 20000 // n)
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((batch, n), np.float32) + 1j * rng.standard_normal((batch, n), np.float32)).astype(np.complex64)
    y = libf.fft_cpx(x)
    assert rel_l2(y, np.fft.fft(x.astype(np.complex128), axis=1)) <= TOL32
    z = libf.fft_cpx(x, K.FLAG_INVERSE)
    assert rel_l2(z, np.fft.ifft(x.astype(np.complex128), axis=1)) <= TOL32


@pytest.mark.parametrize("y,x", [(52, 80), (90, 182), (128, 100), (75, 64)])
def test_run_time_tiles_convolve(libf, y, x):
    rng = np.random.default_rng(y * x)
    a, b = (rng.uniform(0, 1, (y, x)).astype(np.float32) for _ in range(2))
    ref = np.fft.ifft2(np.fft.fft2(a.astype(float)) * np.fft.fft2(b.astype(float))).real
    got = libf.conv2_scalar(a, b)
    assert rel_l2(got, ref * (1 if y % 2 else 2)) <= TOL32
    c = libf.conv2_cpx(a.astype(np.complex64), b.astype(np.complex64))
    assert rel_l2(c, ref) <= TOL32


# one-stage batches: rows stored 16 bytes at a time, of even and odd length,
# from an aligned address and from 8 bytes past one, and in place
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n", range(2, 17))
def test_one_stage_rows(libf, n, off):
    for batch in (1, 2 * 4096 // n + 3):
        rng = np.random.default_rng(n)
        x = (rng.standard_normal((batch, n), np.float32) + 1j * rng.standard_normal((batch, n), np.float32)).astype(np.complex64)
        tx, px = device(x, off)
        ty, py = device(np.full((batch + 1, n), 7, np.complex64), off)
        ref = np.fft.fft(x.astype(np.complex128), axis=1)
        p = libf._plan("kfft_config_cpx", n, 0)
        assert libf.L.kfft_eval_cpx_batch(p, px, py, batch) == 0, libf.last_error()
        y = ty[off:].cpu().numpy().reshape(batch + 1, n)
        assert rel_l2(y[:batch], ref) <= TOL32
        assert (y[batch] == 7).all()
        assert libf.L.kfft_eval_cpx_batch(p, px, px, batch) == 0, libf.last_error()
        libf.cleanup(p)
        assert rel_l2(tx[off:].cpu().numpy().reshape(batch, n), ref) <= TOL32
