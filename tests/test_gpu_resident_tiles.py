"""FP32 passes on resident grids that copy their tiles in (bulk copies of whole
sequences, asynchronous copies of rows), on device buffers large enough that
they take these kernels: every pass length, partly filled last tiles, rows of
odd length and the stores of products, against FP64."""
import numpy as np
import pytest

import kfft_gb300 as K
from tests.helpers import TOL32, rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TILE = 4096  # points of a full tile


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def rand(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.complex(torch.randn(shape, generator=g, device="cuda"), torch.randn(shape, generator=g, device="cuda"))


def passes(lib, n):
    """The plan's text."""
    p = lib._plan("kfft_config_cpx", n, 0)
    text = lib.describe(p)
    lib.cleanup(p)
    return text


def check_rows(x, y, flags, rows):
    f = np.fft.ifft if flags else np.fft.fft
    for r in sorted(set(rows)):
        ref = f(x[r].cpu().numpy().astype(np.complex128))
        assert rel_l2(y[r].cpu().numpy(), ref) <= TOL32, r


def batch_call(lib, x, y, flags):
    p = lib._plan("kfft_config_cpx", x.shape[1], flags)
    r = lib.L.kfft_eval_cpx_batch(p, x.data_ptr(), y.data_ptr(), x.shape[0])
    lib.cleanup(p)
    assert r == 0, lib.last_error()


# whole sequences: a third round of tiles just begun, two full rounds and a bit
@pytest.mark.parametrize("tiles", [4, 6])
@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_bulk_copied_sequences(libf, n, tiles):
    per_tile = TILE // n
    batch = (tiles * sms() + 2) * per_tile + max(1, per_tile // 2 - 1)
    x = rand((batch, n), n)
    rows = [0, 1, per_tile, batch // 3, batch // 2, batch - per_tile, batch - 2, batch - 1]
    for flags in (K.FLAG_NORMAL, K.FLAG_INVERSE):
        y = torch.full_like(x, 7)
        batch_call(libf, x, y, flags)
        check_rows(x, y, flags, rows)
        z = x.clone()  # and in place
        batch_call(libf, z, z, flags)
        assert torch.equal(z, y)


# rows of several lanes, a tile's among them from two sequences (104 and 80
# lanes, tiles of 32 and 64), on 16 bytes and 8 bytes off them
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n,lengths", [(13312, (128,)), (5120, (64,)), (10240, (128,)), (1 << 18, (1024, 256))])
def test_rows_of_sequences(libf, n, lengths, off):
    text = passes(libf, n)
    for r in lengths:
        assert f"R={r}" in text, text
    batch = (6 * sms() * TILE) // n + 2
    buf = torch.zeros(batch * n + off, dtype=torch.complex64, device="cuda")
    x = buf[off:].view(batch, n)
    x.copy_(rand((batch, n), n))
    y = torch.empty_like(x)
    for flags in (K.FLAG_NORMAL, K.FLAG_INVERSE):
        batch_call(libf, x, y, flags)
        check_rows(x, y, flags, [0, 1, batch // 2, batch - 2, batch - 1])


# down the columns of an array: pass lengths 16 .. 1024, even and odd numbers of columns
@pytest.mark.parametrize("y,x", [(16, 234000), (16, 234375), (32, 117000), (32, 117649), (64, 58500), (64, 59049),
                                 (128, 30030), (256, 15625), (512, 7350), (512, 7371), (1024, 4096), (1024, 3993)])
def test_columns(libf, y, x):
    assert f"R={y}" in passes(libf, y)
    a = rand((y, x), x)
    out = torch.empty_like(a)
    for flags, f in ((K.FLAG_NORMAL, torch.fft.fft2), (K.FLAG_INVERSE, torch.fft.ifft2)):
        p = libf._plan("kfft_config2_cpx", x, y, flags)
        assert libf.L.kfft_eval2_cpx(p, a.data_ptr(), out.data_ptr()) == 0, libf.last_error()
        libf.cleanup(p)
        ref = f(a.to(torch.complex128))
        assert float(torch.linalg.norm(out - ref) / torch.linalg.norm(ref)) <= TOL32


# the stores of products: Bluestein's filter and chirp (over several passes and
# over one), Rader's scatter (likewise)
@pytest.mark.parametrize("n,kind,batch", [(500051, "bluestein", 5), (1019, "bluestein", 2000), (2027, "bluestein", 1000),
                                          (257, "rader", 16000), (65537, "rader", 66)])
def test_products(libf, n, kind, batch):
    assert kind in passes(libf, n)
    x = rand((batch, n), n)
    y = torch.empty_like(x)
    for flags in (K.FLAG_NORMAL, K.FLAG_INVERSE):
        batch_call(libf, x, y, flags)
        check_rows(x, y, flags, [0, 1, batch // 2, batch - 2, batch - 1])


@pytest.mark.parametrize("y,x", [(1024, 4096), (512, 8192), (256, 16384), (256, 16385 - 10)])
def test_convolution_product(libf, y, x):
    a, b = rand((y, x), 1), rand((y, x), 2)
    out = torch.empty_like(a)
    p = libf._plan("kfft_config2_conv_cpx", x, y, K.FLAG_NORMAL)
    assert libf.L.kfft_eval2_conv_cpx(p, a.data_ptr(), b.data_ptr(), out.data_ptr()) == 0, libf.last_error()
    libf.cleanup(p)
    ref = torch.fft.ifft2(torch.fft.fft2(a.to(torch.complex128)) * torch.fft.fft2(b.to(torch.complex128)))
    assert float(torch.linalg.norm(out - ref) / torch.linalg.norm(ref)) <= 2 * TOL32
