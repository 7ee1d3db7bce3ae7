"""Timed cases of the engine: what a program does with it through its C entry points.

A case is a dict of plain values; ``kind`` names the entry points it goes
through, the rest their sizes and options:

  cpx      complex 1D batch on device buffers, queued on the current stream
           (kfft_eval_cpx_async)
  call     one complex 1D transform per call, synchronous (kfft_eval_cpx), on
           device buffers or, with ``host``, on a drop-in caller's host arrays
  uneven   a batch of complex sequences of different lengths in one launch
           (kfft_eval_cpx_uneven_async)
  real     real 1D batch (kfft_eval_scalar_batch / kfft_evali_scalar_batch)
  cpx2     complex 2D (kfft_eval2_cpx)
  real2    real 2D (kfft_eval2_scalar / kfft_evali2_scalar)
  conv     circular convolution of two real sequences (kfft_eval_conv_scalar)
  conv2    circular convolution of two real images (kfft_eval2_conv_scalar)

``dir`` is "fwd", "inv" or "both" (the forward transform, then the inverse of
its result).  Random inputs are uniform or normal as each workload has them.
"""
import math

import numpy as np
import torch

import kfft_gb300
from kfft_gb300 import FLAG_INVERSE, FLAG_NORMAL

REAL = {"float": torch.float32, "double": torch.float64}
CPX = {"float": torch.complex64, "double": torch.complex128}
SIZE = {"float": 8, "double": 16}  # bytes of a complex value


def listed():
    return [
        # one short spectrum per call, as a program with a loop of its own has it
        {"name": "call_f32_1024", "kind": "call", "precision": "float", "n": 1024, "host": False},
        # a C caller of the reference library, relinked: host arrays in and out
        {"name": "call_host_f64_4096", "kind": "call", "precision": "double", "n": 4096, "host": True},
        # the plain double-precision batch, forward and back
        {"name": "cpx_f64_4096x256", "kind": "cpx", "precision": "double", "n": 4096, "batch": 256,
         "dir": "both"},
        # many sequences of a medium length, float
        {"name": "cpx_f32_2p18x64", "kind": "cpx", "precision": "float", "n": 1 << 18, "batch": 64,
         "dir": "both"},
        # one long sequence, float
        {"name": "cpx_f32_2p24", "kind": "cpx", "precision": "float", "n": 1 << 24, "batch": 1,
         "dir": "fwd"},
        # a length from a sweep over arbitrary integers (1 + 101 k), most of which have a large prime
        {"name": "cpx_f32_500051x34", "kind": "cpx", "precision": "float", "n": 500051, "batch": 34,
         "dir": "fwd"},
        # batches of uneven lengths, half smooth, a quarter with a factor 11 or 13, a quarter prime
        {"name": "uneven_f32_512", "kind": "uneven", "precision": "float", "count": 512, "lo": 16,
         "hi": 1 << 20, "lengths_seed": 2, "dir": "fwd"},
        {"name": "uneven_f64_256", "kind": "uneven", "precision": "double", "count": 256, "lo": 16,
         "hi": 1 << 18, "lengths_seed": 3, "dir": "inv"},
        # long real records, to the spectrum and back
        {"name": "real_f32_2p22x16", "kind": "real", "precision": "float", "n": 1 << 22, "batch": 16,
         "dir": "both"},
        # 2D: a large float array, and a double one
        {"name": "cpx2_f32_8192", "kind": "cpx2", "precision": "float", "x": 8192, "y": 8192,
         "dir": "fwd"},
        {"name": "cpx2_f64_4096", "kind": "cpx2", "precision": "double", "x": 4096, "y": 4096,
         "dir": "both"},
        # a 4096^2 image filtered with a 63 x 63 kernel, both padded to 4160^2
        {"name": "conv2_f32_4160", "kind": "conv2", "precision": "float", "x": 4160, "y": 4160},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _length(rng, lo, hi):
    """A length between lo and hi: a power of two, a smooth number or any integer."""
    n = _log_int(rng, lo, hi)
    how = rng.random()
    if how < 0.3:
        return min(hi, 1 << max(1, int(round(math.log2(n)))))
    if how < 0.65:
        while n > lo and not _smooth(n, 13):
            n -= 1
    return max(n, lo)


def draw(rng):
    precision = rng.choice(["float", "float", "double"])
    points = 1 << (24 if precision == "float" else 22)  # of a 1D batch or a 2D array
    kind = rng.choice(["call", "cpx", "cpx", "cpx", "uneven", "real", "cpx2", "real2", "conv", "conv2"])
    way = rng.choice(["fwd", "inv", "both"])
    if kind == "call":
        return {"kind": kind, "precision": precision, "n": _length(rng, 16, 1 << 16),
                "host": rng.random() < 0.3}
    if kind in ("cpx", "real"):
        n = _length(rng, 16, points >> (1 if kind == "real" else 0))
        return {"kind": kind, "precision": precision, "n": n,
                "batch": _log_int(rng, 1, max(1, points // n)), "dir": way}
    if kind == "uneven":
        return {"kind": kind, "precision": precision, "count": _log_int(rng, 16, 384), "lo": 16,
                "hi": _log_int(rng, 1 << 12, 1 << (20 if precision == "float" else 18)),
                "lengths_seed": rng.randrange(1 << 20), "dir": "inv" if way == "inv" else "fwd"}
    if kind == "conv":
        return {"kind": kind, "precision": precision, "n": _length(rng, 256, points >> 2)}
    x = _length(rng, 32, 4096)
    y = _length(rng, 32, min(4096, points // x))
    if kind == "conv2":
        return {"kind": kind, "precision": precision, "x": x, "y": y}
    return {"kind": kind, "precision": precision, "x": x, "y": y,
            "dir": "both" if kind == "real2" and way == "inv" else way}


# ---- inputs ---------------------------------------------------------------------


def _smooth(n, top):
    for p in (2, 3, 5, 7, 11, 13):
        if p > top:
            break
        while n % p == 0:
            n //= p
    return n == 1


def _is_prime(n):
    return n > 1 and all(n % p for p in range(2, math.isqrt(n) + 1))


def _uneven_lengths(case):
    """Log-uniform lengths, snapped: half 7-smooth, a quarter 7-smooth times 11 or 13, a quarter prime."""
    rng = np.random.default_rng(case["lengths_seed"])
    out = []
    for i in range(case["count"]):
        n = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        if i % 4 < 2:
            while not _smooth(n, 7):
                n -= 1
        elif i % 4 == 2:
            f = (11, 13)[i // 4 % 2]
            m = max(2, n // f)
            while not _smooth(m, 7):
                m -= 1
            n = m * f
        else:
            n = max(n, 17)
            while not _is_prime(n):
                n -= 1
        out.append(n)
    return [out[i] for i in rng.permutation(len(out))]


def _random(case, seed, shape, kind):
    g = torch.Generator(device="cuda").manual_seed(seed * 1000003 + 17)
    dt = (CPX if kind != "real" else REAL)[case["precision"]]
    if kind == "normal":
        real = REAL[case["precision"]]
        return torch.complex(torch.randn(shape, generator=g, dtype=real, device="cuda"),
                             torch.randn(shape, generator=g, dtype=real, device="cuda"))
    v = torch.rand(shape if kind == "real" else tuple(shape) + (2,), generator=g,
                   dtype=REAL[case["precision"]], device="cuda")
    v = v * 2 - 1
    return v if kind == "real" else torch.view_as_complex(v).to(dt)


def _inputs(case, seed):
    """The input tensors of a case, on the GPU."""
    kind = case["kind"]
    if kind == "call":
        return [_random(case, seed, (case["n"],), "uniform")]
    if kind == "cpx":
        return [_random(case, seed, (case["batch"], case["n"]), "normal")]
    if kind == "uneven":
        return [_random(case, seed, (sum(_uneven_lengths(case)),), "normal")]
    if kind == "real":
        x = _random(case, seed, (case["batch"], case["n"]), "real")
        return [torch.fft.fft(x) if case["n"] % 2 else torch.fft.rfft(x)] if case["dir"] == "inv" else [x]
    if kind == "cpx2":
        return [_random(case, seed, (case["y"], case["x"]), "uniform")]
    if kind == "real2":
        return [_random(case, seed, (case["y"], case["x"]), "real")]
    if kind == "conv":
        # a signal and a decaying response, zero-padded to the same length
        n = case["n"]
        b = _random(case, seed + 1, (n,), "real") * torch.exp(
            -torch.arange(n, device="cuda") * (8.0 / n)).to(REAL[case["precision"]])
        b[n // 2:] = 0
        return [_random(case, seed, (n,), "real"), b]
    # conv2: a non-negative image and a 63 x 63 Gaussian, zero-padded
    y, x = case["y"], case["x"]
    image = _random(case, seed, (y, x), "real") * 0.5 + 0.5
    ky, kx = min(63, y), min(63, x)
    image[y - min(y // 2, ky - 1):] = 0
    image[:, x - min(x // 2, kx - 1):] = 0
    gy, gx = (torch.exp(-((torch.arange(k, dtype=torch.float64, device="cuda") - k // 2) ** 2) / 128.0)
              for k in (ky, kx))
    g = gy[:, None] * gx[None, :]
    kernel = torch.zeros((y, x), dtype=REAL[case["precision"]], device="cuda")
    kernel[:ky, :kx] = (g / g.sum()).to(kernel.dtype)
    return [image, kernel]


# ---- plans and calls --------------------------------------------------------------


class _Plan:
    """A plan that is released with its last reference."""

    def __init__(self, lib, handle, release):
        if not handle:
            raise RuntimeError("no plan: " + lib.last_error())
        self.handle, self._release = handle, release

    def __del__(self):
        if self.handle and torch is not None:
            torch.cuda.synchronize()
            self._release(self.handle)
            self.handle = None


def _plan(lib, config, *args):
    return _Plan(lib, getattr(lib.L, config)(*args, None, None), lib.L.kfft_cleanup)


def prepare(case, seed):
    lib = kfft_gb300.load(case["precision"])
    kind = case["kind"]
    state = {"case": case, "lib": lib}
    ins = _inputs(case, seed)
    way = case.get("dir", "fwd")
    plans = {}
    sides = [(d, f) for d, f in (("fwd", FLAG_NORMAL), ("inv", FLAG_INVERSE)) if way in (d, "both")]
    cpx, real = CPX[case["precision"]], REAL[case["precision"]]
    outs = {}

    def empty(shape, dtype):
        return torch.empty(shape, dtype=dtype, device="cuda")

    if kind == "call":
        plans["fwd"] = _plan(lib, "kfft_config_cpx", case["n"], FLAG_NORMAL)
        if case["host"]:
            ins = [v.cpu().numpy() for v in ins]
            outs["fwd"] = np.empty_like(ins[0])
        else:
            outs["fwd"] = torch.empty_like(ins[0])
    elif kind == "cpx":
        for d, f in sides:
            plans[d] = _plan(lib, "kfft_config_cpx", case["n"], f)
            outs[d] = torch.empty_like(ins[0])
    elif kind == "uneven":
        lengths = np.array(_uneven_lengths(case), dtype=np.uint32)
        f = FLAG_INVERSE if way == "inv" else FLAG_NORMAL
        plans[way] = _Plan(lib, lib.L.kfft_config_cpx_uneven(len(lengths), lengths.ctypes.data, f),
                           lib.L.kfft_release_uneven)
        outs[way] = torch.empty_like(ins[0])
    elif kind == "real":
        n, b = case["n"], case["batch"]
        for d, f in sides:
            plans[d] = _plan(lib, "kfft_config_scalar", n, f)
            outs[d] = empty((b, n), real) if d == "inv" else empty((b, n if n % 2 else n // 2 + 1), cpx)
    elif kind in ("cpx2", "real2"):
        config = "kfft_config2_cpx" if kind == "cpx2" else "kfft_config2_scalar"
        for d, f in sides:
            plans[d] = _plan(lib, config, case["x"], case["y"], f)
            outs[d] = empty((case["y"], case["x"]), real if kind == "real2" and d == "inv" else cpx)
    elif kind == "conv":
        plans["conv"] = _plan(lib, "kfft_config_conv_scalar", case["n"], FLAG_NORMAL)
        outs["conv"] = empty((case["n"],), real)
    else:
        plans["conv"] = _plan(lib, "kfft_config2_conv_scalar", case["x"], case["y"], FLAG_NORMAL)
        outs["conv"] = empty((case["y"], case["x"]), real)
    state.update(ins=ins, plans=plans, outs=outs)
    return state


def _at(v):
    return v.ctypes.data if isinstance(v, np.ndarray) else v.data_ptr()


def run(state):
    case, lib, outs = state["case"], state["lib"].L, state["outs"]
    src = state["ins"][0]
    kind = case["kind"]
    for d, plan in state["plans"].items():
        p, dst = plan.handle, outs[d]
        if kind == "call":
            r = lib.kfft_eval_cpx(p, _at(src), _at(dst))
        elif kind == "cpx":
            r = lib.kfft_eval_cpx_async(p, _at(src), _at(dst), case["batch"],
                                        torch.cuda.current_stream().cuda_stream)
        elif kind == "uneven":
            r = lib.kfft_eval_cpx_uneven_async(p, _at(src), _at(dst),
                                               torch.cuda.current_stream().cuda_stream)
        elif kind == "real":
            call = lib.kfft_eval_scalar_batch if d == "fwd" else lib.kfft_evali_scalar_batch
            r = call(p, _at(src), _at(dst), case["batch"])
        elif kind == "cpx2":
            r = lib.kfft_eval2_cpx(p, _at(src), _at(dst))
        elif kind == "real2":
            r = (lib.kfft_eval2_scalar if d == "fwd" else lib.kfft_evali2_scalar)(p, _at(src), _at(dst))
        elif kind == "conv":
            r = lib.kfft_eval_conv_scalar(p, _at(src), _at(state["ins"][1]), _at(dst))
        else:
            r = lib.kfft_eval2_conv_scalar(p, _at(src), _at(state["ins"][1]), _at(dst))
        if r != kfft_gb300.RET_SUCCESS:
            raise RuntimeError("%s: %s" % (case, state["lib"].last_error()))
        src = dst
    return dict(outs)


# ---- what the work is, and its result in 64 bits ----------------------------------


def work(case):
    """Bytes: each input read once and each output written once, per transform.  Flops: 5 N log2 N
    per complex transform and half of that per real one."""
    kind, s = case["kind"], SIZE[case["precision"]]
    sides = 2 if case.get("dir") == "both" else 1

    def cost(n):
        return 5.0 * n * math.log2(max(n, 2))

    if kind == "call":
        return {"bytes": 2 * s * case["n"], "flops": cost(case["n"])}
    if kind == "cpx":
        n, b = case["n"], case["batch"]
        return {"bytes": sides * 2 * s * n * b, "flops": sides * b * cost(n)}
    if kind == "uneven":
        lengths = _uneven_lengths(case)
        return {"bytes": 2 * s * sum(lengths), "flops": sum(cost(n) for n in lengths)}
    if kind == "real":
        n, b = case["n"], case["batch"]
        bins = n if n % 2 else n // 2 + 1
        return {"bytes": sides * b * (s * n // 2 + s * bins), "flops": sides * b * cost(n) / 2}
    if kind == "conv":
        n = case["n"]
        return {"bytes": 3 * s * n // 2, "flops": 3 * cost(n) / 2}
    n = case["x"] * case["y"]
    if kind == "cpx2":
        return {"bytes": sides * 2 * s * n, "flops": sides * cost(n)}
    if kind == "real2":
        return {"bytes": sides * 3 * s * n // 2, "flops": sides * cost(n) / 2}
    return {"bytes": 3 * s * n // 2, "flops": 3 * cost(n) / 2}


def exact(case, seed):
    kind, way = case["kind"], case.get("dir", "fwd")
    ins = [v.to(torch.complex128 if v.is_complex() else torch.float64) for v in _inputs(case, seed)]
    x = ins[0]
    if kind == "call":
        return {"fwd": torch.fft.fft(x)}
    if kind in ("cpx", "cpx2"):
        fwd, inv = (torch.fft.fft, torch.fft.ifft) if kind == "cpx" else (torch.fft.fft2, torch.fft.ifft2)
        if way == "both":
            return {"fwd": fwd(x), "inv": x}
        return {way: (inv if way == "inv" else fwd)(x)}
    if kind == "uneven":
        f = torch.fft.ifft if way == "inv" else torch.fft.fft
        return {way: torch.cat([f(v) for v in torch.split(x, _uneven_lengths(case))])}
    # the inverse of a real transform of an even length is twice the input, as the reference has it
    if kind == "real":
        twice = 1.0 if case["n"] % 2 else 2.0
        if way == "inv":
            n = case["n"]
            return {"inv": torch.fft.ifft(x).real if n % 2 else 2.0 * torch.fft.irfft(x, n=n)}
        out = {"fwd": torch.fft.fft(x) if case["n"] % 2 else torch.fft.rfft(x)}
        return {**out, "inv": twice * x} if way == "both" else out
    if kind == "real2":
        out = {"fwd": torch.fft.fft2(x)}
        return {**out, "inv": (1.0 if case["y"] % 2 else 2.0) * x} if way == "both" else out
    n = case["n"] if kind == "conv" else case["y"]
    twice = 1.0 if n % 2 else 2.0
    if kind == "conv":
        return {"conv": twice * torch.fft.irfft(torch.fft.rfft(x) * torch.fft.rfft(ins[1]), n=n)}
    return {"conv": twice * torch.fft.irfft2(torch.fft.rfft2(x) * torch.fft.rfft2(ins[1]),
                                             s=(case["y"], case["x"]))}
