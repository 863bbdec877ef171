"""The transforms a user of this library runs, at the sizes they run them.

Every case is one call of a compiled computation: ``FFT`` (``c2c``, one or several axes,
forward or inverse, optionally with the fused output fftshift and 1/N scale),
``spectrogram`` and the real transforms ``RFFT`` / ``IRFFT``.  Sizes are the ones of the
benchmark workloads (``bench.py``), of the serving stream's ranges (1-D lengths 61 to
2^20 with powers of two and ragged lengths, 2-D sides up to 2048, spectrograms of up to
2^22 samples) and of the test suite.
"""

from __future__ import annotations

import math

import numpy
import torch

from reikna_b200 import transformations as tr
from reikna_b200.core import ArrayMetadata
from reikna_b200.fft import FFT, IRFFT, RFFT
from reikna_b200.spectrogram import frames, spectrogram

MAX_ELEMS = 2**24  # elements of the largest array (256^3)


def _c2c(shape, axes, dtype="complex64", inverse=False, shift_scale=False, name=None):
    case = {"kind": "c2c", "shape": "x".join(map(str, shape)), "axes": ",".join(map(str, axes)), "dtype": dtype,
            "inverse": inverse, "shift_scale": shift_scale}
    return dict(case, name=name) if name else case


def _spec(samples, nfft, hop, transposed=False, name=None):
    case = {"kind": "spectrogram", "samples": samples, "nfft": nfft, "hop": hop, "transposed": transposed}
    return dict(case, name=name) if name else case


def _real(kind, rows, n, dtype="float32", name=None):
    case = {"kind": kind, "rows": rows, "n": n, "dtype": dtype}
    return dict(case, name=name) if name else case


def listed():
    return [
        # a small batch of 1-D transforms: one call of a few microseconds, launch and host cost count
        _c2c((64, 4096), (1,), name="c2c_64x4096"),
        # many short lines (radar / communications frames), back to the time domain
        _c2c((16384, 1024), (1,), inverse=True, name="c2c_inv_16384x1024"),
        # long records: a line no longer fits one CTA
        _c2c((16, 262144), (1,), name="c2c_16x262144"),
        # a prime length
        _c2c((1000, 3001), (1,), name="c2c_1000x3001"),
        # the longest prime records of the serving stream
        _c2c((64, 65521), (1,), name="c2c_64x65521"),
        # images: the largest power of two, and a round decimal size, backward
        _c2c((2048, 2048), (0, 1), name="c2c_2048x2048"),
        _c2c((1000, 1000), (0, 1), inverse=True, name="c2c_inv_1000x1000"),
        # volumes with the zero frequency moved to the centre and 1/N, single and double precision
        _c2c((256, 256, 256), (0, 1, 2), shift_scale=True, name="c2c_256cube_shift"),
        _c2c((128, 128, 128), (0, 1, 2), dtype="complex128", shift_scale=True, name="c2c_128cube_c128_shift"),
        # a 2^22-sample signal's spectrogram
        _spec(2**22, 1024, 256, name="spectrogram_2^22"),
        # real signals: spectra of a ragged size, and signals from many short spectra
        _real("rfft", 1000, 1000, name="rfft_1000x1000"),
        _real("irfft", 16384, 1024, name="irfft_16384x1024"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng, n, max_elems):
    """A batch such that rows * n is between the smallest and the largest listed work."""
    hi = max(1, max_elems // n)
    lo = min(hi, max(1, 2**17 // n))
    return min(hi, max(1, _log_int(rng, lo, hi)))


def draw(rng):
    kind = rng.choice(["1d", "1d", "1d_ragged", "1d_ragged", "2d", "2d_ragged", "3d", "3d_ragged", "spectrogram", "rfft",
                       "irfft"])
    dtype = "complex128" if rng.random() < 0.2 else "complex64"
    cap = MAX_ELEMS if dtype == "complex64" else MAX_ELEMS // 4
    inverse = rng.random() < 0.5
    if kind == "1d":
        n = 2 ** rng.randint(6, 20)
        return _c2c((_rows(rng, n, cap), n), (1,), dtype, inverse)
    if kind == "1d_ragged":
        n = _log_int(rng, 61, 65521)
        return _c2c((_rows(rng, n, cap // 4), n), (1,), dtype, inverse)
    if kind == "2d":
        a, b = 2 ** rng.randint(6, 11), 2 ** rng.randint(6, 11)
        if rng.random() < 0.5:
            return _c2c((a, b), (0, 1), dtype, inverse)
        return _c2c((max(1, min(_rows(rng, a * b, cap), 256)), a, b), (1, 2), dtype, inverse)
    if kind == "2d_ragged":
        return _c2c((_log_int(rng, 64, 2048), _log_int(rng, 64, 2048)), (0, 1), dtype, inverse)
    if kind == "3d":
        shape = [2 ** rng.randint(5, 8) for _ in range(3)]
        while shape[0] * shape[1] * shape[2] > cap:
            shape[shape.index(max(shape))] //= 2
        return _c2c(tuple(shape), (0, 1, 2), dtype, inverse, not inverse and rng.random() < 0.5)
    if kind == "3d_ragged":
        shape = [_log_int(rng, 24, 160) for _ in range(3)]
        return _c2c(tuple(shape), (0, 1, 2), dtype, inverse, not inverse and rng.random() < 0.5)
    if kind == "spectrogram":
        nfft = 2 ** rng.randint(8, 11)
        hop = rng.choice([nfft // 4, nfft // 2, rng.randint(nfft // 4, nfft)])
        return _spec(_log_int(rng, 2**16, 2**22), nfft, hop, rng.random() < 0.3)
    rdtype = "float64" if dtype == "complex128" else "float32"
    n = 2 ** rng.randint(6, 14) if rng.random() < 0.6 else 2 * _log_int(rng, 32, 8192)
    return _real(kind, _rows(rng, n, cap if n & (n - 1) == 0 else cap // 4), n, rdtype)


def _shape(case):
    return tuple(int(s) for s in case["shape"].split("x"))


def _axes(case):
    return tuple(int(a) for a in case["axes"].split(","))


def _inputs(case, seed):
    """The call's input array: N(0,1) samples (real and imaginary parts independent); for a
    spectrogram white noise plus a few sinusoids."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = case["kind"]
    if kind == "spectrogram":
        x = torch.randn(case["samples"], dtype=torch.float32, device="cuda", generator=gen)
        t = torch.arange(case["samples"], dtype=torch.float32, device="cuda")
        for f in torch.rand(4, device="cuda", generator=gen).tolist():
            x += 3.0 * torch.sin(t * (f * math.pi))
        return x
    if kind == "rfft":
        return torch.randn(case["rows"], case["n"], dtype=getattr(torch, case["dtype"]), device="cuda", generator=gen)
    if kind == "irfft":
        # bins of a real signal: real at the zero and the Nyquist frequency
        cdt = torch.complex64 if case["dtype"] == "float32" else torch.complex128
        x = torch.randn(case["rows"], case["n"] // 2 + 1, dtype=cdt, device="cuda", generator=gen)
        x.imag[:, 0] = 0
        x.imag[:, -1] = 0
        return x
    x = torch.randn(*_shape(case), dtype=getattr(torch, case["dtype"]), device="cuda", generator=gen)
    return x * math.sqrt(2.0)


def prepare(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    args = ()
    if kind == "c2c":
        comp = FFT(x, axes=_axes(case))
        if case["shift_scale"]:
            shift, scale = tr.fftshift(x, axes=_axes(case)), tr.mul_const(x, 1.0 / x.numel())
            comp.parameter.output.connect(shift, shift.input, shifted=shift.output)
            comp.parameter.shifted.connect(scale, scale.input, result=scale.output)
        out = torch.empty_like(x)
        args = (1 if case["inverse"] else 0,)
    elif kind == "spectrogram":
        comp = spectrogram(case["samples"], case["nfft"], case["hop"], transposed=case["transposed"])
        shape = (frames(case["samples"], case["nfft"], case["hop"]), case["nfft"] // 2 + 1)
        out = torch.empty(shape[::-1] if case["transposed"] else shape, dtype=torch.float32, device="cuda")
    elif kind == "rfft":
        meta = ArrayMetadata((case["rows"], case["n"]), numpy.dtype(case["dtype"]))
        comp = RFFT(meta)
        cdt = torch.complex64 if case["dtype"] == "float32" else torch.complex128
        out = torch.empty(case["rows"], case["n"] // 2 + 1, dtype=cdt, device="cuda")
    else:
        comp = IRFFT(x)
        out = torch.empty(case["rows"], case["n"], dtype=getattr(torch, case["dtype"]), device="cuda")
    return {"call": comp.compile(x.device), "out": out, "in": x, "args": args}


def run(state):
    state["call"](None, state["out"], state["in"], *state["args"])
    return state["out"]


def work(case):
    """Each input element read once, each output element written once; 5 N log2 N
    operations a complex transform, half that for a real one."""
    kind = case["kind"]
    if kind == "c2c":
        shape, axes = _shape(case), _axes(case)
        elems = math.prod(shape)
        esz = 8 if case["dtype"] == "complex64" else 16
        return {"bytes": 2 * elems * esz, "flops": 5.0 * elems * sum(math.log2(shape[a]) for a in axes)}
    if kind == "spectrogram":
        rows, n = frames(case["samples"], case["nfft"], case["hop"]), case["nfft"]
        return {"bytes": 4 * case["samples"] + 4 * rows * (n // 2 + 1), "flops": 2.5 * rows * n * math.log2(n)}
    rows, n = case["rows"], case["n"]
    esz = 4 if case["dtype"] == "float32" else 8
    return {"bytes": esz * rows * (n + 2 * (n // 2 + 1)), "flops": 2.5 * rows * n * math.log2(n)}


def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "c2c":
        axes = _axes(case)
        y = (torch.fft.ifftn if case["inverse"] else torch.fft.fftn)(x.to(torch.complex128), dim=axes)
        if case["shift_scale"]:
            y = torch.fft.fftshift(y, dim=axes) / x.numel()
        return y
    if kind == "spectrogram":
        n, rows = case["nfft"], frames(case["samples"], case["nfft"], case["hop"])
        u = torch.arange(n, dtype=torch.float64, device=x.device)
        window = 0.5 * (1.0 - torch.cos(2.0 * math.pi * u / (n - 1)))
        y = torch.fft.rfft(x.to(torch.float64).unfold(0, n, case["hop"])[:rows] * window, dim=1).abs()
        return y.T.contiguous() if case["transposed"] else y
    if kind == "rfft":
        return torch.fft.rfft(x.to(torch.float64), dim=1)
    return torch.fft.irfft(x.to(torch.complex128), n=case["n"], dim=1)
