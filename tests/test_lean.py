"""The lean line passes (csrc/rk_lean.cuh) at the edges of their tiles, and against the
general line kernel, which RK_FLAG_NO_TMA plans keep using."""

from __future__ import annotations

import math

import numpy
import pytest

from helpers import fft_bound, normal_array, rel_l2

gpu = pytest.mark.gpu


def _run(x, out, axes, inverse=0, flags=0, connect=None):
    import torch

    from reikna_b200.fft import FFT

    comp = FFT(x, axes=axes)
    if connect:
        connect(comp, out)
    comp.compile(flags=flags)(None, out, x, inverse)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _check(got, x, axes, inverse=0):
    a = x.astype(numpy.complex128)
    ref = (numpy.fft.ifftn if inverse else numpy.fft.fftn)(a, axes=axes)
    assert rel_l2(got, ref) < fft_bound(x.dtype, math.prod(x.shape[k] for k in axes))


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("n", [2**k for k in range(4, 15)])
@pytest.mark.parametrize("rows", [1, 3, 33])
def test_contiguous_lines(rng, cuda, dtype, n, rows):
    import torch

    if rows * n > 2**18:
        rows = max(1, 2**18 // n) + 1
    x = normal_array(rng, (rows, n), dtype)
    t = torch.from_numpy(x).to(cuda)
    for inverse in (0, 1):
        _check(_run(t, torch.empty_like(t), (1,), inverse), x, (1,), inverse)
    _check(_run(t, t, (1,)), x, (1,))  # in place


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("n", [2**k for k in range(1, 11)])
@pytest.mark.parametrize("inner", [1, 5, 16, 49])
def test_strided_lines(rng, cuda, dtype, n, inner):
    import torch

    x = normal_array(rng, (3, n, inner, 2), dtype)
    t = torch.from_numpy(x).to(cuda)
    for inverse in (0, 1):
        _check(_run(t, torch.empty_like(t), (1,), inverse), x, (1,), inverse)
    _check(_run(t, t, (1,)), x, (1,))


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("n", [2**k for k in range(14, 21)])
@pytest.mark.parametrize("shape", ["rows", "strided"])
def test_two_pass_lines(rng, cuda, dtype, n, shape):
    import torch

    if shape == "strided" and n > 2**17:
        pytest.skip("covered by the row form's lengths")
    rows = 3 if n < 2**19 else 1
    s, axes = ((rows, n), (1,)) if shape == "rows" else ((n, 3), (0,))
    x = normal_array(rng, s, dtype)
    t = torch.from_numpy(x).to(cuda)
    for inverse in (0, 1):
        _check(_run(t, torch.empty_like(t), axes, inverse), x, axes, inverse)
    _check(_run(t, t, axes), x, axes)


@gpu
@pytest.mark.parametrize("rows", [1, 4, 5])
def test_few_two_pass_lines(rng, cuda, rows):
    """complex128 lines of 2^18 points on both sides of the first pass's choice of plan."""
    import torch

    x = normal_array(rng, (rows, 2**18), numpy.complex128)
    t = torch.from_numpy(x).to(cuda)
    for inverse in (0, 1):
        _check(_run(t, torch.empty_like(t), (1,), inverse), x, (1,), inverse)
    _check(_run(t, t, (1,)), x, (1,))


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("shape,axes", [((6, 64, 32), (0,)), ((5, 64, 33), (1,)), ((4, 5, 256), (2,)), ((16, 8, 7), (0, 1)),
                                        ((32, 32, 32), (0, 1, 2)), ((2, 3, 4, 5, 16), (1, 4))])
def test_output_shift_and_scale(rng, cuda, dtype, shape, axes):
    """fftshift on power-of-two axes (half the axis: a register swap), on other dims of the
    array and on odd ones, with a complex scale."""
    import torch

    from reikna_b200 import transformations as tr

    x = normal_array(rng, shape, dtype)
    t = torch.from_numpy(x).to(cuda)
    every = tuple(range(len(shape)))
    factor = 0.25 - 0.5j

    def connect(comp, out):
        sh, sc = tr.fftshift(out, axes=every), tr.mul_const(out, out.cpu().numpy().dtype.type(factor))
        comp.parameter.output.connect(sh, sh.input, shifted=sh.output)
        comp.parameter.shifted.connect(sc, sc.input, result=sc.output)

    got = _run(t, torch.empty_like(t), axes, connect=connect)
    ref = numpy.fft.fftshift(numpy.fft.fftn(x.astype(numpy.complex128), axes=axes), axes=every) * factor
    assert rel_l2(got, ref) < fft_bound(dtype, math.prod(shape[k] for k in axes))


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("perm", [(0, 1, 2), (2, 1, 0), (1, 0, 2), (0, 2, 1)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_any_order_as_the_general_path(rng, cuda, dtype, perm, axis):
    """Input and output views with permuted dims and gaps between rows: the lean route and
    the general one agree with each other and with numpy."""
    import torch

    from reikna_b200 import _native as N

    shape = (32, 64, 16)
    base = normal_array(rng, tuple(2 * shape[p] if k == 0 else shape[p] for k, p in enumerate(perm)), dtype)
    inv = tuple(numpy.argsort(perm))
    t = torch.from_numpy(base).to(cuda)[::2].permute(inv)
    x = base[::2].transpose(inv)
    out = torch.empty_strided(t.shape, t.stride(), dtype=t.dtype, device=cuda)
    _check(_run(t, out, (axis,)), x, (axis,))
    lean = out.cpu().numpy()
    general = _run(t, torch.empty_strided(t.shape, t.stride(), dtype=t.dtype, device=cuda), (axis,), flags=N.FLAG_NO_TMA)
    assert rel_l2(lean, general) < 2 * fft_bound(dtype, shape[axis])


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("n", [6, 9, 15, 17, 31, 33, 63, 65, 100, 129, 255, 257, 500, 513, 1000, 1025, 2047, 2049, 4095, 4097, 8191])
@pytest.mark.parametrize("form", ["rows", "columns"])
def test_bluestein_lines(rng, cuda, dtype, n, form):
    """Lengths at both ends of each padded length M, whole-line and three-pass, along
    contiguous and strided axes."""
    import torch

    shape, axes = ((3 if n > 2000 else 37, n), (1,)) if form == "rows" else ((2, n, 5), (1,))
    x = normal_array(rng, shape, dtype)
    t = torch.from_numpy(x).to(cuda)
    for inverse in (0, 1):
        _check(_run(t, torch.empty_like(t), axes, inverse), x, axes, inverse)
    _check(_run(t, t, axes), x, axes)


@gpu
@pytest.mark.parametrize("dtype,n,rows", [(numpy.complex64, 16001, 3), (numpy.complex64, 65521, 2), (numpy.complex64, 131101, 2),
                                          (numpy.complex64, 300007, 1), (numpy.complex64, 600011, 1),
                                          (numpy.complex128, 16385, 2), (numpy.complex128, 70001, 1)])
def test_long_bluestein_lines(rng, cuda, dtype, n, rows):
    import torch

    x = normal_array(rng, (rows, n), dtype)
    t = torch.from_numpy(x).to(cuda)
    for inverse in (0, 1):
        _check(_run(t, torch.empty_like(t), (1,), inverse), x, (1,), inverse)
    _check(_run(t, t, (1,)), x, (1,))


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("shape,axes", [((33, 20), (0, 1)), ((3, 1001), (1,)), ((1500, 6), (0,)), ((2, 9001), (1,)), ((5, 6, 7), (0, 1, 2))])
def test_bluestein_shift_and_scale(rng, cuda, dtype, shape, axes):
    import torch

    from reikna_b200 import transformations as tr

    x = normal_array(rng, shape, dtype)
    t = torch.from_numpy(x).to(cuda)
    every = tuple(range(len(shape)))
    factor = 0.25 - 0.5j

    def connect(comp, out):
        sc, sh = tr.mul_const(out, out.cpu().numpy().dtype.type(factor)), tr.fftshift(out, axes=every)
        comp.parameter.output.connect(sc, sc.input, scaled=sc.output)
        comp.parameter.scaled.connect(sh, sh.input, result=sh.output)

    for inverse in (0, 1):
        got = _run(t, torch.empty_like(t), axes, inverse, connect=connect)
        ref = (numpy.fft.ifftn if inverse else numpy.fft.fftn)(x.astype(numpy.complex128), axes=axes)
        ref = numpy.fft.fftshift(ref, axes=every) * factor
        assert rel_l2(got, ref) < fft_bound(dtype, math.prod(shape[k] for k in axes))


@gpu
@pytest.mark.parametrize("dtype", [numpy.float32, numpy.float64])
@pytest.mark.parametrize("n", [2**k for k in range(5, 15)])
@pytest.mark.parametrize("rows", [1, 37])
def test_real_lines(rng, cuda, dtype, n, rows):
    """Half lengths inside a warp and beyond, full and partial tiles, odd starting samples."""
    import torch

    from reikna_b200.core import ArrayMetadata
    from reikna_b200.fft import IRFFT, RFFT

    base = torch.from_numpy(rng.standard_normal(rows * n + 1).astype(dtype)).to(cuda)
    cdt = torch.complex64 if dtype == numpy.float32 else torch.complex128
    bound = fft_bound(numpy.complex64 if dtype == numpy.float32 else numpy.complex128, n)
    for start in (0, 1):
        t = base[start:start + rows * n].view(rows, n)
        ref = numpy.fft.rfft(t.cpu().numpy().astype(numpy.float64), axis=1)
        for last in (False, True):
            out = torch.full((rows, n // 2 + (0 if last else 1)), float("nan"), dtype=cdt, device=cuda)
            call = RFFT(ArrayMetadata((rows, n), dtype), dont_store_last=last).compile()
            if start and dtype == numpy.float64 and n > 8192:
                # beyond the one-pass lengths the real array is read as complex pairs
                with pytest.raises(ValueError, match="boundary"):
                    call(None, out, t)
                continue
            call(None, out, t)
            torch.cuda.synchronize()
            assert rel_l2(out.cpu().numpy(), ref[:, :out.shape[1]]) < bound
    spec = torch.from_numpy(ref).to(cdt).to(cuda)
    back = torch.empty(rows, n, dtype=t.dtype, device=cuda)
    IRFFT(spec).compile()(None, back, spec)
    torch.cuda.synchronize()
    assert rel_l2(back.cpu().numpy(), numpy.fft.irfft(spec.cpu().numpy().astype(numpy.complex128), n=n, axis=1)) < bound


@gpu
@pytest.mark.parametrize("nfft", [2**k for k in range(5, 13)])
@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("hop", ["quarter", "odd"])
def test_spectrogram_lines(rng, cuda, nfft, transposed, hop):
    import torch

    from reikna_b200.spectrogram import frames, spectrogram

    hop = nfft // 4 if hop == "quarter" else nfft // 3 | 1
    n = nfft + 52 * hop + 3
    x = rng.standard_normal(n).astype(numpy.float32)
    rows, bins = frames(n, nfft, hop), nfft // 2 + 1
    out = torch.full((bins, rows) if transposed else (rows, bins), float("nan"), dtype=torch.float32, device=cuda)
    spectrogram(n, nfft, hop, transposed=transposed).compile()(None, out, torch.from_numpy(x).to(cuda))
    torch.cuda.synchronize()
    win = 0.5 * (1.0 - numpy.cos(2.0 * numpy.pi * numpy.arange(nfft) / (nfft - 1)))
    ref = numpy.abs(numpy.fft.rfft(numpy.stack([x[k * hop:k * hop + nfft] * win for k in range(rows)]).astype(numpy.float64), axis=1))
    assert rel_l2(out.cpu().numpy(), ref.T if transposed else ref) < fft_bound(numpy.complex64, nfft)


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("shape", [(3, 64, 64), (2, 128, 128), (3, 256, 256), (5, 128, 128, 2), (2, 3, 256, 256)])
@pytest.mark.parametrize("shift", [False, True])
def test_plane_as_rows_and_columns(rng, cuda, dtype, shape, shift):
    """Planes whose columns are transformed in place in the output, and through a
    temporary where the output is remapped; out of place, in place and strided."""
    import torch

    from reikna_b200 import transformations as tr

    axes = (1, 2) if shape[-1] == 2 else (len(shape) - 2, len(shape) - 1)
    x = normal_array(rng, shape, dtype)
    t = torch.from_numpy(x).to(cuda)

    def connect(comp, out):
        sh = tr.fftshift(out, axes=axes)
        comp.parameter.output.connect(sh, sh.input, shifted=sh.output)

    for inverse in (0, 1):
        ref = (numpy.fft.ifftn if inverse else numpy.fft.fftn)(x.astype(numpy.complex128), axes=axes)
        if shift:
            ref = numpy.fft.fftshift(ref, axes=axes)
        for out in (torch.empty_like(t), t.clone()):
            src = t if out.data_ptr() != t.data_ptr() else out
            assert rel_l2(_run(src, out, axes, inverse, connect=connect if shift else None), ref) < fft_bound(dtype, shape[axes[0]] * shape[axes[1]])
        same = t.clone()
        assert rel_l2(_run(same, same, axes, inverse, connect=connect if shift else None), ref) < fft_bound(dtype, shape[axes[0]] * shape[axes[1]])


MIXED = [6, 10, 12, 14, 15, 18, 21, 22, 24, 26, 33, 35, 36, 39, 45, 48, 49, 55, 60, 65, 66, 77, 78, 90, 91, 96, 99, 100, 104, 105, 110, 112,
         117, 121, 130, 132, 143, 144, 154, 156, 169, 180, 182, 195, 196, 210, 225, 240, 243, 286, 343, 360, 385, 500, 625, 720, 729, 1000,
         1001, 1080, 1155, 1331, 1536, 1920, 2197, 2401, 3000, 3003, 3072, 4000, 4095, 5000, 6000, 6561, 7350, 8000, 8085, 8190]


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("form", ["rows", "columns"])
@pytest.mark.parametrize("n", MIXED)
def test_mixed_radix_lines(rng, cuda, dtype, form, n):
    """Every radix, two to four stages, whole and partial tiles; out of place, in place and
    with the output shifted by half an odd or even length."""
    import torch

    from reikna_b200 import transformations as tr

    rows = 1 if n > 4000 else 3 if n > 700 else 67
    shape, axes = ((rows, n), (1,)) if form == "rows" else ((2, n, 5 if n > 700 else 21), (1,))
    x = normal_array(rng, shape, dtype)
    t = torch.from_numpy(x).to(cuda)
    for inverse in (0, 1):
        _check(_run(t, torch.empty_like(t), axes, inverse), x, axes, inverse)

    def connect(comp, out):
        sh = tr.fftshift(out, axes=axes)
        comp.parameter.output.connect(sh, sh.input, shifted=sh.output)

    got = _run(t, torch.empty_like(t), axes, connect=connect)
    ref = numpy.fft.fftshift(numpy.fft.fftn(x.astype(numpy.complex128), axes=axes), axes=axes)
    assert rel_l2(got, ref) < fft_bound(dtype, n)
    _check(_run(t, t, axes), x, axes)


def test_mixed_radix_is_chosen_for_small_factors():
    from reikna_b200 import _native as N

    for n, note in ((1000, "mixed"), (97, "bluestein-fused"), (7350, "mixed"), (2 * 17, "bluestein-fused"), (1024, "single")):
        assert N.describe(N.desc(N.FMT_C64, (5, n), (1,)))["passes"][0]["note"] == note
        if note == "mixed":
            assert N.describe(N.desc(N.FMT_C64, (5, n), (1,), N.FLAG_BATCHABLE))["passes"][0]["note"] == "bluestein-fused"


@gpu
@pytest.mark.parametrize("dtype", [numpy.float32, numpy.float64])
@pytest.mark.parametrize("half", [6, 9, 17, 30, 31, 33, 97, 100, 121, 255, 500, 513, 625, 1001, 1023, 1500, 2049, 3000, 4095, 4097, 6000, 8191, 8193])
@pytest.mark.parametrize("rows", [1, 23])
def test_real_lines_of_any_length(rng, cuda, dtype, half, rows):
    """RFFT and IRFFT in one mixed-radix or Bluestein pass: even and odd half lengths, both
    ends of the padded lengths, and the first lengths beyond (the multi-kernel route)."""
    import torch

    from reikna_b200.core import ArrayMetadata
    from reikna_b200.fft import IRFFT, RFFT

    n = 2 * half
    x = rng.standard_normal((rows, n)).astype(dtype)
    t = torch.from_numpy(x).to(cuda)
    cdt = torch.complex64 if dtype == numpy.float32 else torch.complex128
    bound = fft_bound(numpy.complex64 if dtype == numpy.float32 else numpy.complex128, n)
    ref = numpy.fft.rfft(x.astype(numpy.float64), axis=1)
    for last in (False, True):
        out = torch.full((rows, half + (0 if last else 1)), float("nan"), dtype=cdt, device=cuda)
        RFFT(ArrayMetadata((rows, n), dtype), dont_store_last=last).compile()(None, out, t)
        torch.cuda.synchronize()
        assert rel_l2(out.cpu().numpy(), ref[:, :out.shape[1]]) < bound
    bins = ref.astype(numpy.complex64 if dtype == numpy.float32 else numpy.complex128)
    bins[:, 0] += 3j   # ignored, as numpy does
    bins[:, -1] -= 2j
    spec = torch.from_numpy(bins).to(cuda)
    back = torch.full((rows, n), float("nan"), dtype=t.dtype, device=cuda)
    IRFFT(spec).compile()(None, back, spec)
    torch.cuda.synchronize()
    assert rel_l2(back.cpu().numpy(), numpy.fft.irfft(bins.astype(numpy.complex128), n=n, axis=1)) < bound


@gpu
def test_real_plans_of_any_length_take_scales(rng, cuda):
    """Edge scales of one-pass real plans (through the C-ABI) in their bodies."""
    import torch

    from reikna_b200 import _native as N

    for half in (500, 97):
        c = 0.5 + 0.25j
        x = torch.from_numpy(rng.standard_normal((5, 2 * half)).astype(numpy.float32)).to(cuda)
        d = N.desc(N.FMT_C64, (5, half), (1,), N.FLAG_REAL_POST | N.FLAG_REAL_ANY)
        d.input = N.edge(N.FMT_C64, (5, half))
        d.output = N.edge(N.FMT_C64, (5, half + 1))
        d.output.scale_re, d.output.scale_im = c.real, c.imag
        out = torch.empty((5, half + 1), dtype=torch.complex64, device=cuda)
        N.Plan(d).execute([out.data_ptr()], [x.data_ptr()], stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert rel_l2(out.cpu().numpy(), numpy.fft.rfft(x.cpu().numpy().astype(numpy.float64)) * c) < fft_bound(numpy.complex64, 2 * half)


@gpu
def test_dependent_launches_in_graphs_and_streams(rng, cuda):
    """Chains of early-placed launches behind copies, forks and joins, captured and not: each
    result is that of the calls one by one."""
    import torch

    from reikna_b200.fft import FFT

    src = torch.from_numpy(normal_array(rng, (24, 96, 250), numpy.complex64)).to(cuda)
    a, b, c = torch.empty_like(src), torch.empty_like(src), torch.empty_like(src)
    both, last = FFT(src, axes=(1, 2)).compile(), FFT(src, axes=(0,)).compile()
    side = torch.cuda.Stream()

    def chain():
        a.copy_(src)
        both(None, b, a, 0)              # rows, columns
        fork = torch.cuda.Event()
        fork.record()
        side.wait_event(fork)
        with torch.cuda.stream(side):
            last(None, c, b, 0)          # reads b beside the next call's reads
        both(None, a, b, 1)              # back to src
        join = torch.cuda.Event()
        join.record(side)
        torch.cuda.current_stream().wait_event(join)
        c.mul_(2.0)
        b.zero_()

    ref = 2 * numpy.fft.fftn(src.cpu().numpy().astype(numpy.complex128))
    for _ in range(3):
        chain()
    torch.cuda.synchronize()
    assert rel_l2(c.cpu().numpy(), ref) < fft_bound(numpy.complex64, src.numel())
    assert rel_l2(a.cpu().numpy(), src.cpu().numpy()) < 2 * fft_bound(numpy.complex64, 96 * 250)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for scale in (1.0, 3.0):
        src.mul_(scale)
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        ref = 2 * numpy.fft.fftn(src.cpu().numpy().astype(numpy.complex128))
        assert rel_l2(c.cpu().numpy(), ref) < fft_bound(numpy.complex64, src.numel())
        assert rel_l2(a.cpu().numpy(), src.cpu().numpy()) < 2 * fft_bound(numpy.complex64, 96 * 250)


@gpu
@pytest.mark.parametrize("dtype", [numpy.float32, numpy.float64])
@pytest.mark.parametrize("half", [9, 13, 25, 30, 50, 100])
@pytest.mark.parametrize("rows", [81, 4099])
def test_many_short_real_lines(rng, cuda, dtype, half, rows):
    """Tiles of many lines, whose bin pairs are spread over the CTA's threads; whole tiles
    and a partial last one, with and without the Nyquist bin."""
    import torch

    from reikna_b200.core import ArrayMetadata
    from reikna_b200.fft import IRFFT, RFFT

    x = rng.standard_normal((rows, 2 * half)).astype(dtype)
    t = torch.from_numpy(x).to(cuda)
    cdt = torch.complex64 if dtype == numpy.float32 else torch.complex128
    bound = fft_bound(numpy.complex64 if dtype == numpy.float32 else numpy.complex128, 2 * half)
    ref = numpy.fft.rfft(x.astype(numpy.float64), axis=1)
    for last in (False, True):
        out = torch.full((rows, half + (0 if last else 1)), float("nan"), dtype=cdt, device=cuda)
        RFFT(ArrayMetadata((rows, 2 * half), dtype), dont_store_last=last).compile()(None, out, t)
        torch.cuda.synchronize()
        assert rel_l2(out.cpu().numpy(), ref[:, :out.shape[1]]) < bound
    spec = torch.from_numpy(ref).to(cdt).to(cuda)
    back = torch.full((rows, 2 * half), float("nan"), dtype=t.dtype, device=cuda)
    IRFFT(spec).compile()(None, back, spec)
    torch.cuda.synchronize()
    assert rel_l2(back.cpu().numpy(), x) < 2 * bound
