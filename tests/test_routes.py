"""Which calls the lean passes take over, where that could go wrong: passes after a
clustered plane, members of a batch, installed kernels, overlapping arrays, planes split
into rows and columns."""

from __future__ import annotations

import math

import numpy
import pytest

from helpers import fft_bound, normal_array, rel_l2

gpu = pytest.mark.gpu


def _rel(got, ref) -> float:
    import torch

    return float(torch.linalg.norm((got - ref).flatten()) / torch.linalg.norm(ref.flatten()))


@gpu
@pytest.mark.parametrize("shape,dtype,notes", [
    ((257, 128, 128), numpy.complex128, ["plane", "bluestein-fused"]),
    ((1031, 256, 256), numpy.complex64, ["plane", "bluestein-A1", "bluestein-B1", "bluestein-A2", "bluestein-B2"]),
])
def test_bluestein_axis_after_a_clustered_plane(cuda, shape, dtype, notes):
    """Bodies that only the lean kernels have (1024 complex128 points a strided line, the
    three-pass form) behind planes of more than 64 MB, which keep the clustered kernel."""
    import torch

    from reikna_b200.core import ArrayMetadata
    from reikna_b200.fft import FFT

    comp = FFT(ArrayMetadata(shape, dtype), axes=(0, 1, 2))
    assert [p["note"] for p in comp.describe(0)["passes"]] == notes
    call = comp.compile()
    torch.manual_seed(3)
    x = torch.randn(shape, dtype=torch.complex64 if dtype == numpy.complex64 else torch.complex128, device=cuda)
    out = torch.empty_like(x)
    for inverse in (0, 1):
        call(None, out, x, inverse)
        ref = (torch.fft.ifftn if inverse else torch.fft.fftn)(x.to(torch.complex128))
        assert _rel(out, ref) < fft_bound(dtype, math.prod(shape))


@gpu
@pytest.mark.parametrize("shape,axis", [((3, 16001), 1), ((5, 1000), 1), ((100, 6), 0), ((7, 3001), 1)])
def test_batch_of_plans_without_the_batchable_flag(rng, cuda, shape, axis):
    """Members whose own passes are lean-only (three-pass Bluestein, mixed radix) and one
    whose pass has a tile body, beside a plain member."""
    import torch

    from reikna_b200 import _native as N

    sizes = [(shape, axis), ((16, 512), 1)]
    xs = [normal_array(rng, s, numpy.complex64) for s, _ in sizes]
    ts = [torch.from_numpy(x).to(cuda) for x in xs]
    outs = [torch.empty_like(t) for t in ts]
    batch = N.Batch([N.Plan(N.desc(N.FMT_C64, s, (a,))) for s, a in sizes])
    for inverse in (0, 1):
        batch.execute([([o.data_ptr()], [t.data_ptr()], inverse, ()) for o, t in zip(outs, ts)],
                      stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        for x, o, (s, a) in zip(xs, outs, sizes):
            ref = (numpy.fft.ifft if inverse else numpy.fft.fft)(x.astype(numpy.complex128), axis=a)
            assert rel_l2(o.cpu().numpy(), ref) < fft_bound(numpy.complex64, s[a])
    assert N.device_status(clear=True) == 0
    batch.close()


@gpu
def test_batch_refuses_one_pass_real_members(cuda):
    from reikna_b200 import _native as N

    d = N.desc(N.FMT_C64, (5, 97), (1,), N.FLAG_REAL_POST | N.FLAG_REAL_ANY)
    d.input, d.output = N.edge(N.FMT_C64, (5, 97)), N.edge(N.FMT_C64, (5, 98))
    with pytest.raises(NotImplementedError):
        N.Batch([N.Plan(d)])


MARK = """#include "rk_params.h"
extern "C" __global__ void mark(const rk::PassParams p) {
    if (blockIdx.x == 0 && threadIdx.x == 0) ((float2*)p.st.ptr)[0] = make_float2(42.0f, 0.0f);
}
"""


@gpu
def test_an_installed_kernel_runs_in_every_call(cuda):
    """rk_fft_call and rk_fft_execute both leave the prepared lean launches for it."""
    import torch

    from reikna_b200 import _native as N
    from reikna_b200 import _rtc

    plan = N.Plan(N.desc(N.FMT_C64, (3, 64, 5), (1,)))
    x = torch.ones((3, 64, 5), dtype=torch.complex64, device=cuda)
    stream = torch.cuda.current_stream().cuda_stream
    out = torch.zeros_like(x)
    plan.call(out.data_ptr(), x.data_ptr(), 0, stream)
    torch.cuda.synchronize()
    assert out[0, 0, 0] == 64
    plan.set_pass_kernel(0, _rtc.compile_cubin(MARK), "mark")
    for run in (lambda: plan.call(out.data_ptr(), x.data_ptr(), 0, stream),
                lambda: plan.execute([out.data_ptr()], [x.data_ptr()], stream=stream)):
        out.zero_()
        run()
        torch.cuda.synchronize()
        assert out[0, 0, 0] == 42 and torch.count_nonzero(out) == 1


@gpu
@pytest.mark.parametrize("shape,axis,passes", [((5, 1000), 1, 1), ((3, 16001), 1, 4), ((64, 1024), 1, 1), ((4, 1024, 64), 1, 1),
                                               ((3, 300, 5), 1, 1)])
def test_passes_without_a_general_kernel_take_no_installed_one(cuda, shape, axis, passes):
    """Mixed-radix and three-pass Bluestein passes, and lines the TMA-fed kernel would run;
    their launch shapes are those of the kernels that do run."""
    from reikna_b200 import _native as N
    from reikna_b200 import _rtc

    plan = N.Plan(N.desc(N.FMT_C64, shape, (axis,)))
    info = plan.pass_info()
    assert len(info) == passes and all(p["nt"] > 0 and p["nl"] > 0 for p in info)
    cubin = _rtc.compile_cubin(MARK)
    for i in range(passes):
        with pytest.raises(NotImplementedError, match="plain line passes"):
            plan.set_pass_kernel(i, cubin, "mark")


@gpu
@pytest.mark.parametrize("dtype", [numpy.float32, numpy.float64])
@pytest.mark.parametrize("n", [200, 194, 256, 3000])
@pytest.mark.parametrize("start", [0, 8, 600, 6000])
def test_real_transforms_of_overlapping_arrays(rng, cuda, dtype, n, start):
    """RFFT and IRFFT (mixed-radix, Bluestein and power-of-two bodies) whose arrays share
    memory, the second one `start` samples behind the first or in front of it."""
    import torch

    from reikna_b200.core import ArrayMetadata
    from reikna_b200.fft import IRFFT, RFFT

    rows = 2**18 // n
    cdt = torch.complex64 if dtype == numpy.float32 else torch.complex128
    bound = fft_bound(numpy.complex64 if dtype == numpy.float32 else numpy.complex128, n)
    x = rng.standard_normal((rows, n)).astype(dtype)
    spec = numpy.fft.rfft(x.astype(numpy.float64), axis=1)
    bins = rows * (n // 2 + 1)
    forward = RFFT(ArrayMetadata((rows, n), dtype)).compile()
    inverse = IRFFT(ArrayMetadata((rows, n // 2 + 1), spec.astype(numpy.complex64).dtype if dtype == numpy.float32 else spec.dtype)).compile()
    for behind in (False, True):
        buf = torch.zeros(rows * n + 2 * rows + start, dtype=torch.float32 if dtype == numpy.float32 else torch.float64, device=cuda)
        a, b = (0, start) if behind else (start, 0)
        real = buf[a:a + rows * n].view(rows, n)
        half = buf[b:b + 2 * bins].view(cdt).view(rows, n // 2 + 1)
        real.copy_(torch.from_numpy(x))
        forward(None, half, real)
        torch.cuda.synchronize()
        assert rel_l2(half.cpu().numpy(), spec) < bound
        half.copy_(torch.from_numpy(spec).to(cdt))
        inverse(None, real, half)
        torch.cuda.synchronize()
        assert rel_l2(real.cpu().numpy(), x) < bound


@gpu
@pytest.mark.parametrize("dtype,n,cols", [(numpy.complex64, 1500, 40), (numpy.complex128, 257, 40), (numpy.complex128, 1500, 24)])
def test_long_strided_lines_shifted_within_their_array(rng, cuda, dtype, n, cols):
    """Lean passes in place of several general ones, which went through temporaries."""
    import torch

    from reikna_b200.fft import FFT

    x = normal_array(rng, (n, cols), dtype)
    ref = numpy.fft.fft(x.astype(numpy.complex128), axis=0)
    for a, b in ((0, 1), (1, 0)):
        buf = torch.zeros((n + 1, cols), dtype=torch.complex64 if dtype == numpy.complex64 else torch.complex128, device=cuda)
        src, dst = buf[a:a + n], buf[b:b + n]
        src.copy_(torch.from_numpy(x))
        FFT(src, axes=(0,)).compile()(None, dst, src)
        torch.cuda.synchronize()
        assert rel_l2(dst.cpu().numpy(), ref) < fft_bound(dtype, n)


@gpu
def test_first_overlapping_call_inside_a_capture(rng, cuda):
    """The private copy is allocated by the call that needs it first, also where a stream
    captures that call."""
    import torch

    from reikna_b200.core import ArrayMetadata
    from reikna_b200.fft import RFFT

    rows, n = 300, 200
    x = rng.standard_normal((rows, n)).astype(numpy.float32)
    buf = torch.zeros(rows * (n + 2), dtype=torch.float32, device=cuda)
    real, half = buf[:rows * n].view(rows, n), buf.view(torch.complex64).view(rows, n // 2 + 1)
    call = RFFT(ArrayMetadata((rows, n), numpy.float32)).compile()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(None, half, real)
    for _ in range(2):
        real.copy_(torch.from_numpy(x))
        graph.replay()
        torch.cuda.synchronize()
        assert rel_l2(half.cpu().numpy(), numpy.fft.rfft(x.astype(numpy.float64), axis=1)) < fft_bound(numpy.complex64, n)


def test_choices_tuned_on_earlier_kernels_are_tuned_again():
    import hashlib

    from reikna_b200 import _native as N
    from reikna_b200 import autotune, batch
    from reikna_b200.core import ArrayMetadata
    from reikna_b200.fft import FFT

    comp = FFT(ArrayMetadata((1000, 1000), numpy.complex64))
    desc = bytes(comp.native_descriptor(0)[0])
    assert autotune._key(comp, False) != hashlib.sha256(b"fft-tune-1" + desc).hexdigest()[:32]
    assert batch._desc_key([comp.native_descriptor(0)[0]]) != hashlib.sha256(b"3" + desc).hexdigest()[:32]
    # the flag those choices held for most plans turns the kernels of today off
    assert [p["note"] for p in comp.describe(0)["passes"]] == ["mixed", "mixed"]
    assert "mixed" not in [p["note"] for p in comp.describe(N.FLAG_NO_TMA)["passes"]]


@gpu
@pytest.mark.parametrize("shape,dtype,launches", [
    ((64, 64, 64), numpy.complex64, 2), ((65, 64, 64), numpy.complex64, 1), ((148, 64, 64), numpy.complex64, 1),
    ((149, 64, 64), numpy.complex64, 2), ((1152, 64, 64), numpy.complex64, 2), ((1153, 64, 64), numpy.complex64, 1),
    ((1280, 128, 128), numpy.complex64, 2), ((1281, 128, 128), numpy.complex64, 1), ((100, 64, 64), numpy.complex128, 2)])
def test_planes_on_both_sides_of_the_split(cuda, shape, dtype, launches):
    """Planes as one launch or as rows and columns, where the choice changes."""
    import torch

    from reikna_b200.core import ArrayMetadata
    from reikna_b200.fft import FFT

    call = FFT(ArrayMetadata(shape, dtype), axes=(1, 2)).compile()
    assert call.launches == launches
    torch.manual_seed(5)
    x = torch.randn(shape, dtype=torch.complex64 if dtype == numpy.complex64 else torch.complex128, device=cuda)
    out = torch.empty_like(x)
    for inverse in (0, 1):
        call(None, out, x, inverse)
        ref = (torch.fft.ifftn if inverse else torch.fft.fftn)(x.to(torch.complex128), dim=(1, 2))
        assert _rel(out, ref) < fft_bound(dtype, shape[1] * shape[2])


@gpu
@pytest.mark.parametrize("dtype", [numpy.complex64, numpy.complex128])
@pytest.mark.parametrize("shape,axes", [((6, 128, 128), (0, 1, 2)), ((16, 128, 128), (0, 1, 2)), ((5, 64, 64), (0, 1, 2)),
                                        ((2, 17, 64, 64), (1, 2, 3)), ((5, 256, 256), (0, 1, 2))])
@pytest.mark.parametrize("shift", [False, True])
@pytest.mark.parametrize("views", [False, True])
def test_planes_split_through_a_temporary(rng, cuda, dtype, shape, axes, shift, views):
    """Planes with another axis behind them: rows and columns through the plan's temporary,
    then power-of-two, mixed-radix or Bluestein lines; out of place, in place and on strided
    views, with and without a shift of every transformed axis on the output."""
    import torch

    from reikna_b200 import transformations as tr
    from reikna_b200.fft import FFT

    if shape[-1] == 256 and dtype == numpy.complex128:
        pytest.skip("no plane pass of this size and type")
    x = normal_array(rng, shape, dtype)
    base = torch.zeros((2 * shape[0],) + shape[1:], dtype=torch.from_numpy(x).dtype, device=cuda)
    t = base[1::2] if views else torch.empty(shape, dtype=base.dtype, device=cuda)
    t.copy_(torch.from_numpy(x))
    out = torch.empty_like(base)[::2] if views else torch.empty_like(t)
    for inverse in (0, 1):
        comp = FFT(t, axes=axes)
        if shift:
            sh = tr.fftshift(out, axes=axes)
            comp.parameter.output.connect(sh, sh.input, shifted=sh.output)
        call = comp.compile()
        assert comp.describe(0)["passes"][0]["note"] == "plane" and call.launches == 3
        call(None, out, t, inverse)
        torch.cuda.synchronize()
        ref = (numpy.fft.ifftn if inverse else numpy.fft.fftn)(x.astype(numpy.complex128), axes=axes)
        if shift:
            ref = numpy.fft.fftshift(ref, axes=axes)
        bound = fft_bound(dtype, math.prod(shape[a] for a in axes))
        assert rel_l2(out.cpu().numpy(), ref) < bound
        same = t.clone() if not views else out
        if views:
            same.copy_(t)
        call(None, same, same, inverse)
        torch.cuda.synchronize()
        assert rel_l2(same.cpu().numpy(), ref) < bound
    assert torch.equal(t.cpu(), torch.from_numpy(x))


@pytest.mark.parametrize("form", ["rows", "columns"])
def test_lengths_of_the_mixed_radix_tests_take_that_kernel(form):
    """The lengths test_mixed_radix_lines runs are mixed-radix plans, but for odd ones of four
    stages with a 13, and complex128 ones whose tile does not fit shared memory."""
    from reikna_b200 import _native as N
    from test_lean import MIXED

    for fmt in (N.FMT_C64, N.FMT_C128):
        for n in MIXED:
            rows = 1 if n > 4000 else 3 if n > 700 else 67
            shape, axis = ((rows, n), 1) if form == "rows" else ((2, n, 5 if n > 700 else 21), 1)
            note = N.describe(N.desc(fmt, shape, (axis,)))["passes"][0]["note"]
            expected = n not in (3003, 4095) and (fmt == N.FMT_C64 or n <= 6000)
            assert (note == "mixed") == expected, (fmt, n, note)


@pytest.mark.parametrize("rows,real,flags,lengths", [(64, True, 0, [128, 128]), (65, True, 0, [64, 256]), (65, False, 0, [128, 128]),
                                                     (65, False, 16, [64, 256]), (64, False, 16, [128, 128])])
def test_long_complex128_lines_split_by_the_kernel_that_reads_them(rows, real, flags, lengths):
    from reikna_b200 import _native as N

    d = N.desc(N.FMT_C128, (rows, 2**14), (1,), flags)
    if real:
        d.input = N.edge(N.FMT_F64, (rows, 2**14))
    assert [p["L"] for p in N.describe(d)["passes"]] == lengths


@gpu
def test_long_real_float64_lines_beyond_l2(cuda):
    import torch

    from reikna_b200 import _native as N

    n = 2**14
    d = N.desc(N.FMT_C128, (67, n), (1,))
    d.input = N.edge(N.FMT_F64, (67, n))
    torch.manual_seed(4)
    x = torch.randn((67, n), dtype=torch.float64, device=cuda)
    out = torch.empty((67, n), dtype=torch.complex128, device=cuda)
    plan = N.Plan(d)
    for inverse in (0, 1):
        plan.execute([out.data_ptr()], [x.data_ptr()], inverse=inverse, stream=torch.cuda.current_stream().cuda_stream)
        ref = (torch.fft.ifft if inverse else torch.fft.fft)(x, dim=1)
        assert _rel(out, ref) < fft_bound(numpy.complex128, n)


STALE = """
import torch
from reikna_b200 import _native as N
x = torch.ones((4, 64), dtype=torch.complex64, device="cuda")
out = torch.empty_like(x)
lean, general = (N.Plan(N.desc(N.FMT_C64, (4, 64), (1,), f)) for f in (0, N.FLAG_NO_TMA))
side = torch.cuda.Stream()
torch.cuda.synchronize()
refused = 0
with torch.cuda.stream(side):
    graph = torch.cuda.CUDAGraph()
    graph.capture_begin(capture_error_mode="global")
    try:
        torch.cuda.synchronize()      # not permitted while a stream captures: ends the capture
    except RuntimeError:
        pass
    for run in (lambda: lean.call(out.data_ptr(), x.data_ptr(), 0, side.cuda_stream),
                lambda: lean.execute([out.data_ptr()], [x.data_ptr()], stream=side.cuda_stream)):
        try:
            run()
        except N.NativeError:
            refused += 1
    try:
        graph.capture_end()
    except RuntimeError:
        pass
assert refused == 2
out.zero_()
stream = torch.cuda.current_stream().cuda_stream
general.execute([out.data_ptr()], [x.data_ptr()], stream=stream)
torch.cuda.synchronize()
assert out[0, 0] == 64 and out[0, 1] == 0
print("done")
"""


@gpu
def test_a_refused_launch_leaves_no_error_behind(cuda):
    """A launch the runtime refuses is that call's error, not the next call's."""
    import subprocess
    import sys
    from pathlib import Path

    root = Path(__file__).resolve().parent.parent
    res = subprocess.run([sys.executable, "-c", STALE], cwd=root, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "done" in res.stdout, res.stdout + res.stderr
