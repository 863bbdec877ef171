"""Which calls the lean passes take over, where that could go wrong: passes after a
clustered plane, members of a batch, installed kernels, overlapping arrays, planes split
into rows and columns."""

from __future__ import annotations

import math

import numpy
import pytest

from helpers import fft_bound

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
