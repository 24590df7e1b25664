"""The 64-register row kernels (csrc/rows.cuh rows_dense, csrc/rrows.cuh): one
row more and one fewer than the smallest pass that takes them, a part tile,
both directions.
Bounds: the parity bar 5e-7 log2 N against an FP64 transform."""
import math

import pytest

POINTS = 1 << 22


@pytest.mark.gpu
@pytest.mark.parametrize("less", [0, 1])
@pytest.mark.parametrize("n,core", [(4096, 4096), (8192, 8192), (509, 1024), (1009, 2048), (2039, 4096), (4079, 8192)])
def test_complex(ffb, torch_cuda, n, core, less):
    torch = torch_cuda
    batch = POINTS // core + 1 - 2 * less
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    x = torch.view_as_complex(torch.randn(batch, n, 2, generator=gen, device="cuda"))
    y = torch.empty_like(x)
    with ffb.plan1d(n, ffb.C2C, batch) as p:
        for d, f in ((ffb.FORWARD, torch.fft.fft), (ffb.INVERSE, lambda v: torch.fft.ifft(v, norm="forward"))):
            p.execute(x, y, d)
            ref = f(x.to(torch.complex128))
            assert float((y - ref).norm() / ref.norm()) <= 5e-7 * math.log2(n)


@pytest.mark.gpu
@pytest.mark.parametrize("half", [512, 1024, 2048, 4096, 8192])
def test_real(ffb, torch_cuda, half):
    torch = torch_cuda
    n, batch = 2 * half, POINTS // half + 1
    gen = torch.Generator(device="cuda")
    gen.manual_seed(half)
    x = torch.randn(batch, n, generator=gen, device="cuda")
    y = torch.empty(batch, half + 1, dtype=torch.complex64, device="cuda")
    z = torch.empty_like(x)
    with ffb.plan1d(n, ffb.R2C, batch) as p, ffb.plan1d(n, ffb.C2R, batch) as q:
        p.execute(x, y)
        ref = torch.fft.rfft(x.double())
        assert float((y - ref).norm() / ref.norm()) <= 5e-7 * math.log2(n)
        q.execute(y, z)
        assert float((z.double() - n * x.double()).norm() / (n * x.double()).norm()) <= 1e-6 * math.log2(n)
