"""The wide column kernel (csrc/wcols.cuh): every sequence, column and row
outputs with the four-step twiddle, last tiles with dead column pairs (columns
come in pairs: a tensor copy wants an even row length).  Bounds: the parity bar 5e-7 log2 N against an FP64
transform.  The CPU tests run the kernel body in host emulation, which takes
passes of four tiles or more."""
import math

import numpy as np
import pytest

import hostcheck as H


def _err(a, b):
    return np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())


# columns of 4096, 2048, 1536 and 1024 points: 4, 8, 8 and 16 to a tile
@pytest.mark.parametrize("n0,n1", [(4096, 18), (2048, 34), (1536, 40), (1024, 66)])
def test_emulated_columns(n0, n1):
    rng = np.random.default_rng(n0)
    x = rng.uniform(-1, 1, (n0, n1)) + 1j * rng.uniform(-1, 1, (n0, n1))
    bound = 5e-7 * math.log2(n0 * n1)
    assert _err(H.fft2(x, "c2c_fwd"), np.fft.fft2(x)) <= bound
    assert _err(H.fft2(x, "c2c_inv"), np.fft.ifft2(x, norm="forward")) <= bound


@pytest.mark.parametrize("n,batch", [(1 << 21, 2), (3 << 19, 1)])
def test_emulated_four_step(n, batch):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))
    assert _err(H.c2c(x, -1), np.fft.fft(x)) <= 5e-7 * math.log2(n)
    assert _err(H.c2c(x, 1), np.fft.ifft(x, norm="forward")) <= 5e-7 * math.log2(n)


# enough columns for four tiles per SM; the last tile partial
@pytest.mark.gpu
@pytest.mark.parametrize("n0,n1", [(4096, 2378), (2048, 4746), (1536, 4742), (1024, 9490)])
def test_columns(ffb, torch_cuda, n0, n1):
    torch = torch_cuda
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n0)
    x = torch.view_as_complex(torch.randn(n0, n1, 2, generator=gen, device="cuda"))
    y = torch.empty_like(x)
    bound = 5e-7 * math.log2(n0 * n1)
    with ffb.plan2d(n0, n1, ffb.C2C) as p:
        for d, f in ((ffb.FORWARD, torch.fft.fft2), (ffb.INVERSE, lambda v: torch.fft.ifft2(v, norm="forward"))):
            p.execute(x, y, d)
            ref = f(x.to(torch.complex128))
            assert float((y - ref).norm() / ref.norm()) <= bound
    assert ffb.device_wait_failures() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n,batch", [(1 << 23, 2), (3 << 21, 2)])
def test_four_step(ffb, torch_cuda, n, batch):
    torch = torch_cuda
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    x = torch.view_as_complex(torch.randn(batch, n, 2, generator=gen, device="cuda"))
    y = torch.empty_like(x)
    with ffb.plan1d(n, ffb.C2C, batch) as p:
        for d, f in ((ffb.FORWARD, torch.fft.fft), (ffb.INVERSE, lambda v: torch.fft.ifft(v, norm="forward"))):
            p.execute(x, y, d)
            ref = f(x.to(torch.complex128))
            assert float((y - ref).norm() / ref.norm()) <= 5e-7 * math.log2(n)
