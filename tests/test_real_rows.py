"""Real transforms on the compile-time row kernels (csrc/rrows.cuh): every
sequence length, single rows, part tiles, rows that do not start on a pair
(which fall back to the mixed-radix tiles).  Bounds: the parity bar 5e-7 log2 N (single) / 1e-15 log2 N
(double) against numpy's FP64 transform."""
import math

import numpy as np
import pytest

import hostcheck as H

HALVES = [128, 256, 512, 1024, 1536, 1701, 2048, 4096, 8192, 16384]


def _bound(double, n):
    return (1e-15 if double else 5e-7) * math.log2(n)


def _err(a, b):
    return np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())


@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("half", HALVES)
def test_emulated(half, double):
    n, batch = 2 * half, 1 if half > 4096 else 5
    x = np.random.default_rng(half).uniform(-1, 1, (batch, n))
    spec = np.fft.rfft(x)
    assert _err(H.r2c(x, double), spec) <= _bound(double, n)
    assert _err(H.c2r(spec, n, double), x * n) <= _bound(double, n)


@pytest.mark.gpu
@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("half,batch", [(h, 1) for h in HALVES] + [(h, 1337) for h in HALVES[:7]])
def test_rows(ffb, torch_cuda, half, batch, double):
    torch = torch_cuda
    n = 2 * half
    rt = np.float64 if double else np.float32
    h = np.random.default_rng(half).uniform(-1, 1, batch * n).astype(rt)
    ref = np.fft.rfft(h.reshape(batch, n).astype(np.float64))
    # rows on a pair and, where the transform is one on-chip pass, off it (a
    # transform of several passes reads its rows as complex elements)
    for off in (0, 1) if half < 16384 else (0,):
        a = torch.zeros(off + batch * n, dtype=torch.float64 if double else torch.float32, device="cuda")
        a[off:] = torch.from_numpy(h).cuda()
        y = torch.empty(batch, half + 1, dtype=torch.complex128 if double else torch.complex64, device="cuda")
        z = torch.empty_like(a)
        with ffb.plan1d(n, ffb.D2Z if double else ffb.R2C, batch) as p:
            p.execute(a.data_ptr() + off * a.element_size(), y)
        assert _err(y.cpu().numpy(), ref) <= _bound(double, n)
        with ffb.plan1d(n, ffb.Z2D if double else ffb.C2R, batch) as p:
            p.execute(y, z.data_ptr() + off * z.element_size())
        assert _err(z[off:].cpu().numpy(), n * h.astype(np.float64)) <= 2 * _bound(double, n)
