"""The mixed-radix tile kernel (csrc/mixed.cuh) at the sizes where its index
arithmetic can go wrong: two to five stages, first and last runs of four
elements, batches that leave a part tile, odd and even lengths of every real
form, real rows that do not start on a pair, and strided tiles.  Bounds: the
parity bar 5e-7 log2 N (single) / 1e-15 log2 N (double) against numpy's FP64
transform.  The CPU tests run the kernel body in host emulation."""
import ctypes
import math

import numpy as np
import pytest

import hostcheck as H

# (n, batch): 24 = 6 4 and 30 = 6 5 the shortest chains, 36 = 6 6, 1200 three
# stages, 1331 = 11^3 and 323 = 17 19 the large radices, 4900 and 14406 long,
# 1013 and 67 convolutions
LENGTHS = [(24, 1), (30, 7), (36, 33), (323, 5), (1200, 3), (1331, 2), (4900, 2), (67, 9), (1013, 3)]


def _bound(double, n):
    return (1e-15 if double else 5e-7) * math.log2(n)


def _err(a, b):
    return np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())


def _real_spectrum(rng, batch, n):
    x = rng.uniform(-1, 1, (batch, n // 2 + 1)) + 1j * rng.uniform(-1, 1, (batch, n // 2 + 1))
    x[:, 0] = x[:, 0].real
    if n % 2 == 0:
        x[:, -1] = x[:, -1].real
    return x


@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("n,batch", LENGTHS)
def test_emulated_rows(n, batch, double):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))
    assert _err(H.c2c(x, -1, double), np.fft.fft(x)) <= _bound(double, n)
    assert _err(H.c2c(x, 1, double), np.fft.ifft(x, norm="forward")) <= _bound(double, n)
    for m in (n, 2 * n):  # the n-point real forms and the half-length ones
        r = rng.uniform(-1, 1, (batch, m))
        assert _err(H.r2c(r, double), np.fft.rfft(r)) <= _bound(double, m)
        s = _real_spectrum(rng, batch, m)
        assert _err(H.c2r(s, m, double), np.fft.irfft(s, m, norm="forward")) <= _bound(double, m)


@pytest.mark.parametrize("n0,n1", [(24, 100), (60, 30), (120, 67), (323, 36)])
def test_emulated_strided(n0, n1):
    rng = np.random.default_rng(n0)
    x = rng.uniform(-1, 1, (n0, n1)) + 1j * rng.uniform(-1, 1, (n0, n1))
    assert _err(H.fft2(x, "c2c_fwd"), np.fft.fft2(x)) <= _bound(False, n0 * n1)
    assert _err(H.fft2(x, "c2c_inv"), np.fft.ifft2(x, norm="forward")) <= _bound(False, n0 * n1)


@pytest.mark.parametrize("double", [False, True])
def test_emulated_unaligned_reals(double):
    """Real rows from an address off a pair: the scalar loads."""
    n, batch, dist = 250, 5, 250
    rng = np.random.default_rng(5)
    t = np.float64 if double else np.float32
    raw = rng.uniform(-1, 1, 1 + batch * dist).astype(t)
    x = raw[1:].reshape(batch, dist)
    out = np.empty((batch, n // 2 + 1), np.complex128 if double else np.complex64)
    h = H.plan1d(n, 0x6A if double else 0x2A, batch)
    fn = H.lib().flagfftExecD2Z if double else H.lib().flagfftExecR2C
    assert fn(h, ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(out.ctypes.data)) == 0
    H.lib().flagfftDestroy(h)
    assert _err(out, np.fft.rfft(x.astype(np.float64))) <= _bound(double, n)


@pytest.mark.gpu
@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("n,batch", LENGTHS + [(14406, 2), (1000, 700), (30, 5001)])
def test_rows(ffb, torch_cuda, n, batch, double):
    torch = torch_cuda
    rng = np.random.default_rng(n)
    ct, rt = (np.complex128, np.float64) if double else (np.complex64, np.float32)
    x = (rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))).astype(ct)
    a = torch.from_numpy(x).cuda()
    b = torch.empty_like(a)
    with ffb.plan1d(n, ffb.Z2Z if double else ffb.C2C, batch) as p:
        for d, ref in ((ffb.FORWARD, np.fft.fft(x.astype(np.complex128))),
                       (ffb.INVERSE, np.fft.ifft(x.astype(np.complex128), norm="forward"))):
            p.execute(a, b, d)
            assert _err(b.cpu().numpy(), ref) <= _bound(double, n)
    for m in (n, 2 * n):
        r = rng.uniform(-1, 1, 1 + batch * m).astype(rt)
        s = _real_spectrum(rng, batch, m).astype(ct)
        sa = torch.from_numpy(s).cuda()
        fwd = torch.empty(batch, m // 2 + 1, dtype=sa.dtype, device="cuda")
        for off in (0, 1):  # rows on and off a pair
            ra = torch.zeros(off + batch * m, dtype=torch.float64 if double else torch.float32, device="cuda")
            ra[off:] = torch.from_numpy(r[:batch * m]).cuda()
            back = torch.empty_like(ra)
            with ffb.plan1d(m, ffb.D2Z if double else ffb.R2C, batch) as p:
                p.execute(ra.data_ptr() + off * ra.element_size(), fwd)
            assert _err(fwd.cpu().numpy(), np.fft.rfft(r[:batch * m].reshape(batch, m).astype(np.float64))) <= \
                _bound(double, m)
            with ffb.plan1d(m, ffb.Z2D if double else ffb.C2R, batch) as p:
                p.execute(sa, back.data_ptr() + off * back.element_size())
            got = back[off:].cpu().numpy().reshape(batch, m)
            assert _err(got, np.fft.irfft(s.astype(np.complex128), m, norm="forward")) <= _bound(double, m)
