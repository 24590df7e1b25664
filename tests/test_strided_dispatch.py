"""Which kernel takes a strided pass of a compile-time sequence: the column
kernel wherever it can copy the pass, the tile kernel from one CTA per SM on,
the mixed-radix tiles below.  Host-emulation build (the rules are the plan's)."""
import ctypes

import numpy as np
import pytest

import hostcheck as H

C2C, Z2Z = 0x29, 0x69


def _column_pass(n0, n1, code):
    plan = H.plan2d(n0, n1, code)
    text = H.describe(plan).split("-- Forward execution --")[-1].split("-- Inverse execution --")[0]
    H.lib().flagfftDestroy(plan)
    return [ln for ln in text.splitlines() if ln.strip().startswith("pass ")][1]


@pytest.mark.parametrize("n0,n1,code", [(1024, 16, C2C), (1024, 256, C2C), (1536, 24, C2C), (2048, 128, C2C),
                                        (1024, 64, Z2Z), (1536, 16, Z2Z), (2048, 8, Z2Z)])
def test_column_kernel_keeps_few_groups(n0, n1, code):
    line = _column_pass(n0, n1, code)
    assert "tma-columns(" in line, line
    # (the fallback for buffers off 16 bytes)
    assert "mixed tiles" not in line, line


@pytest.mark.parametrize("n0,n1,mixed", [(2048, 2048, True), (2048, 2040, False), (1536, 2048, False)])
def test_fallback_off_16_bytes(n0, n1, mixed):
    line = _column_pass(n0, n1, C2C)
    assert "tma-columns(" in line and ("mixed tiles" in line) == mixed, line


@pytest.mark.parametrize("n0,n1,code", [(512, 256, C2C), (256, 512, C2C), (256, 512, Z2Z), (512, 512, Z2Z)])
def test_narrow_tiles_below_one_cta_per_sm(n0, n1, code):
    assert "mixed tiles" in _column_pass(n0, n1, code)


# 32-byte row segments only below one 64-byte tile per SM, and in single
# precision only for three stages or more (256 = 16 16, 512 = 8 8 8)
@pytest.mark.parametrize("n0,n1,code,width", [(256, 512, C2C, 8), (240, 512, C2C, 8), (512, 256, C2C, 4),
                                              (300, 128, C2C, 4), (256, 256, Z2Z, 2)])
def test_narrow_tile_width(n0, n1, code, width):
    assert f"per_cta={width} " in _column_pass(n0, n1, code)


# single precision, not a power of two: narrow tiles below half a CTA per SM
@pytest.mark.parametrize("n1,mixed", [(588, True), (592, False)])
def test_columns_of_1701(n1, mixed):
    assert ("mixed tiles" in _column_pass(1701, n1, C2C)) == mixed


@pytest.mark.parametrize("n0,n1,code", [(256, 2376, C2C), (512, 2400, C2C), (256, 2376, Z2Z)])
def test_tile_kernel_from_one_cta_per_sm(n0, n1, code):
    line = _column_pass(n0, n1, code)
    assert " tiles smem" in line and "mixed" not in line and "tma-columns" not in line, line


@pytest.mark.parametrize("n0,n1", [(1024, 20), (2048, 24), (1024, 66), (2048, 34), (4096, 18)])
def test_columns_off_16_bytes(n0, n1):
    """Single-precision columns of a buffer on 8 bytes only: the tile and the
    mixed-radix kernels, also where an aligned pass takes the wide columns."""
    rng = np.random.default_rng(n0)
    raw = (rng.uniform(-1, 1, n0 * n1 + 4) + 1j * rng.uniform(-1, 1, n0 * n1 + 4)).astype(np.complex64)
    first = 1 if raw.ctypes.data % 16 == 0 else 0
    x = raw[first:first + n0 * n1]
    assert x.ctypes.data % 16 == 8
    out = np.empty_like(raw)[first:first + n0 * n1]
    plan = H.plan2d(n0, n1, C2C)
    assert H.lib().flagfftExecC2C(plan, ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(out.ctypes.data), -1) == 0
    H.lib().flagfftDestroy(plan)
    ref = np.fft.fft2(x.reshape(n0, n1).astype(np.complex128)).ravel()
    assert np.linalg.norm(out - ref) <= 5e-7 * np.log2(n0 * n1) * np.linalg.norm(ref)


# a prime times a small factor: the convolutions of the second pass, whose
# outputs are strided, take no more of a tile than leaves every SM one, or an
# SM three; a tile of a few butterflies one warp
@pytest.mark.parametrize("n,batch,code,shape", [(3027, 60, C2C, "per_cta=1 threads=256 "),
                                                (12108, 173, C2C, "per_cta=2 threads=256 "),
                                                (134, 15650, Z2Z, "per_cta=2 threads=32 ")])
def test_strided_convolution_tiles(n, batch, code, shape):
    plan = H.plan1d(n, code, batch)
    text = H.describe(plan).split("-- Forward execution --")[-1].split("-- Inverse execution --")[0]
    H.lib().flagfftDestroy(plan)
    line = [ln for ln in text.splitlines() if ln.strip().startswith("pass ")][1]
    assert shape in line and "mixed tiles" in line, line


@pytest.mark.parametrize("n,batch,double", [(2018, 2, False), (3027, 60, False), (134, 40, True), (201, 3, True)])
def test_strided_convolution_values(n, batch, double):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))
    bound = (1e-15 if double else 5e-7) * np.log2(n)
    for d, ref in ((-1, np.fft.fft(x)), (1, np.fft.ifft(x, norm="forward"))):
        assert np.linalg.norm(H.c2c(x, d, double) - ref) <= bound * np.linalg.norm(ref)
