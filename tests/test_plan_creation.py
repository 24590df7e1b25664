"""Plans of every size class can be made: the lowering finds a tile shape for
each pass it sends to the mixed-radix tiles, up to the one that fills a CTA's
shared memory (231425 to 232448 bytes: 7220, 7225 and 14450 points a buffer
pair, 1800 to 3610 points in the narrowest strided tiles).  Host-emulation
build; nothing is executed."""
import ctypes

import pytest

import hostcheck as H

C2C, R2C, C2R, Z2Z, D2Z, Z2D = 0x29, 0x2A, 0x2C, 0x69, 0x6A, 0x6C


def _smooth(lo, hi):
    out = []

    def grow(v, primes):
        if v > hi:
            return
        if v >= lo:
            out.append(v)
        for k, p in enumerate(primes):
            grow(v * p, primes[k:])

    grow(1, (2, 3, 5, 7))
    return sorted(out)


def _refused(plans):
    bad = []
    for rank, shape, code in plans:
        h = ctypes.c_void_p()
        rc = H.lib().flagfftPlan1d(ctypes.byref(h), shape[0], code, shape[1]) if rank == 1 else \
            H.lib().flagfftPlan2d(ctypes.byref(h), shape[0], shape[1], code)
        if rc:
            bad.append((rank, shape, code, rc))
        else:
            H.lib().flagfftDestroy(h)
    return bad


def test_rows_that_fill_a_cta():
    plans = [(1, (n, b), t) for b in (1, 300) for n, codes in
             [(14450, (C2C, D2Z, Z2D)), (28900, (R2C, C2R)), (7220, (Z2Z,)), (7225, (Z2Z, D2Z, Z2D)),
              (14440, (D2Z, Z2D))] for t in codes]
    assert _refused(plans) == []


# four-steps up to 2^22 points; a real transform of even length lowers to the
# complex one of half its length
@pytest.mark.parametrize("code", [C2C, Z2Z])
def test_smooth_lengths(code):
    assert _refused([(1, (n, 1), code) for n in _smooth(2, 1 << 22)]) == []


# every 7-smooth column length and the others whose narrowest tile fills a
# CTA, over few and many columns; the row axis of the same lengths
@pytest.mark.parametrize("columns", [16, 64, 2000])
@pytest.mark.parametrize("code", [C2C, Z2Z])
def test_image_axes(code, columns):
    axes = _smooth(2, 4096) + [2052, 2394, 3610, 7220, 7225, 14450]
    assert _refused([(2, (n, columns), code) for n in axes]) == []
    assert _refused([(2, (16, n), code) for n in axes]) == []


def test_image_shapes():
    assert _refused([(2, s, t) for s, t in [((3600, 2400), C2C), ((2400, 2400), C2C), ((2880, 2160), C2C),
                                            ((1800, 1200), Z2Z), ((3600, 2400), R2C), ((3600, 2400), C2R)]]) == []
