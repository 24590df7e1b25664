"""Buffers that the kernels cannot address are refused on the host, before any
launch: complex data off its element size, reals off theirs, and the reals of
a transform of several passes off a pair.  Host-emulation build only: such an
address must never reach a GPU."""
import ctypes
import math

import numpy as np
import pytest

import hostcheck as H

C2C, R2C, C2R, Z2Z, D2Z, Z2D = 0x29, 0x2A, 0x2C, 0x69, 0x6A, 0x6C
UNALIGNED = 9


def _bytes(n):
    raw = np.zeros(n + 64, np.uint8)
    return raw, raw.ctypes.data + -raw.ctypes.data % 32


def _exec(code, n, batch, in_off, out_off, x=None):
    """Status and output bytes of one call whose buffers start `off` bytes past
    a 32-byte boundary."""
    L = H.lib()
    dbl = code in (Z2Z, D2Z, Z2D)
    cx, half = 16 if dbl else 8, n // 2 + 1
    nin = batch * (half * cx if code in (C2R, Z2D) else n * cx // 2 if code in (R2C, D2Z) else n * cx)
    nout = batch * (half * cx if code in (R2C, D2Z) else n * cx // 2 if code in (C2R, Z2D) else n * cx)
    keep, a = _bytes(nin)
    keep2, b = _bytes(nout)
    if x is not None:
        ctypes.memmove(a + in_off, x.ctypes.data, nin)
    h = H.plan1d(n, code, batch)
    fn = {C2C: "C2C", Z2Z: "Z2Z", R2C: "R2C", D2Z: "D2Z", C2R: "C2R", Z2D: "Z2D"}[code]
    args = (h, a + in_off, b + out_off) + ((-1,) if code in (C2C, Z2Z) else ())
    rc = getattr(L, "flagfftExec" + fn)(*args)
    L.flagfftDestroy(h)
    return rc, ctypes.string_at(b + out_off, nout), keep, keep2


# 65536 in two passes and the Hermitian one; 60022 = 2 x 30011 through a
# convolution chain of the half length
@pytest.mark.parametrize("n", [65536, 60022])
@pytest.mark.parametrize("double", [False, True])
def test_reals_of_several_passes_start_on_a_pair(n, double):
    fwd, inv, real = (D2Z, Z2D, 8) if double else (R2C, C2R, 4)
    assert _exec(fwd, n, 1, real, 0)[0] == UNALIGNED
    assert _exec(inv, n, 1, 0, real)[0] == UNALIGNED
    assert _exec(fwd, n, 1, 2 * real, 0)[0] == 0
    assert _exec(inv, n, 1, 0, 2 * real)[0] == 0


@pytest.mark.parametrize("double", [False, True])
def test_complex_off_its_element(double):
    cx = 16 if double else 8
    for code in (Z2Z, D2Z, Z2D) if double else (C2C, R2C, C2R):
        for n in (64, 1000, 1009, 65536):
            if code not in (R2C, D2Z):
                assert _exec(code, n, 1, cx // 2, 0)[0] == UNALIGNED
            if code not in (C2R, Z2D):
                assert _exec(code, n, 1, 0, cx // 2)[0] == UNALIGNED
    assert _exec(D2Z if double else R2C, 64, 1, 2, 0)[0] == UNALIGNED


@pytest.mark.parametrize("n", [4096, 1000, 1009, 30011])
def test_other_reals_need_no_pair(n):
    x = np.random.default_rng(n).uniform(-1, 1, (2, n)).astype(np.float32)
    rc, out, *_ = _exec(R2C, n, 2, 4, 0, x)
    got = np.frombuffer(out, np.complex64).reshape(2, -1)
    ref = np.fft.rfft(x.astype(np.float64))
    assert rc == 0 and np.linalg.norm(got - ref) <= 2e-6 * math.log2(n) * np.linalg.norm(ref)


def test_batch_plans_and_server():
    L = H.lib()
    i, vp = ctypes.c_int, ctypes.c_void_p
    L.flagfftB200PlanBatch.argtypes = [ctypes.POINTER(vp), i, ctypes.POINTER(i), ctypes.POINTER(i), i]
    h = vp()
    assert L.flagfftB200PlanBatch(ctypes.byref(h), 1, (i * 1)(64), (i * 1)(2), C2C) == 0
    keep, a = _bytes(1 << 20)
    assert L.flagfftExecC2C(h, a + 4, a + (1 << 16), -1) == UNALIGNED
    assert L.flagfftExecC2C(h, a, a + (1 << 16) + 4, -1) == UNALIGNED
    L.flagfftDestroy(h)
    L.flagfftB200ServerCreate.argtypes = [ctypes.POINTER(vp), ctypes.c_longlong, i]
    L.flagfftB200ServerSubmit.argtypes = [vp, i, i, i, i, vp, vp, ctypes.POINTER(ctypes.c_longlong)]
    L.flagfftB200ServerDestroy.argtypes = [vp]
    srv, tk = vp(), ctypes.c_longlong()
    assert L.flagfftB200ServerCreate(ctypes.byref(srv), 1 << 30, 1) == 0
    try:
        for code, n, off_in, off_out in [(C2C, 64, 4, 0), (Z2Z, 64, 0, 8), (R2C, 65536, 4, 0), (C2R, 65536, 0, 4)]:
            assert L.flagfftB200ServerSubmit(srv, code, n, 1, -1, a + off_in, a + (1 << 19) + off_out,
                                             ctypes.byref(tk)) == UNALIGNED
    finally:
        L.flagfftB200ServerDestroy(srv)
