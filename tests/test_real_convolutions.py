"""Real transforms through a fused convolution on either side of each line
between the in-place and the mixed-radix tiles: the kernel that is taken, and
one transform of each against numpy's FP64 one in host emulation.  Bounds: the
parity bar 5e-7 log2 N (single) / 1e-15 log2 N (double)."""
import math

import numpy as np
import pytest

import hostcheck as H

R2C, C2R, D2Z, Z2D = 0x2A, 0x2C, 0x6A, 0x6C


def _mixed(n, code, batch):
    plan = H.plan1d(n, code, batch)
    text = H.describe(plan)
    H.lib().flagfftDestroy(plan)
    (line,) = [ln for ln in text.splitlines() if ln.strip().startswith("pass ")]
    return "mixed tiles" in line


# 2003 and 4006: a 4096-point convolution, 997: 2048 points, 4079: 8192, 4001:
# Rader of 4000, 3001 and 6002: Rader of 3000, 503: 1024 points
@pytest.mark.parametrize("n,code,batch,mixed", [
    (2003, R2C, 296, False), (2003, R2C, 297, True), (4006, C2R, 296, False), (4006, C2R, 297, True),
    (997, R2C, 592, False), (997, C2R, 593, True), (503, R2C, 1, True),
    (4001, R2C, 148, False), (4001, C2R, 149, True), (6002, R2C, 1, True), (3001, C2R, 148, True),
    (4079, R2C, 1, False), (4079, C2R, 5000, False)])
def test_single_precision_lines(n, code, batch, mixed):
    assert _mixed(n, code, batch) == mixed


# 331: Rader of 330 = 11 x 10 x 3, in 2^20 points from 3178 transforms on
@pytest.mark.parametrize("n,code,batch,mixed", [
    (2003, D2Z, 148, True), (2003, D2Z, 149, False), (8002, Z2D, 148, True), (8002, Z2D, 149, False),
    (997, D2Z, 444, True), (997, Z2D, 445, False), (6002, D2Z, 5000, True),
    (331, D2Z, 3177, True), (331, Z2D, 3178, False), (199, D2Z, 9600, True)])
def test_double_precision_lines(n, code, batch, mixed):
    assert _mixed(n, code, batch) == mixed


@pytest.mark.parametrize("n,batch,double", [(997, 1, False), (2003, 1, False), (2003, 297, False), (4001, 1, False),
                                            (4079, 1, False), (4006, 1, False), (2003, 149, True), (997, 445, True),
                                            (331, 3178, True)])
def test_values(n, batch, double):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (batch, n))
    bound = (1e-15 if double else 5e-7) * math.log2(n)
    ref = np.fft.rfft(x)
    got = H.r2c(x, double)
    assert np.linalg.norm(got - ref) <= bound * np.linalg.norm(ref)
    back = H.c2r(ref, n, double)
    assert np.linalg.norm(back - x * n) <= bound * np.linalg.norm(x * n)
