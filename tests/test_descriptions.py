"""A plan's description names the kernel that its passes run on (for buffers
that keep the kernel's copy rules).  Host-emulation build; there the wide
column kernel takes passes of four tiles or more (four per SM on a GPU)."""
import pytest

import hostcheck as H

C2C, R2C, C2R, Z2Z, D2Z = 0x29, 0x2A, 0x2C, 0x69, 0x6A


def _passes(plan):
    try:
        text = H.describe(plan).split("-- Forward execution --")[-1].split("-- Inverse execution --")[0]
        return [ln.split(": ", 1)[1] for ln in text.splitlines() if ln.strip().startswith("pass ")]
    finally:
        H.lib().flagfftDestroy(plan)


@pytest.mark.parametrize("n,batch,code,named,absent", [
    (4096, 256, C2C, "", "64-register"), (4096, 1024, C2C, "64-register", "tiles"),
    (1009, 2048, C2C, "64-register", "tiles"), (1009, 2048, Z2Z, "", "64-register"),
    (2048, 64, R2C, "real rows", "tiles"), (2048, 8192, R2C, "real rows 64-register", "tiles"),
    (2048, 64, D2Z, "real rows", "64-register"), (3000, 64, R2C, "mixed tiles", "real rows"),
    (1200, 64, C2C, "mixed tiles", "64-register")])
def test_rows(n, batch, code, named, absent):
    (line,) = _passes(H.plan1d(n, code, batch))
    assert named in line and absent not in line, line


def test_real_rows_shape():
    (line,) = _passes(H.plan1d(2048, R2C, 8192))
    assert "per_cta=2 threads=128 real rows 64-register smem=17456 " in line, line


@pytest.mark.parametrize("n0,n1,code,wide", [(4096, 12, C2C, False), (4096, 16, C2C, True), (4096, 16, Z2Z, False)])
def test_columns(n0, n1, code, wide):
    line = _passes(H.plan2d(n0, n1, code))[1]
    assert ("wide-tma-columns" in line) == wide and "tma-columns(threads=" in line, line


def test_rows_of_1024_points_from_the_column_kernel():
    """A four-step's first pass of 1024 points writes rows: not the wide form."""
    first, second = _passes(H.plan1d(1 << 20, C2C, 4))
    assert " tma-columns(" in first and "+twiddle" in first and "wide" not in first, first
    assert "wide-tma-columns(" in second, second
