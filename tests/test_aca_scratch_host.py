"""Scratch of the node applications (km_aca.cu) and of the panel QR (km_pqr.cu) of an ACA factor: host arithmetic,
no GPU.

The calls run in a process of their own: an integer division by zero ends it on x86-64.
"""
import ctypes
import subprocess
import sys

import pytest

SCRIPT = """
import ctypes as C, sys
f = C.CDLL(sys.argv[1])._ZN2km14gapply_scratchEiiil  # km::gapply_scratch(int, int, int, int64_t)
f.restype, f.argtypes = C.c_int64, [C.c_int, C.c_int, C.c_int, C.c_int64]
print(f(*map(int, sys.argv[2:])))
"""


def gapply_scratch(lib, *args):
    r = subprocess.run([sys.executable, "-c", SCRIPT, lib._name, *map(str, args)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr)
    return int(r.stdout)


@pytest.mark.parametrize("n,cols", [(0, 0), (0, 8), (4, 0)])
def test_level_without_items_needs_none(lib, n, cols):
    """The root level has no panel to update; a level may also hold only items that go through the products
    over all SMs, which are not counted here (0 columns)."""
    assert gapply_scratch(lib, n, 1, cols, 1) == 0


@pytest.mark.parametrize("n,r,cols,rows", [(1, 300, 1000, 131072), (1, 300, 1, 131072), (2, 300, 200, 65536), (1, 64, 4096, 1 << 20),
                                           (16, 100, 8, 8192), (1, 24, 5, 700)])
def test_scratch_does_not_grow_with_the_rows(lib, n, r, cols, rows):
    """Two sides and the coefficients besides; the split stops at 6 CTAs an SM (152 SMs, 8 columns a CTA at most)
    and at 64 chunks: 2 r values for each column of a chunk, of which there are fewer than 6 * 152 / 2 more than
    CTAs of 8 columns, plus the coefficients' own 2 r values a column."""
    ctas = n * -(-cols // 8)
    most = 2 * r * 8 * (2 * ctas + 6 * 152 // 2)
    got = gapply_scratch(lib, n, r, cols, rows)
    assert 0 <= got <= min(most, 2 * r * 65 * 8 * ctas)


@pytest.mark.parametrize("n,k,rows", [(32, 400, 8192), (1024, 100, 256), (2, 350, 8192), (8, 4000, 12288), (2, 1, 1)])
def test_panel_scratch_is_what_its_chunks_take(lib, n, k, rows):
    """Partial products: 32 values a column and row chunk of a panel, with at most 4 CTAs an SM (152 SMs) more than
    panels, or chunks of 512 rows; two 32 x 32 factors a block."""
    lib._ZN2km16panel_qr_scratchEiil.restype = ctypes.c_int64
    got = lib._ZN2km16panel_qr_scratchEiil(ctypes.c_int(n), ctypes.c_int(k), ctypes.c_int64(rows))
    chunks = max(4 * 152 + n, n * -(-rows // 512))
    assert 0 < got <= n * -(-k // 32) * 2 * 32 * 32 + chunks * k * 32
