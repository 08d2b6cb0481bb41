"""Scratch of the node applications of an ACA factor (km_aca.cu): host arithmetic, no GPU.

The calls run in a process of their own: an integer division by zero ends it on x86-64.
"""
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
