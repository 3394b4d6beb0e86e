"""What callers without the package's tuning table run with: the C ABI, and the C++
templates by the same defaults."""
import subprocess
import sys

import mdiscriminator_b200 as mdx
from mdiscriminator_b200 import build as mdx_build

READ = """
import ctypes
import mdiscriminator_b200 as mdx
L = ctypes.CDLL(mdx.LIB_PATH)  # not mdx.lib(), which installs the table
for elem in (mdx.ELEM_U32, mdx.ELEM_REC8, mdx.ELEM_REC16):
    for m in (2, 8, 16, 64):
        for n in (1, 1 << 20, 1 << 28, 0xffffffff):
            t = mdx.Tuning()
            assert L.mdx_get_tuning(elem, m, ctypes.c_uint64(n), ctypes.byref(t)) == mdx.MDX_OK
            assert (t.plain_two_kernel, t.plain_ctas_per_sm, t.tile_threads, t.tile_bytes) == (1, 0, 256, 64)
t = mdx.Tuning()  # the one-kernel form by its knob
assert L.mdx_set_tuning(mdx.ELEM_U32, 8, 20, 20, ctypes.byref(t)) == mdx.MDX_OK
assert L.mdx_get_tuning(mdx.ELEM_U32, 8, ctypes.c_uint64(1 << 20), ctypes.byref(t)) == mdx.MDX_OK
assert t.plain_two_kernel == 0
"""


def test_two_kernels_without_a_table():
    mdx_build.build()
    subprocess.run([sys.executable, "-c", READ], check=True)
    assert mdx.get_tuning(mdx.ELEM_U32, 8, 1 << 28)["plain_two_kernel"] == 1
