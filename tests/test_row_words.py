"""Which aligned words the byte-row loads read (r3d_row_words, compiled from
the header): for every row length, address and position, words that hold the
wanted bytes and lie inside the row, never outside the buffer that starts and
ends with it; and words wherever they do."""
import ctypes
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = """
#include "r3d_rows.h"
uint32_t row_words(uint32_t off, uint32_t x, uint32_t n) { return r3d_row_words(off, x, n); }
"""


def test_words_lie_inside_the_row(tmp_path):
    src = tmp_path / "rows.c"
    src.write_text(SRC)
    so = str(tmp_path / "rows.so")
    subprocess.run(["/usr/bin/gcc", "-O1", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "render3d_b200", "csrc"), "-o", so,
                    str(src)], check=True)
    lib = ctypes.CDLL(so)
    for start in range(4):  # the row's address
        for n in range(1, 40):
            for x in range(n):
                off = (start + x) % 4
                k = lib.row_words(off, x, n)
                lo, hi = x - off, x - off + 4 * k  # bytes of the row that are read
                inside = x - off >= 0 and x - off + (8 if off else 4) <= n
                assert bool(k) == inside, (start, n, x)
                if k:
                    assert 0 <= lo and hi <= n
                    assert lo <= x and x + 4 <= hi
