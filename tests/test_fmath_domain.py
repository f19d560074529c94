"""r3d_log2_ge1f and r3d_exp2_posf against the general functions on their
domains, compiled from the header as the kernels' host twin: every mantissa
of the first two binades from 1, all exponents with random mantissas and the
ones next to the split at sqrt(2); every 61st float of [0, 126] and the
half-way points where the exponent rounds.  Bit for bit."""
import ctypes
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "r3d_fmath.h"
static long lg(uint32_t b) {
  float x = r3d_u2f(b);
  return r3d_f2u(r3d_log2f(x)) != r3d_f2u(r3d_log2_ge1f(x));
}
static long ex(float x) { return r3d_f2u(r3d_exp2f(x)) != r3d_f2u(r3d_exp2_posf(x)); }
long run_log2(void) {
  long bad = 0;
  for (uint32_t b = 0x3f800000u; b < 0x40800000u; b++) bad += lg(b);
  for (uint32_t e = 127; e < 255; e++) {
    for (uint32_t m = 0; m < 0x800000u; m += 997u) bad += lg(e << 23 | m);
    for (uint32_t m = 0x3504f0u; m < 0x3504f8u; m++) bad += lg(e << 23 | m);
    bad += lg(e << 23 | 0x7fffffu);
  }
  return bad + (r3d_log2_ge1f(R3D_FM_INF) != 128.0f);
}
long run_exp2(void) {
  long bad = ex(0.0f) + ex(126.0f);
  for (uint32_t b = 1; b < 0x42fc0000u; b += 61u) bad += ex(r3d_u2f(b));
  for (int k = 0; k < 126; k++) {
    float h = (float)k + 0.5f;
    bad += ex(h) + ex(nextafterf(h, 0.0f)) + ex(nextafterf(h, 200.0f)) + ex((float)k);
  }
  return bad;
}
"""


def test_domain_versions_are_the_general_ones(tmp_path):
    c = tmp_path / "f.c"
    c.write_text(SRC)
    so = tmp_path / "f.so"
    subprocess.run(["/usr/bin/gcc", "-O2", "-std=c2x", "-D_GNU_SOURCE", "-ffp-contract=off",
                    "-march=native", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "include"),
                    str(c), "-o", str(so), "-lm"], check=True)
    lib = ctypes.CDLL(str(so))
    for fn in (lib.run_log2, lib.run_exp2):
        fn.restype = ctypes.c_long
        assert fn() == 0
