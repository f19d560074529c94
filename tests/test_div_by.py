"""r3d_div_by and r3d_div_rcp against IEEE division, compiled from the header as the kernels'
host twin: every divisor up to 8200 (tile and ring sizes and far beyond), and
powers of two and their neighbours up to the stated bound, with random
dividends, whole ones, and the ones nearest to a rounding boundary (b times a
quotient half way between two floats, and its neighbours)."""
import ctypes
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "r3d_fmath.h"
static uint64_t st = 88172645463325252ull;
static uint32_t rnd(void) { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return (uint32_t)(st >> 16); }
static long check(float a, uint32_t b) {
  float fb = (float)b, rb = 1.0f / fb;
  return r3d_f2u(a / fb) != r3d_f2u(r3d_div_by(a, fb, rb));
}
static long divisor(uint32_t b, int n) {
  long bad = 0;
  for (int i = 0; i < n; i++) {
    uint32_t r = rnd();
    /* 2^-40 .. 2^40, both signs */
    bad += check(r3d_u2f((r & 0x807fffffu) | ((87u + rnd() % 80u) << 23)), b);
    bad += check((float)(r >> 8), b);
    /* q half way between two floats: a 25-bit odd number */
    double mid = (double)((r & 0xffffffu) * 2u + 1u + 0x1000000u) * (double)b;
    float a = (float)mid;
    bad += check(a, b) + check(nextafterf(a, INFINITY), b) + check(nextafterf(a, 0.0f), b);
  }
  return bad + check(0.0f, b);
}
/* any divisor: dividends near a rounding boundary of the quotient too */
long run_rcp(void) {
  long bad = 0;
  for (int i = 0; i < 4000000; i++) {
    uint32_t r = rnd(), q = rnd();
    float b = r3d_u2f((r & 0x807fffffu) | ((100u + rnd() % 40u) << 23));
    if (i % 4 == 0) b = r3d_u2f((r & 0x80000007u) | ((100u + rnd() % 40u) << 23) | (i % 8 ? 0x7ffff8u : 0u));
    float rb = 1.0f / b, a = r3d_u2f((q & 0x807fffffu) | ((100u + rnd() % 40u) << 23));
    if (i & 1) {
      double mid = ((double)(q & 0xffffffu) * 2.0 + 1.0 + 0x1000000) * (double)b;
      a = (float)(mid * (i & 2 ? 0x1p-30 : 0x1p-8));
    }
    for (int k = 0; k < 3; k++, a = nextafterf(a, INFINITY))
      bad += r3d_f2u(a / b) != r3d_f2u(r3d_div_rcp(a, b, rb));
  }
  return bad + (r3d_f2u(0.0f / 3.0f) != r3d_f2u(r3d_div_rcp(0.0f, 3.0f, 1.0f / 3.0f)));
}
long run(void) {
  long bad = 0;
  for (uint32_t b = 1; b <= 8200u; b++) bad += divisor(b, 400);
  for (uint32_t k = 13; k < 20; k++)
    for (int d = -1; d <= 1; d++) bad += divisor((1u << k) + d, 20000);
  return bad + divisor((1u << 20) - 1u, 20000);
}
"""


def test_div_by_is_ieee_division(tmp_path):
    c = tmp_path / "d.c"
    c.write_text(SRC)
    so = tmp_path / "d.so"
    subprocess.run(["/usr/bin/gcc", "-O2", "-std=c2x", "-D_GNU_SOURCE", "-ffp-contract=off", "-march=native",
                    "-shared", "-fPIC", "-I" + os.path.join(ROOT, "include"), str(c), "-o", str(so),
                    "-lm"], check=True)
    lib = ctypes.CDLL(str(so))
    for fn in (lib.run, lib.run_rcp):
        fn.restype = ctypes.c_long
        assert fn() == 0
