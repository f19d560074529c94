"""Runs a script in a child process with a few CUDA runtime calls behind a
shim that can be told to refuse them: the failing calls of the tests that
import this are error codes made on the host."""
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static int copy_in;              /* refuse the copy_in-th copy from now */
static size_t lo = 1, hi;        /* refuse allocations of lo..hi bytes */
static int refused;
/* the runtime is loaded with the library under test, outside the global scope */
static void *real_of(const char *name) {
  void *h = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
  return h ? dlsym(h, name) : 0;
}
void shim_copy(int n) { copy_in = n; }
void shim_alloc(size_t a, size_t b) { lo = a, hi = b; }
int shim_refused(void) { int r = refused; refused = 0; return r; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) {
  static int (*real)(void *, const void *, size_t, int, void *);
  if (!real) *(void **)&real = real_of("cudaMemcpyAsync");
  if (copy_in > 0 && --copy_in == 0) { refused++; return 1; }  /* cudaErrorInvalidValue */
  return real(d, s, n, k, st);
}
int cudaMalloc(void **p, size_t n) {
  static int (*real)(void **, size_t);
  if (!real) *(void **)&real = real_of("cudaMalloc");
  if (n >= lo && n <= hi) { refused++; return 2; }  /* cudaErrorMemoryAllocation */
  return real(p, n);
}
"""

HEAD = """
import ctypes, sys
sys.path.insert(0, {root!r})
import numpy as np
import render3d_b200 as rb
shim = ctypes.CDLL({so!r})
shim.shim_alloc.argtypes = [ctypes.c_size_t, ctypes.c_size_t]
lut = rb.scroll_ramp_tf()
W, H = 48, 40

def look(c, mode_of=None, **kw):
    p = rb.camera_view(0.6, -0.5, 1.8, W, H, lut, step_voxels=0.5, **kw)
    p.brick_mode = mode_of if mode_of is not None else 0
    return c.raycast(p, W, H)

def refused(f, code):
    try:
        f()
    except rb.R3DError as e:
        assert code in str(e), str(e)
    else:
        raise AssertionError("accepted")
    assert shim.shim_refused() >= 1

c = rb.Context(0)
c.set_transfer(lut)
"""


def run(tmp_path, body: str) -> None:
    so = str(tmp_path / "shim.so")
    src = tmp_path / "shim.c"
    src.write_text(SHIM)
    subprocess.run(["/usr/bin/gcc", "-O1", "-shared", "-fPIC", "-o", so, str(src), "-ldl"], check=True)
    script = tmp_path / "script.py"
    script.write_text(HEAD.format(root=ROOT, so=so) + textwrap.dedent(body) + "\nprint('done')\n")
    r = subprocess.run([sys.executable, str(script)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=so))
    assert r.returncode == 0 and r.stdout.endswith("done\n"), (r.returncode, r.stdout, r.stderr)
