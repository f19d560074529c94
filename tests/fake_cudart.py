"""Runs a script in a child process with a few CUDA runtime calls behind a
shim that can be told to refuse them, so that the failing calls of the tests
that import this are error codes made on the host, and that notes the kernels
launched and asked about."""
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
typedef struct { unsigned x, y, z; } dim3_;
static const void *launched[64];
static unsigned grid[64], launches;
static const void *asked;
static int answer;
unsigned shim_launches(void) { return launches; }
const void *shim_kernel(unsigned k) { return launched[k % 64]; }
unsigned shim_grid(unsigned k) { return grid[k % 64]; }
const void *shim_asked(int *blocks) { *blocks = answer; return asked; }
int cudaLaunchKernel(const void *f, dim3_ g, dim3_ b, void **a, size_t sm, void *st) {
  static int (*real)(const void *, dim3_, dim3_, void **, size_t, void *);
  if (!real) *(void **)&real = real_of("cudaLaunchKernel");
  launched[launches % 64] = f;
  grid[launches++ % 64] = g.x;
  return real(f, g, b, a, sm, st);
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t sm,
                                                           unsigned fl) {
  static int (*real)(int *, const void *, int, size_t, unsigned);
  if (!real) *(void **)&real = real_of("cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags");
  const int e = real(n, f, b, sm, fl);
  asked = f, answer = *n;
  return e;
}
static size_t largest;
size_t shim_largest(void) { size_t n = largest; largest = 0; return n; }
int cudaMalloc(void **p, size_t n) {
  static int (*real)(void **, size_t);
  if (!real) *(void **)&real = real_of("cudaMalloc");
  if (n >= lo && n <= hi) { refused++; return 2; }  /* cudaErrorMemoryAllocation */
  if (n > largest) largest = n;
  return real(p, n);
}
/* the device's free memory, as the library under test is told */
static size_t left_free;
void shim_free(size_t n) { left_free = n; }
int cudaMemGetInfo(size_t *f, size_t *t) {
  static int (*real)(size_t *, size_t *);
  if (!real) *(void **)&real = real_of("cudaMemGetInfo");
  const int e = real(f, t);
  if (left_free) *f = left_free;
  return e;
}
"""

HEAD = """
import ctypes, sys
sys.path.insert(0, {root!r})
import numpy as np
import render3d_b200 as rb
shim = ctypes.CDLL({so!r})
shim.shim_alloc.argtypes = [ctypes.c_size_t, ctypes.c_size_t]
shim.shim_free.argtypes = [ctypes.c_size_t]
shim.shim_largest.restype = ctypes.c_size_t
shim.shim_kernel.restype = shim.shim_asked.restype = ctypes.c_void_p
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
