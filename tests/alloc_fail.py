"""A stand-in for the library's allocator that fails where a test asks it to, as
a preloaded object: build(dir) -> its path.  In the process that preloads it,
fail(what, min_bytes, times) makes the next `times` allocations named `what` of
at least min_bytes report that the device is out of memory."""
import ctypes
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "axion_grav_gb300", "libaxgpu.so")
CODE = r"""
#include <dlfcn.h>
#include <cstddef>
#include <cstring>
struct axg_ctx;
static char name[64];
static size_t least;
static int left, failed;
extern "C" void alloc_fail(const char *what, size_t min_bytes, int times) {
  std::strncpy(name, what, sizeof(name) - 1);
  least = min_bytes;
  left = times;
  failed = 0;
}
extern "C" int alloc_failed() { return failed; }
int axg_alloc(axg_ctx *ctx, void **ptr, size_t bytes, const char *what) {
  using F = int (*)(axg_ctx *, void **, size_t, const char *);
  static F real = (F)dlsym(dlopen("@LIB@", RTLD_NOLOAD | RTLD_NOW), "_Z9axg_allocP7axg_ctxPPvmPKc");
  if (left > 0 && bytes >= least && !std::strcmp(what, name)) {
    --left;
    ++failed;
    *ptr = nullptr;
    return -3;  // AXG_ERR_NOMEM
  }
  return real(ctx, ptr, bytes, what);
}
"""


def build(directory):
    src, so = os.path.join(directory, "alloc_fail.cpp"), os.path.join(directory, "alloc_fail.so")
    with open(src, "w") as f:
        f.write(CODE.replace("@LIB@", LIB))
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", src, "-o", so, "-ldl"], check=True)
    return so


def fail(what, min_bytes, times):
    ctypes.CDLL(None).alloc_fail(what.encode(), ctypes.c_size_t(min_bytes), times)


def failed():
    return ctypes.CDLL(None).alloc_failed()
