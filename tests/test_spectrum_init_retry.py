"""axg_spec_init after a failed attempt: the next call has to start again (and
here fail again), not take the members that were made for a finished set.
Run on the host: the program below stands in for the library's allocator, and
without a device every CUDA call fails."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "axion_grav_gb300", "csrc")
CODE = r"""
#include <cstdio>
#include <cstdlib>
#include "axg_internal.h"
int axg_spec_init(axg_ctx *ctx);
static int allocs, fail_at, live;
int axg_alloc(axg_ctx *ctx, void **ptr, size_t bytes, const char *what) {
  *ptr = nullptr;
  if (++allocs == fail_at) return AXG_ERR_NOMEM;
  *ptr = std::calloc(1, bytes);
  ++live;
  return AXG_OK;
}
void axg_free(axg_ctx *ctx, void **ptr) {
  if (*ptr) --live;
  std::free(*ptr);
  *ptr = nullptr;
}
int main(int argc, char **argv) {
  fail_at = std::atoi(argv[1]);
  axg_ctx ctx;
  ctx.p.num_bin = 4;
  ctx.p.dspa = 0.5;
  ctx.n = 16;
  ctx.n3 = 16 * 16 * 16;
  const int first = axg_spec_init(&ctx), after = live;
  allocs = 0;
  const int second = axg_spec_init(&ctx);
  std::printf("%d %d %d %d\n", first, second, after, live);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(built, tmp_path_factory):
    cuda = "/usr/local/cuda"
    if not os.path.exists(os.path.join(cuda, "include", "cuda.h")):
        pytest.skip("CUDA headers not found")
    d = tmp_path_factory.mktemp("specinit")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(CODE)
    lib = os.path.join(ROOT, "axion_grav_gb300")
    subprocess.run(["g++", "-std=c++17", "-rdynamic", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(cuda, "include"), str(src), "-o", str(exe), "-L", lib, "-l:libaxgpu.so",
                    "-Wl,-rpath," + lib, "-Wl,--unresolved-symbols=ignore-in-shared-libs"], check=True)
    return str(exe)


# 0: the first CUDA call after the allocations fails; else the allocation of that number
@pytest.mark.parametrize("fail_at", [0, 1, 2, 4, 6])
def test_second_attempt_reports_the_error_again(program, fail_at):
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([program, str(fail_at)], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    first, second, after, live = map(int, r.stdout.split())
    assert first != 0 and second != 0
    assert after == 0 and live == 0
