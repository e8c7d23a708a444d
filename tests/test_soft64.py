"""axg_soft64.h (double products on the integer pipes) against the host's own
multiplication, bit for bit, and the window that says where it may be used.
The header is plain C++ but for a carry chain in device code; that chain is
covered by the bit-exact evolution tests on the GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "axion_grav_gb300", "csrc")
CODE = r"""
#include "axg_soft64.h"
extern "C" void products(const double *a, const double *b, long n, double *p, double *q, unsigned char *okp,
                         unsigned char *okq) {
  for (long i = 0; i < n; ++i) {
    uint32_t ok = ~0u;
    p[i] = axs_mul(a[i], b[i], &ok);
    okp[i] = (ok & AXS_WINDOW) != 0;
    const axs_const c = axs_const_of(b[i]);
    ok = c.ok ? ~0u : 0u;
    q[i] = axs_mulc(a[i], &c, &ok);
    okq[i] = (ok & AXS_WINDOW) != 0;
  }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("soft64")
    src, so = d / "s.cpp", d / "s.so"
    src.write_text(CODE)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def products(lib, a, b):
    n = len(a)
    p, q = np.empty(n), np.empty(n)
    op, oq = np.empty(n, np.uint8), np.empty(n, np.uint8)
    vp = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    lib.products(vp(a), vp(b), ctypes.c_long(n), vp(p), vp(q), vp(op), vp(oq))
    return p, q, op.astype(bool), oq.astype(bool)


def doubles(rng, n, emin, emax, ones=0, zeros=0):
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    if zeros:
        m &= ~((np.uint64(1) << rng.integers(0, zeros, n).astype(np.uint64)) - np.uint64(1))
    if ones:
        m |= (np.uint64(1) << rng.integers(0, ones, n).astype(np.uint64)) - np.uint64(1)
    e = rng.integers(emin + 1023, emax + 1024, n).astype(np.uint64)
    s = rng.integers(0, 2, n).astype(np.uint64)
    return (s << np.uint64(63) | e << np.uint64(52) | m).view(np.float64)


# significands with long runs of zeros or ones make products that end in a tie
# (1 0...0), just beside one, or round up through a carry into the exponent
@pytest.mark.parametrize("kw", [{}, {"zeros": 53}, {"ones": 53}, {"zeros": 27}])
@pytest.mark.parametrize("erange", [(-40, 40), (-511, 512), (-1022, 1023)])
def test_products_equal_the_hosts(lib, kw, erange):
    rng = np.random.default_rng(7)
    a, b = doubles(rng, 200_000, *erange, **kw), doubles(rng, 200_000, *erange, **kw)
    p, q, op, oq = products(lib, a, b)
    with np.errstate(all="ignore"):
        exact = a * b
    assert np.array_equal(p[op].view(np.uint64), exact[op].view(np.uint64))
    assert np.array_equal(q[oq].view(np.uint64), exact[oq].view(np.uint64))
    if erange == (-40, 40):
        assert op.all() and oq.all()


def test_operands_outside_the_window_are_refused(lib):
    bad = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0 ** -1022, 2.0 ** -512, 2.0 ** 513, 1.7e308])
    good = np.full(len(bad), 1.5)
    for a, b in ((bad, good), (good, bad)):
        _, _, op, oq = products(lib, a, b)
        assert not op.any() and not oq.any()
    edge = np.array([2.0 ** -511, 2.0 ** 512])
    p, _, op, _ = products(lib, edge, np.array([2.0 ** -511, 2.0 ** 511]))
    assert op.all() and np.array_equal(p, [2.0 ** -1022, 2.0 ** 1023])
    # in the window each, but the product overflows
    _, _, op, _ = products(lib, np.array([1.9 * 2.0 ** 512]), np.array([1.9 * 2.0 ** 512]))
    assert not op.any()
