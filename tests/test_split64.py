"""axs_split (axg_soft64.h), a double as the sum of two floats formed on integers,
against the conversions it stands for: the same sum, no bit less."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.test_soft64 import CSRC, doubles

CODE = r"""
#include "axg_soft64.h"
extern "C" void split(const double *x, long n, float *h, float *l, unsigned char *ok) {
  for (long i = 0; i < n; ++i) ok[i] = axs_split(x[i], h + i, l + i) != 0;
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("split64")
    src, so = d / "s.cpp", d / "s.so"
    src.write_text(CODE)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def run(x):
        h, l, ok = np.empty(len(x), np.float32), np.empty(len(x), np.float32), np.empty(len(x), np.uint8)
        vp = lambda a: a.ctypes.data_as(ctypes.c_void_p)
        lib.split(vp(x), ctypes.c_long(len(x)), vp(h), vp(l), vp(ok))
        return h, l, ok.astype(bool)

    return run


# long runs of zeros or ones in the significand: ties of h and of l, carries into the exponent
@pytest.mark.parametrize("kw", [{}, {"zeros": 53}, {"ones": 53}, {"zeros": 30}, {"ones": 29}])
def test_sum_equals_the_conversions(split, kw):
    rng = np.random.default_rng(5)
    x = np.concatenate([doubles(rng, 300_000, -74, 126, **kw), [1.0, -1.0, 2.0 ** -74, np.nextafter(2.0 ** 127, 0)]])
    h, l, ok = split(x)
    ch = x.astype(np.float32)
    cl = (x - ch.astype(np.float64)).astype(np.float32)
    s, c = h.astype(np.float64) + l, ch.astype(np.float64) + cl
    assert ok.all() and np.array_equal(s, c)
    assert np.all(np.abs(x - s) <= 2.0 ** -49 * np.abs(x))
    assert np.all(np.abs(l) <= 2.0 ** -24 * 2.0 ** (np.floor(np.log2(np.abs(x))) + 1))


def test_refused(split):
    bad = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, np.nextafter(2.0 ** -74, 0), 2.0 ** 127, 1e308]
    assert not split(np.array(bad))[2].any()
