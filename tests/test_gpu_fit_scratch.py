"""String fits when the device is short of memory: a scratch that does not fit is
asked for in smaller pieces, with the same fits.  The allocator that fails is
preloaded into a process of its own."""
import os
import subprocess
import sys

import pytest

from tests import alloc_fail

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys
import numpy as np
import axion_grav_gb300 as ag
from tests.alloc_fail import fail, failed
from tests.test_gpu_defects import fields, params

n, limit = int(sys.argv[1]), int(sys.argv[2])
phi = fields("random", n, 9)
phid = 0.1 * fields("random", n, 10)


def fits():
    with ag.Lattice(params(n)) as lat:
        lat.upload(phi, phid)
        sl, wa, sv, cnt = lat.id_defects(1, 4.0)
        return sl, wa, sv, cnt, lat.defect_lists(int(cnt[0]), int(cnt[1]))


a = fits()
assert a[3][0] * 200 > limit  # what the fits of all cells at once take
fail("string fits", limit, 100)
b = fits()
assert failed() >= 1
for x, y in zip(a[:4], b[:4]):
    assert np.array_equal(x, y)
for x, y in zip(a[4], b[4]):
    assert np.array_equal(x, y)
print("fits ok")
"""


# 24: some thousand cells, a warp each; 56: rounds of the eight-lane kernel, and
# of the one that gives a warp to each cell
@pytest.mark.parametrize("n,limit", [(24, 400_000), (56, 8_000_000), (56, 700_000)])
def test_fits_in_smaller_rounds(n, limit, tmp_path):
    env = dict(os.environ, LD_PRELOAD=alloc_fail.build(str(tmp_path)), PYTHONPATH=alloc_fail.ROOT)
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(n), str(limit)], env=env, cwd=alloc_fail.ROOT,
                       capture_output=True, text=True, timeout=280)
    assert r.returncode == 0 and "fits ok" in r.stdout, r.stdout + r.stderr
