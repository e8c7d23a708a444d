"""id_defects after a call that found no memory for its lists: the lists that
were given up do not count as there any more."""
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

n = 16
few, many = fields("strings", n, 1), fields("random", n, 2)
zero = np.zeros_like(few)


def lists(lat, phi):
    lat.upload(phi, zero)
    cnt = lat.id_defects(1, 4.0)[3]
    return (cnt,) + lat.defect_lists(int(cnt[0]), int(cnt[1]))


with ag.Lattice(params(n)) as lat:
    a = lists(lat, few)
    fail(sys.argv[1], 1, 1)
    try:
        lists(lat, many)
        raise SystemExit("the failed allocation went unnoticed")
    except ag.AxgError:
        assert failed() == 1
    b = lists(lat, few)
    c = lists(lat, many)
for x, y in zip(a, b):
    assert np.array_equal(x, y)
assert c[0][0] > a[0][0] and len(c[1]) == c[0][0] and np.all(np.isfinite(c[1]))
print("lists ok")
"""


@pytest.mark.parametrize("what", ["string list", "wall list"])
def test_lists_after_a_failed_allocation(what, tmp_path):
    env = dict(os.environ, LD_PRELOAD=alloc_fail.build(str(tmp_path)), PYTHONPATH=alloc_fail.ROOT)
    r = subprocess.run([sys.executable, "-c", SCRIPT, what], env=env, cwd=alloc_fail.ROOT, capture_output=True,
                       text=True, timeout=280)
    assert r.returncode == 0 and "lists ok" in r.stdout, r.stdout + r.stderr
