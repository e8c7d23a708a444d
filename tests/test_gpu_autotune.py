"""Tuning a lattice leaves it no slower than not tuning it: where the kernel
without tiles is the default and the fastest, it stays."""
import pytest

import axion_grav_gb300 as ag
from tests.test_gpu_evolve import make_params

pytestmark = pytest.mark.gpu


def us_per_step(lat):
    best = float("inf")
    for _ in range(5):
        lat.event_record(0)
        lat.leapfrog(2.0, 1e-3, 16, False, False)
        lat.event_record(1)
        best = min(best, lat.event_elapsed(0, 1) / 16 * 1e3)
    return best


# the default takes 6 to 57 us a step here, the fastest tile 23 to 113
@pytest.mark.parametrize("n", [32, 64])
@pytest.mark.parametrize("prec", [ag.PREC_FP32_MIXED, ag.PREC_FP64_FUSED])
def test_tuned_step_is_no_slower(n, prec):
    with ag.Lattice(make_params(n, prec, ag.GW_UIJ)) as lat:
        lat.ic_gaussian_flat(1.5)
        lat.leapfrog(2.0, 1e-3, 20, False, False)
        default = us_per_step(lat)
        best, ms = lat.autotune(8)
        tuned = us_per_step(lat)
        lat.set_tile(best)
        tile = us_per_step(lat)
    assert best >= 0
    assert tuned < 1.4 * default < tile
    assert ms * 1e3 < 1.4 * tuned
