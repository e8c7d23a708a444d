"""Classification and winding of fields with components that are no numbers or
infinite: the site's phase is no number whichever component is bad, and FP32
decides no cell that touches it."""
import numpy as np
import pytest

import axion_grav_gb300 as ag
from oracle import axo
from tests.test_gpu_defects import fields, params

pytestmark = pytest.mark.gpu

NAN, INF = np.nan, np.inf


def touched(bad):
    """The cells with a bad corner: cell (x, y, z) has its corners at + 0, 1."""
    t = np.zeros_like(bad)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                t |= np.roll(bad, (-dz, -dy, -dx), (0, 1, 2))
    return t


def run(p, phi, which):
    with ag.Lattice(p) as lat:
        lat.upload(phi, np.zeros_like(phi))
        counts = lat.classify_cells(which)
        return counts, lat.defect_flags(), lat.string_winding(), lat.download(phidot=False)[0]


# 12: sites on every face; 34: past a tile; "half": gaps FP32 leaves to FP64
@pytest.mark.parametrize("n,kind", [(12, "random"), (34, "smooth"), (12, "half")])
@pytest.mark.parametrize("which", [7, 1])
@pytest.mark.parametrize("prec", [ag.PREC_FP64_PLAIN, ag.PREC_FP32_MIXED])
@pytest.mark.parametrize("site", [complex(NAN, 1.0), complex(0.3, NAN), complex(NAN, 0.0), complex(-2.0, NAN),
                                  complex(INF, 1.0), complex(0.3, -INF), complex(-INF, INF), complex(NAN, INF)])
def test_bad_components(n, kind, which, prec, site):
    phi = fields(kind, n, 7)
    if prec == ag.PREC_FP32_MIXED:
        phi = phi.astype(np.complex64).astype(np.complex128)
    rng = np.random.default_rng(3)
    bad = np.zeros((n, n, n), bool)
    for _ in range(9):
        bad[tuple(rng.integers(0, n, 3))] = True
    bad[0, 0, 0] = bad[n - 1, 2, 3] = True
    phi[bad] = site
    both = phi.copy()
    p = params(n, prec)
    counts, flags, wind, snap = run(p, phi, which)
    with np.errstate(all="ignore"):
        ref, _ = axo.classify_cells(params(n), snap, which, 0)
        assert np.array_equal(wind, axo.string_winding(params(n), snap))
    ok = ~touched(bad)
    assert np.array_equal(flags[ok], ref[ok])
    assert list(counts) == [int(np.count_nonzero(flags & b)) for b in (1, 2, 4)]
    # the deterministic arctangent makes NaN of either
    both[bad] = complex(NAN, NAN)
    c2, f2, w2, _ = run(p, both, which)
    assert np.array_equal(flags, f2) and np.array_equal(counts, c2) and np.array_equal(wind, w2)
