"""Classification and winding at the edges of their 32 x 8 tiles and of the
plane runs a CTA walks, with cells decided in FP32 and in FP64, against the
oracle."""
import numpy as np
import pytest

import axion_grav_gb300 as ag
from oracle import axo
from tests.test_gpu_defects import fields, params

pytestmark = pytest.mark.gpu


# 4, 6: smaller than a tile; 34, 66: two cells past a tile; 40: rows end on a
# tile, columns inside one
@pytest.mark.parametrize("n", [4, 6, 34, 40, 66])
@pytest.mark.parametrize("kind", ["random", "quarter", "tiny"])
@pytest.mark.parametrize("prec", [ag.PREC_FP64_PLAIN, ag.PREC_FP32_MIXED])
def test_flags_and_windings_match_oracle(n, kind, prec):
    phi = fields(kind, n, n)
    if prec == ag.PREC_FP32_MIXED:
        phi = phi.astype(np.complex64).astype(np.complex128)
    p = params(n, prec)
    with ag.Lattice(p) as lat:
        lat.upload(phi, np.zeros_like(phi))
        snap, _ = lat.download(phidot=False)
        for which in (7, 6, 1):
            counts = lat.classify_cells(which)
            flags, want = axo.classify_cells(params(n), snap, which, 0)
            assert np.array_equal(counts, want)
            assert np.array_equal(lat.defect_flags(), flags)
        assert np.array_equal(lat.string_winding(), axo.string_winding(params(n), snap))


def test_components_at_the_edge_of_single_precision():
    """FP64 fields whose components straddle FP32's range: some decided in
    FP32 with a component taken for zero, some unknown there."""
    n = 12
    rng = np.random.default_rng(4)
    phi = fields("random", n, 1)
    phi.real *= 10.0 ** rng.choice([0, -20, -36, -39, -60, -300, 30, 37, 39, 200], (n, n, n))
    phi.imag *= 10.0 ** rng.choice([0, -20, -36, -39, -60, -300, 30, 37, 39, 200], (n, n, n))
    phi[3, 4, 5] = 0.0
    phi[6, 6, :] = phi[6, 6, :].real  # zero imaginary parts
    p = params(n)
    flags, want = axo.classify_cells(p, phi, 7, 0)
    with ag.Lattice(p) as lat:
        lat.upload(phi, np.zeros_like(phi))
        assert np.array_equal(lat.classify_cells(7), want)
        assert np.array_equal(lat.defect_flags(), flags)
        assert np.array_equal(lat.string_winding(), axo.string_winding(p, phi))
