"""String fits on either route of id_defects (a warp per cell for few cells,
eight lanes per cell with the last ones handed over for many) and with corner
phases that are no numbers: every fitted cell equal to the oracle's."""
import numpy as np
import pytest

import axion_grav_gb300 as ag
from oracle import axo
from tests.test_gpu_defects import fields, params

pytestmark = pytest.mark.gpu

COLS = [0, 1, 2, 3, 4, 5, 6, 7, 8, 10, 11]
WCOLS = [0, 1, 2, 3, 4, 5, 7, 8]


def gpu_fits(p, phi, phid):
    with ag.Lattice(p) as lat:
        lat.upload(phi, phid)
        lat.set_kernel_timing(True)
        _, _, _, cnt = lat.id_defects(1, 4.0)
        names = {k for k, l, _ in lat.kernel_timings() if l}
        S, W = lat.defect_lists(int(cnt[0]), int(cnt[1]))
    return cnt, S, W, names


# 6^3: a handful of cells; 34^3: a warp each, not a multiple of anything;
# 56^3 of noise: tens of thousands, so groups of eight lanes and the hand-over
@pytest.mark.parametrize("kind,n,many", [("random", 6, False), ("smooth", 34, False), ("random", 56, True)])
def test_string_fits_match_oracle(kind, n, many):
    phi = fields(kind, n, 9)
    rng = np.random.default_rng(2)
    phid = (0.1 * (rng.standard_normal((n, n, n)) + 1j * rng.standard_normal((n, n, n)))).astype(np.complex128)
    p = params(n)
    cnt, S, W, names = gpu_fits(p, phi, phid)
    assert cnt[0] > 0 and ("string_simplex" in names) == many
    pick = lambda m: np.sort(rng.choice(int(m), min(int(m), 500), replace=False))
    si, wi = pick(cnt[0]), pick(cnt[1])
    if many:  # the last cells of the list are among those handed over
        si = np.unique(np.concatenate([si, np.arange(int(cnt[0]) - 100, int(cnt[0]))]))
    fs, fw = axo.fit_cells(p, phi, phid, S[si, 11].astype(np.int64), W[wi, 8].astype(np.int64))
    assert np.array_equal(S[si][:, COLS], fs[:, COLS])
    assert np.array_equal(W[wi][:, WCOLS], fw[:, WCOLS])


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_string_fits_with_non_finite_sites(bad):
    n = 12
    phi = fields("random", n, 3)
    phi[2, 3, 4] = phi[7, 7, 0] = bad
    phi[5, 5, 5] = complex(0.3, bad)
    phid = np.zeros_like(phi)
    p = params(n)
    with np.errstate(all="ignore"):
        cnt, S, W, _ = gpu_fits(p, phi, phid)
        fs, fw = axo.fit_cells(p, phi, phid, S[:, 11].astype(np.int64), W[:, 8].astype(np.int64))
    assert np.array_equal(S[:, COLS], fs[:, COLS], equal_nan=True)
    assert np.array_equal(W[:, WCOLS], fw[:, WCOLS], equal_nan=True)
