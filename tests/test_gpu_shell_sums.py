"""Shell sums walked along ky, at the edges of their row runs (lattices of a few
sites, odd multiples of two, past a run of 32) and with one, some and the most
bins (32 copies of a bin down to 8), against the oracle."""
import numpy as np
import pytest

import axion_grav_gb300 as ag
from oracle import axo
from tests.test_gpu_spectrum import params as spec_params, state

pytestmark = pytest.mark.gpu


def gw_params(n, precision, gw, nb):
    return ag.default_params(ngrid=n, precision=precision, gw_mode=gw, dspa=0.75, sigma_cr=1.0, kappa=0.1,
                             tau_cr=1.0, a_now=1.0, num_bin_grav=nb, gw_log_bins=12, seed=3, flags=7)


def noise(n, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    return scale * (rng.standard_normal((n, n, n)) + 1j * rng.standard_normal((n, n, n)))


# White fields, so that an entry's power is at most a few times the largest
# mean of a shell.  An FP32 transform is off by ~sqrt(log2 n^3) 2^-24 < 3e-7 of
# the field's rms, its power by twice that: 1e-5 of the largest mean is 15 times
# it.  The FP64 transforms leave 1e-12.
@pytest.mark.parametrize("n", [4, 6, 16, 34, 66])
@pytest.mark.parametrize("nb", [1, 25, 256])
@pytest.mark.parametrize("precision,tol", [(ag.PREC_FP32_MIXED, 1e-5), (ag.PREC_FP64_FUSED, 1e-11)])
def test_uij_shells(n, nb, precision, tol):
    rng = np.random.default_rng(n)
    u, ud = (rng.standard_normal((6, n, n, n)).astype(np.float32).astype(np.float64) for _ in range(2))
    w, pw, nu, de = axo.uij_grav_spec(gw_params(n, ag.PREC_FP64_PLAIN, ag.GW_UIJ, nb), u, ud, 2.6)
    with ag.Lattice(gw_params(n, precision, ag.GW_UIJ, nb)) as lat:
        lat.upload(np.ones((n, n, n), np.complex128), np.zeros((n, n, n), np.complex128))
        lat.upload_uij(u, ud)
        gw, gpw, gnu, gde = lat.grav_spec_estimation(2.6)
    np.testing.assert_array_equal(gde, de)
    top = np.max(nu / np.maximum(de, 1))
    assert np.all(np.abs(gnu - nu) <= tol * top * de)


@pytest.mark.parametrize("n", [6, 34])
@pytest.mark.parametrize("nb", [1, 256])
@pytest.mark.parametrize("precision", [ag.PREC_FP64_PLAIN, ag.PREC_FP64_FUSED])
def test_green_shells(n, nb, precision):
    phi, phid = 1.0 + noise(n, n, 0.2), noise(n, n + 1, 0.1)
    p = gw_params(n, precision, ag.GW_GREEN, nb)
    acc = np.zeros((4, n, n, n), np.complex128)
    axo.symplectic_integration(p, phi.copy(), phid.copy(), None, None, acc, 2.0, 2.4, 0.4)
    w, pw, nu, de = axo.grav_spec_estimation(p, acc)
    with ag.Lattice(p) as lat:
        lat.upload(phi, phid)
        lat.symplectic_integration(2.0, 2.4, 0.4)
        gw, gpw, gnu, gde = lat.grav_spec_estimation(2.4)
    np.testing.assert_array_equal(gde, de)
    # the accumulators agree to 1e-10 of their largest, the sums of squares to twice that
    assert np.all(np.abs(gnu - nu) <= 1e-9 * np.max(nu / np.maximum(de, 1)) * de)


# the window matrix, directly below m = 104 and by prefix sums from there, and the
# device's table of it: one bin, more than a warp of bins, degraded transforms
@pytest.mark.parametrize("n,nb,deg", [(6, 1, 0), (6, 3, 0), (16, 4, 1), (34, 17, 0), (40, 9, 1), (80, 40, 0), (102, 12, 0), (104, 12, 0), (112, 40, 0)])
def test_window_matrix(n, nb, deg):
    phi, phid = state(n, 5 * n)
    p = spec_params(n, num_bin=nb, degrade_spec=deg)
    flags, cnt = axo.classify_cells(p, phi, 7, 0)
    w, pw, cv, ct, md = axo.spectrum_estimation(p, phid, flags, 3.0)
    with ag.Lattice(p) as lat:
        lat.upload(phi, phid)
        lat.classify_cells(7)
        gw, gpw, gcv, gct = lat.spectrum_estimation(3.0)
    np.testing.assert_array_equal(gct, ct)
    np.testing.assert_allclose(gcv, cv, rtol=1e-10)
    np.testing.assert_allclose(gpw, pw, rtol=1e-8, atol=1e-10 * np.max(np.abs(pw)))


# The Green step's z pass contracts and accumulates what it transforms from 128^3
# on (lines of radix 8 8 2 and 8 8 4); cuFFT's transforms accumulate from memory.
# Both are FP32: a source spectrum is off by < 3e-7 of its largest value, the
# contraction of six by a few times that, so accumulators by 5e-6 of the largest.
@pytest.mark.parametrize("n", [64, 128, 256])
@pytest.mark.parametrize("compat", [ag.COMPAT_REF, ag.COMPAT_INTENDED])
def test_green_accumulation_inside_the_z_pass(monkeypatch, n, compat):
    rng = np.random.default_rng(n)
    phi = (rng.standard_normal((n, n, n), np.float32) + 1j * rng.standard_normal((n, n, n), np.float32))
    phi = phi.astype(np.complex128)
    out = {}
    for ff in ("1", "0"):
        monkeypatch.setenv("AXG_FFT_FF", ff)
        p = gw_params(n, ag.PREC_FP32_MIXED, ag.GW_GREEN, 25)
        p.compat = compat
        with ag.Lattice(p) as lat:
            lat.upload(phi, np.zeros_like(phi))
            lat.set_kernel_timing(True)
            lat.symplectic_integration(2.0, 2.4, 0.2)
            lat.synchronize()
            out[ff] = lat.download_gw_green() if n < 256 else None, lat.grav_spec_estimation(2.4)[2]
            fused = any(k == "gw_z_accumulate_fp32" for k, _, _ in lat.kernel_timings())
        assert fused == (ff == "1" and n >= 128)
    monkeypatch.delenv("AXG_FFT_FF")
    a, b = out["1"], out["0"]
    if n < 256:  # every entry: the Nyquist rows' mirrors and k = 0 too
        assert np.max(np.abs(a[0] - b[0])) <= 5e-6 * np.max(np.abs(b[0]))
    np.testing.assert_allclose(a[1], b[1], rtol=2e-5, atol=1e-10 * np.max(b[1]))
