"""Spectra of fields and accumulators far from one, and of very small and very
large lattice spacings: scaling by a power of two scales the sums of squares by
its square, whichever numbers single precision could square."""
import numpy as np
import pytest

import axion_grav_gb300 as ag
from oracle import axo
from tests.test_gpu_shell_sums import gw_params, noise
from tests.test_gpu_spectrum import params as spec_params, state

pytestmark = pytest.mark.gpu


# The transforms hold values as pairs of floats, so a power of two commutes with
# them; a term of a sum is off by at most 2^-45 of itself, and all are positive.
TOL = 1e-12
SHIFTS = [-80, -62, -45, 55, 66, 80]


def field_spectrum(n, precision, deg, shift):
    phi, phid = state(n, 11 * n + deg)
    if precision == ag.PREC_FP32_MIXED:
        phi, phid = (a.astype(np.complex64).astype(np.complex128) for a in (phi, phid))
    with ag.Lattice(spec_params(n, precision, degrade_spec=deg)) as lat:
        lat.upload(phi, np.ldexp(1.0, shift) * phid)
        lat.classify_cells(7)
        return lat.spectrum_estimation(3.0)


# 16 to 64: the transforms in pairs of floats; 24: cuFFT's in FP64
@pytest.mark.parametrize("n,deg", [(16, 0), (64, 0), (64, 1), (24, 0)])
@pytest.mark.parametrize("precision", [ag.PREC_FP64_PLAIN, ag.PREC_FP32_MIXED])
def test_field_spectrum_scales(n, deg, precision):
    w, pw, cv, ct = field_spectrum(n, precision, deg, 0)
    for s in SHIFTS:
        _, gpw, gcv, gct = field_spectrum(n, precision, deg, s)
        np.testing.assert_array_equal(gct, ct)
        np.testing.assert_allclose(np.ldexp(gcv, -2 * s), cv, rtol=TOL, err_msg=str(s))
        np.testing.assert_allclose(np.ldexp(gpw, -2 * s), pw, rtol=1e-8, atol=1e-10 * np.max(np.abs(pw)))


# dx^3 is a factor of the window and of the field
@pytest.mark.parametrize("n,deg", [(16, 0), (32, 1), (112, 0), (24, 0)])
@pytest.mark.parametrize("dspa", [1e-8, 2.0 ** -10, 3e5])
def test_field_spectrum_of_any_spacing(n, deg, dspa):
    phi, phid = state(n, n)
    p = spec_params(n, degrade_spec=deg, dspa=dspa)
    flags, _ = axo.classify_cells(p, phi, 7, 0)
    w, pw, cv, ct, md = axo.spectrum_estimation(p, phid, flags, 3.0)
    with ag.Lattice(p) as lat:
        lat.upload(phi, phid)
        lat.classify_cells(7)
        gw, gpw, gcv, gct = lat.spectrum_estimation(3.0)
    np.testing.assert_array_equal(gct, ct)
    np.testing.assert_allclose(gcv, cv, rtol=1e-10)
    np.testing.assert_allclose(gpw, pw, rtol=1e-8, atol=1e-10 * np.max(np.abs(pw)))


@pytest.mark.parametrize("shift", [-66, 60])
def test_covariance_scales(shift):
    n = 16
    phi, phid = state(n, 3)
    cov = {}
    for s in (0, shift):
        with ag.Lattice(spec_params(n)) as lat:
            lat.upload(phi, np.ldexp(1.0, s) * phid)
            lat.classify_cells(7)
            lat.spectrum_estimation(3.0)
            cov[s], _ = lat.spectrum_covariance(4, 4, 0.05)
    want = cov[0]
    np.testing.assert_allclose(np.ldexp(cov[shift], -4 * shift), want, rtol=1e-8, atol=1e-10 * np.max(np.abs(want)))


# accumulators as pairs of floats (16, 32, and every FP32-mixed size) and FP64
# ones (18), with the edges of the shell walk: one bin, some, the most
@pytest.mark.parametrize("n", [16, 18, 32])
@pytest.mark.parametrize("nb", [1, 25, 256])
@pytest.mark.parametrize("precision", [ag.PREC_FP64_PLAIN, ag.PREC_FP64_FUSED, ag.PREC_FP32_MIXED])
def test_green_shells_scale(n, nb, precision):
    phi, phid = 1.0 + noise(n, n, 0.2), noise(n, n + 1, 0.1)
    p = gw_params(n, ag.PREC_FP64_PLAIN, ag.GW_GREEN, nb)
    acc = np.zeros((4, n, n, n), np.complex128)
    axo.symplectic_integration(p, phi.copy(), phid.copy(), None, None, acc, 2.0, 2.4, 0.4)
    w, pw, nu, de = axo.grav_spec_estimation(p, acc)
    with ag.Lattice(gw_params(n, precision, ag.GW_GREEN, nb)) as lat:
        for s in [0] + SHIFTS:
            lat.upload_gw_green(np.ldexp(1.0, s) * acc)
            _, _, gnu, gde = lat.grav_spec_estimation(2.4)
            np.testing.assert_array_equal(gde, de)
            # an accumulator is held to 2^-48, its square to 2^-46
            np.testing.assert_allclose(np.ldexp(gnu, -2 * s), nu, rtol=TOL, err_msg=str(s))


def test_uij_powers_near_the_largest_float():
    """One plane wave along z: the power of an entry is a float, the sum of a
    shell need not be one."""
    n, m, tau = 16, 3, 0.5
    p = gw_params(n, ag.PREC_FP64_PLAIN, ag.GW_UIJ, 25)
    u = np.zeros((6, n, n, n))
    u[1] = np.cos(2 * np.pi * m * np.arange(n) / n)[:, None, None]
    ud = np.zeros_like(u)
    k = m * 2 * np.pi / n / p.dspa
    # an entry's power is 2 A^2 (n^3/2)^2 (1 + k^2 tau^2): 0.8 of the largest float
    u *= np.sqrt(0.8 * np.finfo(np.float32).max / 2 / (n ** 3 / 2) ** 2 / (1 + (k * tau) ** 2))
    u = u.astype(np.float32).astype(np.float64)
    w, pw, nu, de = axo.uij_grav_spec(p, u, ud, tau)
    with ag.Lattice(gw_params(n, ag.PREC_FP32_MIXED, ag.GW_UIJ, 25)) as lat:
        lat.upload(np.ones((n, n, n), np.complex128), np.zeros((n, n, n), np.complex128))
        lat.upload_uij(u, ud)
        _, _, gnu, gde = lat.grav_spec_estimation(tau)
    np.testing.assert_array_equal(gde, de)
    assert np.all(np.isfinite(gnu))
    assert np.all(np.abs(gnu - nu) <= 1e-5 * np.max(nu))


@pytest.mark.parametrize("precision", [ag.PREC_FP64_PLAIN, ag.PREC_FP32_MIXED])
@pytest.mark.parametrize("n", [16, 32])
def test_green_shells_of_uneven_entries(n, precision):
    """Entries from 2^-110 to 2^60 side by side, a power of two for every |k|^2:
    whatever a sample of them says, each is summed with its own digits."""
    phi, phid = 1.0 + noise(n, n, 0.2), noise(n, n + 1, 0.1)
    p = gw_params(n, ag.PREC_FP64_PLAIN, ag.GW_GREEN, 256)
    acc = np.zeros((4, n, n, n), np.complex128)
    axo.symplectic_integration(p, phi.copy(), phid.copy(), None, None, acc, 2.0, 2.4, 0.4)
    k = np.round(np.fft.fftfreq(n) * n).astype(int)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    rng = np.random.default_rng(n)
    # numbers per entry: with acc of order one, within FP32's range as pairs
    acc *= np.ldexp(1.0, rng.choice([-110, -90, -60, -40, 0, 0, 30, 60], k2.max() + 1))[k2]
    w, pw, nu, de = axo.grav_spec_estimation(p, acc)
    with ag.Lattice(gw_params(n, precision, ag.GW_GREEN, 256)) as lat:
        lat.upload_gw_green(acc)
        _, _, gnu, gde = lat.grav_spec_estimation(2.4)
    np.testing.assert_array_equal(gde, de)
    # at 2^-110 a pair keeps 2^-149 of one: 39 bits, 2^-38 in the square
    np.testing.assert_allclose(gnu, nu, rtol=2.0 ** -36)


@pytest.mark.parametrize("shift", [-80, 0, 66])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_field_spectrum_of_one_wave(shift, axis):
    """All power in one wave, the rest of the spectrum its transform's rounding."""
    n = 32
    phi = np.full((n, n, n), 1.0 + 0j)
    z = np.exp(2j * np.pi * 5 * np.arange(n) / n)
    phid = np.ldexp(1.0, shift) * np.broadcast_to(z.reshape([n if a == axis else 1 for a in range(3)]), (n, n, n)).copy()
    p = spec_params(n)
    flags, _ = axo.classify_cells(p, phi, 7, 0)
    w, pw, cv, ct, md = axo.spectrum_estimation(p, phid, flags, 3.0)
    with ag.Lattice(p) as lat:
        lat.upload(phi, phid)
        lat.classify_cells(7)
        _, gpw, gcv, gct = lat.spectrum_estimation(3.0)
    np.testing.assert_array_equal(gct, ct)
    top = np.max(cv)
    assert top > 0 and np.all(np.abs(gcv - cv) <= 1e-11 * top)
