"""The fused step's kernels give the same bits whichever one the dispatch picks:
the TMA tiles (on lattices their tile divides and, for FP32, on ragged ones),
and the plain stencil kernel with its columns of planes."""
import numpy as np
import pytest

import axion_grav_gb300 as ag
from oracle import axo
from tests.test_gpu_evolve import make_params, random_state, run_gpu

pytestmark = pytest.mark.gpu


def step(p, st, tile=None, nsteps=3):
    def fn(lat):
        if tile is not None:
            lat.set_tile(tile)
        lat.set_kernel_timing(True)
        lat.leapfrog(1.5, 0.02, nsteps, True, True)
        lat.synchronize()
        return [k for k, l, _ in lat.kernel_timings() if l == nsteps]
    return run_gpu(p, st, fn)


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a[:4], b[:4]) if x is not None)


# N above 80 and a multiple of 4 runs the ragged TMA tiles: one site over a
# tile edge (100 = 3 x 32 + 4), one short (92, 124 = 4 x 32 - 4), ragged in y
# only of the 8-row tile (132 = 16 x 8 + 4), a single wave (128)
@pytest.mark.parametrize("gw,n", [(ag.GW_UIJ, n) for n in (84, 92, 96, 100, 124, 128, 132, 164)] +
                         [(ag.GW_NONE, n) for n in (228, 236, 256)])
def test_tma_tiles_equal_plain_kernel(gw, n, monkeypatch):
    p = make_params(n, ag.PREC_FP32_MIXED, gw)
    st = random_state(n, n, 0.05)
    tma = step(p, st)
    assert tma[4] == ["fused_kd_fp32_%s" % ("uij" if gw else "phi")]
    monkeypatch.setenv("AXG_FUSED_PLAIN", "1")
    plain = step(p, st)
    assert plain[4] == ["fused_kd_fp32_%s_plain" % ("uij" if gw else "phi")]
    assert same(tma, plain)


# the default below the switch to TMA, and sizes TMA cannot address; one and
# four planes a CTA, the last CTA's planes cut off (66, 90)
@pytest.mark.parametrize("gw", [ag.GW_NONE, ag.GW_UIJ])
@pytest.mark.parametrize("prec", [ag.PREC_FP32_MIXED, ag.PREC_FP64_FUSED])
@pytest.mark.parametrize("n", [4, 10, 32, 64])
def test_plain_kernel_equals_tma_tile(n, prec, gw):
    p = make_params(n, prec, gw)
    st = random_state(n, n, 0.05)
    plain = step(p, st)
    assert len(plain[4]) == 1
    if n >= 32:
        for tile in (1, 7, 8, 10):
            assert same(step(p, st, tile), plain)
    else:  # a one-step reference in numpy float64
        f64 = step(make_params(n, ag.PREC_FP64_PLAIN, gw), st)
        for a, b in zip(plain[:4], f64[:4]):
            if a is not None:
                tol = 0 if prec == ag.PREC_FP64_FUSED else 1e-4
                assert np.max(np.abs(a - b)) <= tol * np.max(np.abs(b))


@pytest.mark.parametrize("n", [66, 90, 102])
def test_plain_kernel_planes_against_fp64(n):
    """FP32 lattices TMA cannot address: the four-plane columns against FP64."""
    st = random_state(n, n, 0.05)
    a = step(make_params(n, ag.PREC_FP32_MIXED, ag.GW_UIJ), st)
    b = step(make_params(n, ag.PREC_FP64_PLAIN, ag.GW_UIJ), st)
    assert a[4] == ["fused_kd_fp32_uij_plain"]
    for x, y in zip(a[:4], b[:4]):
        # three steps of rounding 6e-8 in fields whose Laplacian terms are a few times their size
        assert np.max(np.abs(x - y)) <= 2e-5 * np.max(np.abs(y))


# operands the integer products refuse (zeros, subnormals, infinities, huge
# and tiny fields) next to ones they take, for a power-of-two 2 dx and not
@pytest.mark.parametrize("dspa", [0.5, 0.32])
@pytest.mark.parametrize("prec", [ag.PREC_FP64_PLAIN, ag.PREC_FP64_FUSED])
def test_fp64_products_at_the_edges_of_their_window(prec, dspa):
    n = 12
    p = make_params(n, prec, ag.GW_UIJ, dspa=dspa)
    phi, phid, u, ud = random_state(n, 3, 0.05)
    u[:, 3:6] = 0.0
    ud[:, :, 2:4] = 0.0
    phid[2] = 0.0
    phi[5, 5:8] = phi[5, 5, 5]  # vanishing differences
    u[0, 7] *= 1e-310
    u[1, 7] = 1e300
    u[2, 7] *= 1e-160
    phi[8, 8, 8] = 1e-200 + 1e-320j
    u[3, 9, 9, 9] = np.inf
    ref = tuple(a.copy() for a in (phi, phid, u, ud))
    with np.errstate(all="ignore"):
        axo.leapfrog(p, *ref, None, 1.5, 0.02, 3, True, True)
        got = run_gpu(p, (phi, phid, u, ud), lambda lat: lat.leapfrog(1.5, 0.02, 3, True, True))
    for a, b in zip(got[:4], ref):
        assert np.array_equal(a, b, equal_nan=True)
