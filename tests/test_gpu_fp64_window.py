"""FP64 steps whose operands lie outside the integer products' window throughout
(a coefficient of zero, a real field, fields at rest and no u_ij) and run on
hardware products: the oracle's bits."""
import numpy as np
import pytest

import axion_grav_gb300 as ag
from oracle import axo
from tests.test_gpu_evolve import make_params, random_state, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["free", "real", "imaginary", "rest", "fact1"])
@pytest.mark.parametrize("gw", [ag.GW_NONE, ag.GW_UIJ])
@pytest.mark.parametrize("prec", [ag.PREC_FP64_PLAIN, ag.PREC_FP64_FUSED])
@pytest.mark.parametrize("n,dspa", [(12, 0.5), (34, 0.32), (64, 0.5)])
def test_bits_outside_the_window(n, dspa, prec, gw, kind):
    kw = dict(potential=ag.POT_QUARTIC, vev=1.0, **{"lambda": 0.0 if kind == "free" else 1.0})
    p = make_params(n, prec, gw, dspa=dspa, **kw)
    phi, phid, u, ud = random_state(n, 5, 0.05)
    if kind == "real":
        phi, phid = phi.real + 0j, phid.real + 0j
    if kind == "imaginary":
        phi, phid = 1j * phi.imag, 1j * phid.imag
    if kind == "rest":
        phid, u, ud = 0 * phid, 0 * u, 0 * ud
    t, dt = (0.04, 0.04) if kind == "fact1" else (1.5, 0.02)  # fact1 = (1 - dt/t) / (1 + dt/t)
    ref = tuple(a.copy() for a in (phi, phid, u, ud))
    axo.leapfrog(p, ref[0], ref[1], ref[2] if gw else None, ref[3] if gw else None, None, t, dt, 3, False, True)
    got = run_gpu(p, (phi, phid, u, ud), lambda lat: lat.leapfrog(t, dt, 3, False, True))
    for a, b in zip(got[:4], ref):
        if a is not None:
            assert np.array_equal(a, b)
