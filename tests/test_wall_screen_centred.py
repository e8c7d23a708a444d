"""The FP32 screen of the wall-direction search in its centred form
(position_wall in axion_grav_gb300/csrc/axg_defects.cu; defects_3d.f90:
1135-1160): chi2 = sum (q_i . d0)^2 + m min(c . d0, 0)^2 with the points'
mean c and q_i = p_i - c.  A direction is left out when its FP32 value less
wall_err of it exceeds the smallest one plus wall_err of that, so the FP64
minimum is never left out if each FP32 value is within wall_err of the FP64
one.  Restated in numpy (float32; the kernel's fused multiply-adds round
less) on random points, points near a plane and points close together."""
import numpy as np

from tests.test_wall_screen import _fp64, _grid


def wall_err(f):
    return 1e-5 * np.sqrt(f) + 2e-6 * f + 1e-10


def _fp32(pp, m, d0):
    f32 = np.float32
    g = d0.astype(f32)
    cen = pp[:m].sum(axis=0) / m
    q, c = (pp[:m] - cen).astype(f32), cen.astype(f32)
    w = np.minimum(c[0] * g[:, 0] + c[1] * g[:, 1] + c[2] * g[:, 2], f32(0))
    f = np.zeros(d0.shape[0], f32)
    for i in range(m):
        d = q[i, 0] * g[:, 0] + q[i, 1] * g[:, 1] + q[i, 2] * g[:, 2]
        f = f + d * d
    return (f32(m) * w) * w + f


def test_centred_screen_within_wall_err():
    rng = np.random.default_rng(17)
    d0 = _grid()
    worst = 0.0
    for trial in range(3000):
        m = int(rng.integers(3, 13))
        pp = rng.uniform(-0.5, 0.5, (m, 3))
        if trial % 4 == 1:  # near a plane through the cell
            n = rng.normal(size=3)
            n /= np.linalg.norm(n)
            pp = np.clip(pp - np.outer(pp @ n, n) * rng.uniform(0.98, 1.0), -0.4999999, 0.4999999)
        if trial % 4 == 2:  # every point near a cube corner
            pp = np.sign(rng.normal(size=(m, 3))) * rng.uniform(0.49, 0.4999999, (m, 3))
        if trial % 4 == 3:  # crossings close to one corner of the cell: every direction has a small chi2
            pp = 0.5 * np.sign(rng.normal(size=3)) * (1 - 10.0 ** rng.uniform(-6, -1) * rng.random((m, 3)))
        f, exact = _fp32(pp, m, d0).astype(np.float64), _fp64(pp, m, d0)
        # the FP64 form S - m w^2 itself cancels to ~1e-15 of S <= 9
        worst = max(worst, np.max((np.abs(f - exact) - 1e-14) / wall_err(f)))
    assert worst < 1.0, worst
