"""The XYZ noise likelihood where it depends on the cancellation of the acceleration noise
in X + Y + Z: data that the models do not describe, from 0.1 mHz, and unequal link
levels, against extended precision (numpy's long double: 64 or 113 bits).

Tolerance: an entry of a bin's covariance carries a rounding of about one eps, which
its tr(C^-1 P) + log det C carries times 1 / lambda, lambda the smallest eigenvalue of
the correlation matrix (~1e-7 here).  The bins round on their own, so their sum is good
to 3 eps times the root of the sum of the squares; plus 1e-13 of the total.
"""
import numpy as np
import pytest

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
T, Q0 = wl.T_YEAR, 3145
L = np.longdouble


def _exact(f, lv, P):
    """Per bin: tr(C^-1 P) + log det C, and the correlation's smallest eigenvalue."""
    x = f / L(wl.FSTAR)
    c, s2 = np.cos(x), np.sin(x) ** 2
    acc = np.where(f < 0.01, L(2.81837551648e-19) / f ** 2 * (1 + (L(0.4e-3) / f) ** 2) * (1 + (f / L(8.0e-3)) ** 4), L(0))
    oms = L(4.39256635604e-16) * f ** 2 * (1 + (L(2.0e-3) / f) ** 4)
    a12, a21, a23, a32, a13, a31 = (lv[k] * acc for k in range(6))
    o12, o21, o23, o32, o13, o31 = (lv[6 + k] * oms for k in range(6))
    dia = [(o12 + o21 + o13 + o31) / 4 + (a12 + a13) + (a21 + a31) * c * c,
           (o23 + o32 + o21 + o12) / 4 + (a23 + a21) + (a32 + a12) * c * c,
           (o31 + o13 + o32 + o23) / 4 + (a31 + a32) + (a13 + a23) * c * c]
    off = [(o12 + o21) / 2 + 2 * (a12 + a21), (o13 + o31) / 2 + 2 * (a13 + a31), (o32 + o23) / 2 + 2 * (a32 + a23)]
    xx, yy, zz = (4 * s2 * v for v in dia)
    xy, xz, yz = (-2 * s2 * c * v for v in off)
    d2 = yy - xy * xy / xx
    t = yz - xy * xz / xx
    d3 = (zz - xz * xz / xx) - t * t / d2
    num = ((yy * zz - yz * yz) * P[0] + (zz * xx - xz * xz) * P[1] + (xx * yy - xy * xy) * P[2]
           + 2 * ((xz * yz - zz * xy) * P[3] + (xy * yz - xz * yy) * P[4] + (xy * xz - xx * yz) * P[5]))
    C = np.array([[xx, xy, xz], [xy, yy, yz], [xz, yz, zz]]).astype(float).transpose(2, 0, 1)
    s = np.sqrt(np.einsum("nii->ni", C))
    lam = np.linalg.eigvalsh(C / (s[:, :, None] * s[:, None, :]))[:, 0]
    return num / (xx * d2 * d3) + np.log(xx) + np.log(d2) + np.log(d3), lam


@pytest.mark.parametrize("N", [400, 4000])
@pytest.mark.parametrize("spread", [0.0, 0.13, 0.5, 1.0])  # decades
def test_mismatched_data(N, spread):
    from glass_gb300 import build

    build.build()
    rng = np.random.default_rng(int(N + 100 * spread))
    inst0, _ = wl.default_noise_params(T)
    lv = inst0 * 10 ** rng.uniform(-spread, spread, (12, 12))
    x = rng.standard_normal((3, 2 * N)) * 1e-20
    re, im = x[:, 0::2].astype(L), x[:, 1::2].astype(L)
    P = [re[a] * re[b] + im[a] * im[b] for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    f = (L(Q0) + np.arange(N).astype(L)) / L(T)
    eng = gg.Engine(0)
    try:
        eng.noise_setup(T, Q0, *x)
        got = eng.noise_logl_host(lv)
    finally:
        eng.close()
    for k in range(len(lv)):
        per, lam = _exact(f, lv[k].astype(L), P)
        ref = -per.sum() - 3 * N * np.log(2 * L("3.14159265358979323846264338327950288"))
        tol = 3 * 2.2e-16 * np.sqrt((per.astype(float) ** 2 / lam ** 2).sum()) + 1e-13 * abs(float(ref))
        assert abs(float(got[k] - ref)) <= tol, (k, float(got[k] - ref) / tol)
