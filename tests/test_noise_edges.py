"""Noise-model likelihoods at the edges of their launch rules and of the fast
cell: bin and cell counts around the CTA sizes, batches from one model to many,
a foreground whose exponential changes fast along the bins, and covariances
that are not positive (the general elimination, NaN as in the reference).

Tolerance 1e-10 of |logL|, as the other noise tests: the inverse's form against
the reference's exp(log|cofactor| - log det), whose rounding (~2e-14 of each
entry) the near-degenerate covariance amplifies.
"""
import numpy as np
import pytest

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
T = wl.T_YEAR
REL = 1e-10


@pytest.fixture(scope="module")
def engine():
    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    yield eng
    eng.close()


@pytest.mark.parametrize("N,n", [(1, 1), (127, 3), (129, 1), (2047, 2), (2049, 5), (300, 700), (4100, 130)])
def test_xyz_sizes(engine, port, N, n):
    rng = np.random.default_rng(N + n)
    q = int(2e-3 * T)
    inst0, sgal0 = wl.default_noise_params(T)
    X, Y, Z = wl.xyz_from_covariance(rng, port.noise_covariance(T, q / T, N, inst0, sgal0))
    inst = inst0 * np.exp(rng.uniform(-0.3, 0.3, (n, 12)))
    sgal = sgal0 + rng.uniform(-0.2, 0.2, (n, 5))
    sgal[::3, 4] = np.log(1e-7)  # a step of many e-folds between a thread's bins
    sgal[::3, 3] = np.log((q + 0.5 * N) / T)
    sgal[1::5, 1] = np.log(1.02 * q / T / 10)  # 10 f1 inside the band
    engine.noise_setup(T, q, X, Y, Z)
    for g in (None, sgal):
        ref = port.noise_logl(T, q / T, X, Y, Z, inst, g)
        np.testing.assert_allclose(engine.noise_logl_host(inst, g), ref, rtol=REL)


@pytest.mark.parametrize("nch", [1, 2])
@pytest.mark.parametrize("N,n", [(1, 1), (129, 2), (2049, 40)])
def test_channel_sizes(engine, port, nch, N, n):
    rng = np.random.default_rng(N + n + nch)
    q = int(3e-3 * T)
    inst0, sgal0 = wl.default_noise_params(T)
    d = rng.standard_normal((2, 2 * N)) * np.sqrt(wl.aenoise_ff(q / T))
    inst = inst0 * np.exp(rng.uniform(-0.3, 0.3, (n, 12)))
    sgal = sgal0 + rng.uniform(-0.2, 0.2, (n, 5))
    engine.noise_setup_channels(T, q, d[0], d[1] if nch == 2 else None)
    for g in (None, sgal):
        ref = port.noise_logl_channels(T, q / T, list(d[:nch]), inst, g)
        np.testing.assert_allclose(engine.noise_logl_host(inst, g), ref, rtol=REL)


def test_covariance_that_is_not_positive(engine, port):
    rng = np.random.default_rng(5)
    N, q = 200, int(4e-3 * T)
    inst0, sgal0 = wl.default_noise_params(T)
    X, Y, Z = wl.xyz_from_covariance(rng, port.noise_covariance(T, q / T, N, inst0, sgal0))
    inst = np.tile(inst0, (5, 1))
    inst[1] *= -1.0  # negative definite: an odd number of negative pivots
    inst[2, 6:8] = -3 * wl.NOISE_SOMS0  # indefinite
    inst[3, 7] = np.nan
    engine.noise_setup(T, q, X, Y, Z)
    with np.errstate(all="ignore"):
        ref = port.noise_logl(T, q / T, X, Y, Z, inst)
    got = engine.noise_logl_host(inst)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.isnan(ref[[1, 2, 3]]).all()
    np.testing.assert_allclose(got[[0, 4]], ref[[0, 4]], rtol=REL)


@pytest.mark.parametrize("NT,Q,layers,n", [(256, 1, 3, 2), (256, 256, 70, 1), (2048, 16, 33, 3), (2048, 64, 130, 90)])
def test_wavelet_sizes(engine, port, NT, Q, layers, n):
    rng = np.random.default_rng(NT + Q + n)
    NF, lmin = 1024, 60
    df = 1.0 / (2 * 15.0 * NF)
    inst0, sgal0 = wl.default_noise_params(T)
    C6 = np.array([port.noise_covariance(T, (lmin + j) * df, 1, inst0, sgal0)[0] for j in range(layers)]) / (NF * NT)
    X, Y, Z = wl.wavelet_noise_data(rng, C6, NT)
    mod = wl.galaxy_modulation_like(NT // Q)
    engine.noise_wavelet_setup(NF, NT, df, lmin, Q, X, Y, Z, mod)
    P = port.noise_coarse_stats(NT, Q, X, Y, Z)
    inst = inst0 * np.exp(rng.uniform(-0.3, 0.3, (n, 12)))
    sgal = sgal0 + rng.uniform(-0.2, 0.2, (n, 5))
    for mode in (0, 1, 2):
        ref = port.noise_wavelet_logl(NF, NT, df, lmin, P, Q, inst, sgal, mode, mod if mode == 2 else None)
        np.testing.assert_allclose(engine.noise_wavelet_logl_host(inst, sgal, mode), ref, rtol=REL)
