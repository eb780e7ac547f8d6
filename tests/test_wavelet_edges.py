"""The FP64 wavelet layers where their forms change: one transform for two layers
or one, the grid's first and last layer, pixel counts that are not a multiple of
four, one to three layers, and a year-long grid, where the carrier phase reaches
1e6 rad.

Tolerance 1e-10 of the channel's largest value, as the other wavelet tests: a
rounding step of the carrier phase is worth 1e-10 rad there, and the carrier and
the delayed times keep the reference's order of operations; the transforms' own
rounding is ~1e-14.
"""
import ctypes

import numpy as np
import pytest

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
REL = 1e-10
_D = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def engine():
    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    yield eng
    eng.close()


@pytest.mark.parametrize("NF,NT,jmin,NL", [(64, 32, 0, 2), (64, 32, 0, 1), (64, 32, 62, 3), (64, 32, 63, 2), (64, 32, 9, 3),
                                           (64, 32, 10, 3), (48, 64, 7, 5), (16, 8, 3, 2), (16, 4, 4, 3),
                                           (1024, 2048, 101, 2)])
def test_layer_transforms(engine, port, NF, NT, jmin, NL):
    lib = gg.load_library()
    win = gg.wdm_window(NL + 1, NT)
    x = np.random.default_rng(NT + jmin).standard_normal(NT * (NL + 1))
    ref = port.wdm_by_layers(NF, NT, jmin, NL, win, x.copy())
    w = (ctypes.c_int * 64)(NF, NT)
    lib.wavelet_transform_timefreq_by_layers(ctypes.cast(w, ctypes.c_void_p), jmin, NL, win.ctypes.data_as(_D),
                                             x.ctypes.data_as(_D))
    assert np.abs(x - ref).max() < REL * np.abs(ref).max()


@pytest.mark.parametrize("NF,NT,t0,A", [(1024, 2048, 0.0, 0.0), (1024, 2048, 4.2e7, 1e-4), (512, 54, 0.0, 0.0),
                                        (768, 1536, 0.0, 0.0)])
def test_waveforms_on_long_grids(engine, port, NF, NT, t0, A):
    wdt = 15.0 * NF
    wdf, T = 1 / (2 * wdt), 15.0 * NF * NT
    kmin, kmax = 5 * NT, 400 * NT
    rng = np.random.default_rng(NF + NT)
    f0 = np.concatenate([[(20 + 1e-3) * wdf, 30.5 * wdf], rng.uniform(10 * wdf, 390 * wdf, 4)])
    params = np.array([wl.draw_source(rng, f, 1e-21, 1e-16, T) for f in f0])
    engine.wavelet_setup(T, t0, NF, NT, wdt, wdf, kmin, kmax, A=A, nx=4.0)
    info, xyz, st = engine.wavelet_waveform_host(params)
    assert (st == 0).all()
    for i, p in enumerate(params):
        lst_o, ref, j, nl = port.wavelet_waveform(p, T, t0, NF, NT, wdt, wdf, kmin, kmax, A, 4.0)
        assert (info[i, 0], info[i, 1]) == (j, nl)
        lst = engine.wavelet_list(info[i])
        np.testing.assert_array_equal(lst, lst_o)
        for c in range(3):
            assert np.abs(xyz[i, c, : len(lst)] - ref[c][lst]).max() < REL * np.abs(ref[c][lst]).max(), (i, c)
