"""The WDM transforms to and from a spectrum keep every layer to itself, as the
reference's layer-by-layer transforms do: a layer's coefficients follow from its own
bins alone, a bin's value from the layers that reach it.  So a layer at 1e12 times the
others' size, or one with a NaN, leaves the others as accurate as they are without it.

Tolerance 1e-12 of the layer's own largest value (of the bins' that no loud layer
reaches): each side rounds at ~1e-16 per factor of two.
"""
import ctypes

import numpy as np
import pytest

import glass_gb300 as gg

pytestmark = pytest.mark.gpu
REL = 1e-12
GRIDS = [(8, 64), (9, 16), (16, 24), (32, 18), (2, 8), (3, 4096)]


@pytest.fixture(scope="module")
def engine():
    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    yield eng
    eng.close()


def _run(engine, name, NF, NT, x, nout):
    import torch

    a, b = torch.from_numpy(np.ascontiguousarray(x)).cuda(), torch.zeros(nout, dtype=torch.float64, device="cuda")
    assert getattr(engine.lib, name)(engine._ctx, gg.PREC_FP64, NF, NT, 0.0, gg.WDM_NX, ctypes.c_void_p(a.data_ptr()),
                                     ctypes.c_void_p(b.data_ptr())) == 0
    torch.cuda.synchronize()
    return b.cpu().numpy()


def _layers(w, NF, NT):
    """Rows: layer 0, 1 .. NF - 1, NF."""
    w = w.reshape(NF, NT)
    return [w[0, ::2], *w[1:], w[0, 1::2]]


@pytest.mark.parametrize("NF,NT", GRIDS)
@pytest.mark.parametrize("loud", [1e12, np.nan, np.inf])
def test_from_spectrum(engine, port, NF, NT, loud):
    rng = np.random.default_rng(NF * NT)
    win = port.wdm_window(NF, NT)
    base = rng.standard_normal(NF * NT + 2)
    for m in range(NF + 1):  # the bin at a layer's centre belongs to that layer alone
        freq = base.copy()
        freq[2 * (m * NT // 2)] = loud
        got = _layers(_run(engine, "glass_gpu_wdm_from_freq", NF, NT, freq, NF * NT), NF, NT)
        ref = _layers(port.wdm_from_freq(NF, NT, win, freq if loud == 1e12 else base), NF, NT)
        for q in range(NF + 1):
            if q == m and loud != 1e12:
                assert not np.isfinite(got[q]).any()
            else:
                assert np.abs(got[q] - ref[q]).max() <= REL * np.abs(ref[q]).max(), (m, q)


@pytest.mark.parametrize("NF,NT", GRIDS)
@pytest.mark.parametrize("loud", [1e12, np.nan, np.inf])
def test_to_spectrum(engine, port, NF, NT, loud):
    rng = np.random.default_rng(NF * NT)
    win = port.wdm_window(NF, NT)
    base = rng.standard_normal((NF, NT))
    h = NT // 2
    for m in range(NF + 1):
        w = base.copy()
        w[0 if m in (0, NF) else m, 1 if m == NF else 0] = loud
        got = _run(engine, "glass_gpu_wdm_to_freq", NF, NT, w, NF * NT + 2).reshape(-1, 2)
        ref = port.wdm_to_freq(NF, NT, win, (w if loud == 1e12 else base).ravel()).reshape(-1, 2)
        k = np.arange(NF * h + 1)
        out = (k < (m - 1) * h) | (k > (m + 1) * h)  # bins that layer m does not reach
        if out.any():
            assert np.abs(got[out] - ref[out]).max() <= REL * np.abs(ref[out]).max(), m
        if loud == 1e12:
            assert np.abs(got - ref).max() <= REL * np.abs(ref).max()
        else:
            assert not np.isfinite(got[min(max(m * h, 0), NF * h)]).all()
