"""The FP64 WDM transforms where their forms change: layers in pairs with an odd
or even number of layers, the smallest grids, odd factors in the four-step split
(lone rows and columns among the mirrored pairs), NT not a multiple of four (one
layer per transform), unaligned series, and the spectrum forms.

Tolerance 1e-12 of the largest value: the transforms round at ~1e-16 per factor of
two on both sides.
"""
import ctypes

import numpy as np
import pytest

import glass_gb300 as gg

pytestmark = pytest.mark.gpu
REL = 1e-12
GRIDS = [(2, 8), (3, 8), (4, 12), (2, 64), (3, 64), (4, 64), (9, 16), (27, 64), (27, 16), (32, 18), (27, 54), (6, 256),
         (12, 4096), (96, 384), (81, 96)]


@pytest.fixture(scope="module")
def engine():
    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    yield eng
    eng.close()


def _close(a, b):
    assert np.abs(a - b).max() < REL * np.abs(b).max()


@pytest.mark.parametrize("NF,NT", GRIDS)
def test_grids(engine, port, NF, NT):
    rng = np.random.default_rng(NF * NT)
    ND = NF * NT
    x = rng.standard_normal(ND)
    win = port.wdm_window(NF, NT)
    _close(engine.wdm_forward_host(NF, NT, x), port.wdm_forward(NF, NT, win, x))
    _close(engine.wdm_inverse_host(NF, NT, x), port.wdm_inverse(NF, NT, win, x))


@pytest.mark.parametrize("NF,NT", [(4, 64), (27, 16), (32, 18)])
def test_spectrum_forms_and_unaligned_series(engine, port, NF, NT):
    import torch

    rng = np.random.default_rng(NF + NT)
    ND = NF * NT
    win = port.wdm_window(NF, NT)
    w = rng.standard_normal(ND)
    freq = port.wdm_to_freq(NF, NT, win, w)
    lib = engine.lib
    args = (engine._ctx, gg.PREC_FP64, NF, NT, 0.0, gg.WDM_NX)
    for off in (0, 1):  # 16-byte aligned, and not
        buf = torch.zeros(2 * ND + 8, dtype=torch.float64, device="cuda")
        a, b = buf[off:off + ND], buf[ND + 4 + off:]
        f = torch.zeros(ND + 2 + off, dtype=torch.float64, device="cuda")[off:]
        a.copy_(torch.from_numpy(w))
        torch.cuda.synchronize()
        assert lib.glass_gpu_wdm_to_freq(*args, ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(f.data_ptr())) == 0
        torch.cuda.synchronize()
        _close(f.cpu().numpy(), freq)
        assert lib.glass_gpu_wdm_from_freq(*args, ctypes.c_void_p(f.data_ptr()), ctypes.c_void_p(a.data_ptr())) == 0
        torch.cuda.synchronize()
        _close(a.cpu().numpy(), port.wdm_from_freq(NF, NT, win, freq))
        x = torch.from_numpy(rng.standard_normal(ND)).cuda()
        b = b[:ND]
        b.copy_(x)
        torch.cuda.synchronize()
        engine.wdm_forward_device(NF, NT, b, b)
        torch.cuda.synchronize()
        coef = port.wdm_forward(NF, NT, win, x.cpu().numpy())
        _close(b.cpu().numpy(), coef)
        engine.wdm_inverse_device(NF, NT, b, b)
        torch.cuda.synchronize()
        _close(b.cpu().numpy(), port.wdm_inverse(NF, NT, win, coef))  # no identity for an odd NF
