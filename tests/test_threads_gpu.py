"""Transforms and wavelet calls of different sizes from several host threads at once, a
context each: every call succeeds and gives what it gives alone, bit for bit.  (The
shared-memory limit of a kernel belongs to the device, so a call must not lower it
under another thread's launch.)
"""
import threading

import numpy as np
import pytest

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def _wdm(precision, NF, NT):
    def make(eng):
        x = np.random.default_rng(NF + NT).standard_normal(NF * NT)
        return lambda: np.concatenate([eng.wdm_forward_host(NF, NT, x, precision), eng.wdm_inverse_host(NF, NT, x, precision)])

    return make


def _wavelet(precision, NF, NT):
    def make(eng):
        wdt = 15.0 * NF
        wdf, T = 1 / (2 * wdt), 15.0 * NF * NT
        kmin, kmax = 5 * NT, 60 * NT
        rng = np.random.default_rng(NT)
        p = np.array([wl.draw_source(rng, f, 1e-21, 1e-16, T) for f in rng.uniform(10 * wdf, 50 * wdf, 2)])
        eng.wavelet_setup(T, 0.0, NF, NT, wdt, wdf, kmin, kmax, nx=4.0)
        eng.wavelet_set_data(np.zeros((3, kmax - kmin)), np.full((3, 3, kmax - kmin), 1e40))
        return lambda: eng.wavelet_waveform_host(p, precision=precision)[1]

    return make


@pytest.mark.parametrize("calls,n", [
    ([_wdm(gg.PREC_FP64, 32, 18), _wdm(gg.PREC_FP64, 27, 54)], 1000),
    ([_wdm(gg.PREC_MIXED, 16, 32), _wdm(gg.PREC_MIXED, 64, 128)], 1000),
    ([_wdm(gg.PREC_FP64, 2048, 4096), _wdm(gg.PREC_FP64, 4096, 4096)], 3),
    ([_wavelet(gg.PREC_FP64, 512, 16), _wavelet(gg.PREC_FP64, 512, 1024)] * 2, 2000),
    ([_wavelet(gg.PREC_MIXED, 512, 16), _wavelet(gg.PREC_MIXED, 512, 1024)] * 2, 2000),
], ids=["wdm-fp64", "wdm-mixed", "wdm-large", "wavelet-fp64", "wavelet-mixed"])
def test_sizes_side_by_side(calls, n):
    from glass_gb300 import build

    build.build()
    engines = [gg.Engine(0) for _ in calls]
    try:
        fns = [make(eng) for make, eng in zip(calls, engines)]
        ref = [f() for f in fns]
        bad, start = [], threading.Barrier(len(fns))

        def work(f, r):
            start.wait()
            try:
                for k in range(n):
                    if not np.array_equal(f(), r):
                        bad.append(f"call {k} differs")
                        return
            except Exception as e:
                bad.append(repr(e))

        threads = [threading.Thread(target=work, args=a) for a in zip(fns, ref)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad, bad
    finally:
        for e in engines:
            e.close()
