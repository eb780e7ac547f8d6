"""The double-float re-evaluation at every template size, on banks of 512 to 8192 bins
(whose width sets the launch's shared memory), for one proposal and for more than a
launch holds at once, clipped by the segment's edges and per channel.

Tolerance 1e-10 of max(1, |h|^2): double-float rounding is 4e-15 of the sums, whose
scale is |h| |r|, and the carrier phase of both forms is good to 1e-11 rad.
"""
import numpy as np
import pytest
import torch

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
T = wl.T_YEAR


@pytest.fixture(scope="module")
def engine():
    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    yield eng
    eng.close()


@pytest.mark.parametrize("NFFT", [512, 1024, 2048, 4096, 8192])
def test_every_size(engine, NFFT):
    rng = np.random.default_rng(NFFT)
    f0s = [1.2e-3, 4e-3, 1.7e-2]
    qmin, rA, rE, iC, src = [], [], [], [], []
    for f0 in f0s:
        p = wl.draw_source(rng, f0, 2e-22, 1e-17)
        q = int(p[0]) - NFFT // 2
        C = wl.aenoise_ff((max(q, 1) + np.arange(NFFT)) / T)
        qmin.append(q), iC.append(1.0 / C), src.append(p)
        for r in (rA, rE):
            r.append((rng.standard_normal(NFFT) + 1j * rng.standard_normal(NFFT)) * np.sqrt(C / 2))
    qmin[1] += NFFT // 2 - 20
    qmin[2] -= NFFT // 2 - 20
    engine.upload(wl.SegmentBank(T=T, NFFT=NFFT, qmin=np.array(qmin, np.int32), dA=np.array(rA), dE=np.array(rE),
                                 invCA=np.array(iC), invCE=np.array(iC) * 1.3))
    src = np.array(src)
    dev = lambda x: torch.tensor(x, device="cuda")
    try:
        for N in [n for n in (32, 64, 128, 256, 512, 1024, 2048, 4096) if n <= NFFT]:
            engine.set_template_size(N)
            for n in (1, 3, 200):
                seg = (np.arange(n) % 3).astype(np.int32)
                p = src[seg].copy()
                p[:, 3] += 0.01 * np.arange(n) / n
                _, ref, hh, st = engine.dlogl_host(seg, p, precision=gg.PREC_FP64)
                assert (st == 0).all()
                tol = 1e-10 * np.maximum(1.0, hh)
                engine.set_mixed_tolerance(1e-15)
                n0 = engine.mixed_reevaluated()
                _, ty, h, st = engine.dlogl_host(seg, p, precision=gg.PREC_MIXED)
                assert engine.mixed_reevaluated() - n0 >= n  # (a first call of a shape records a graph)
                dl, ch, t2 = dev(np.zeros(n)), dev(np.zeros((n, 2))), dev(np.zeros(n))
                engine.dlogl_channels_device(dev(seg), dev(p), dl, ch, t2)
                torch.cuda.synchronize()
                engine.set_mixed_tolerance(1e-3)
                assert (st == 0).all()
                assert (np.abs(ty - ref) <= tol).all() and (np.abs(h - hh) <= tol).all(), (N, n)
                assert (np.abs(t2.cpu().numpy() - ref) <= tol).all()
                assert (np.abs(ch.cpu().numpy().sum(1) - ref) <= tol).all()
    finally:
        engine.set_mixed_tolerance(1e-3)
        engine.set_template_size(0)
