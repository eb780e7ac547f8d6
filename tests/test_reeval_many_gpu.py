"""The double-float re-evaluation of more proposals than are resident at once: small
ones (a CTA each, at 512 points by number) and large ones (a cluster each) of one batch,
per channel, clipped by the segment's edges; and how its time grows with their number.
A proposal's results are the same bits as alone (whose accuracy the re-evaluation's edge
tests check at every size).
"""
import numpy as np
import pytest
import torch

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
T = wl.T_YEAR
F0 = [1.2e-3, 4e-3, 1.7e-2]


@pytest.fixture(scope="module")
def engine():
    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    yield eng
    eng.close()


def _upload(engine, rng, NFFT):
    qmin, rA, rE, iC = [], [], [], []
    for f0 in F0:
        q = int(f0 * T) - NFFT // 2
        C = wl.aenoise_ff((max(q, 1) + np.arange(NFFT)) / T)
        qmin.append(q), iC.append(1.0 / C)
        for r in (rA, rE):
            r.append((rng.standard_normal(NFFT) + 1j * rng.standard_normal(NFFT)) * np.sqrt(C / 2))
    engine.upload(wl.SegmentBank(T=T, NFFT=NFFT, qmin=np.array(qmin, np.int32), dA=np.array(rA), dE=np.array(rE),
                                 invCA=np.array(iC), invCE=np.array(iC) * 1.3))


@pytest.mark.parametrize("NFFT", [512, 1024, 8192])
def test_mixed_sizes(engine, NFFT):
    rng = np.random.default_rng(NFFT)
    _upload(engine, rng, NFFT)
    n = 1400
    seg = (np.arange(n) % 3).astype(np.int32)
    # amplitudes and chirps over the bandwidth rule's range, some near a segment's edge
    p = np.array([wl.draw_source(rng, F0[s], 10 ** rng.uniform(-23, -19.5), 10 ** rng.uniform(-18, -14.5)) for s in seg])
    p[::9, 0] += NFFT // 2 - 10
    dev = lambda x: torch.tensor(x, device="cuda")

    def run(seg, p):
        k = len(seg)
        out = [dev(np.zeros(k)) for _ in range(3)] + [dev(np.zeros(k, np.int32))]
        engine.dlogl_device(dev(seg), dev(p), *out, None, gg.PREC_MIXED)
        dl, ch, ty = dev(np.zeros(k)), dev(np.zeros((k, 2))), dev(np.zeros(k))
        engine.dlogl_channels_device(dev(seg), dev(p), dl, ch, ty)
        torch.cuda.synchronize()
        return [x.cpu().numpy() for x in (*out, dl, ch, ty)]

    try:
        engine.set_mixed_tolerance(1e-15)
        n0 = engine.mixed_reevaluated()
        got = run(seg, p)
        assert engine.mixed_reevaluated() - n0 > 2 * 1000
        for i in range(0, n, 13):
            for a, b in zip(got, run(seg[i:i + 1], p[i:i + 1])):
                np.testing.assert_array_equal(a[i:i + 1], b)
    finally:
        engine.set_mixed_tolerance(1e-3)


@pytest.mark.parametrize("N,most", [(32, 6.5), (512, 22.5)])
def test_time_of_many(engine, N, most):
    """3000 templates against 60, which are resident at once, of 32 and 512 points: 4 and
    20 times the time; 12 and 25 times where each takes a cluster (7 and 21 with
    114 clusters resident instead of 74)."""
    rng = np.random.default_rng(1)
    _upload(engine, rng, 1024)
    dev = lambda x: torch.tensor(x, device="cuda")
    us = {}
    try:
        engine.set_template_size(N)
        engine.set_mixed_tolerance(1e-15)
        engine.set_phase_timing(True)
        for n in (60, 3000):
            seg = (np.arange(n) % 3).astype(np.int32)
            p = dev(np.array([wl.draw_source(rng, F0[s], 2e-22, 1e-17) for s in seg]))
            out = [dev(np.zeros(n)) for _ in range(3)] + [dev(np.zeros(n, np.int32))]
            t = []
            for _ in range(20):
                engine.dlogl_device(dev(seg), p, *out, None, gg.PREC_MIXED)
                torch.cuda.synchronize()
                t.append(engine.last_phase_ms()[3])
            us[n] = np.median(t[5:])
    finally:
        engine.set_phase_timing(False)
        engine.set_mixed_tolerance(1e-3)
        engine.set_template_size(0)
    assert us[3000] < most * us[60], us


@pytest.mark.parametrize("n1024,n512,most", [(70, 23, 1.3), (74, 40, 1.41)])
def test_time_past_one_wave(engine, n1024, n512, most):
    """Templates of 1024 points that take most clusters, and some of 512, against the
    larger ones alone: 1.21 and 1.33 times the time where the 512-point ones follow as
    clusters, 1.39 and 1.49 where a CTA takes one after its share of a larger one."""
    rng = np.random.default_rng(2)
    _upload(engine, rng, 1024)
    dev = lambda x: torch.tensor(x, device="cuda")
    p, seg = {512: [], 1024: []}, {512: [], 1024: []}
    while len(p[512]) < n512 or len(p[1024]) < n1024:
        s = int(rng.integers(3))
        x = wl.draw_source(rng, F0[s], 10 ** rng.uniform(-23, -20), 1e-17)
        N = 2 * gg.ucb_bandwidth(wl.LARM, wl.FSTAR, x[0] / T, x[7] / T / T, x[1], np.exp(x[3]), T, 1024)
        if N in p:
            p[N].append(x), seg[N].append(s)
    us = {}
    try:
        engine.set_mixed_tolerance(1e-15)
        engine.set_phase_timing(True)
        for n in (n1024, n1024 + n512):
            k = n - n1024
            ds = dev(np.array(seg[1024][:n1024] + seg[512][:k], np.int32))
            dp = dev(np.array(p[1024][:n1024] + p[512][:k]))
            out = [dev(np.zeros(n)) for _ in range(3)] + [dev(np.zeros(n, np.int32))]
            t = []
            for _ in range(100):
                engine.dlogl_device(ds, dp, *out, None, gg.PREC_MIXED)
                torch.cuda.synchronize()
                t.append(engine.last_phase_ms()[3])
            us[n] = np.mean(sorted(t[10:])[:70])
    finally:
        engine.set_phase_timing(False)
        engine.set_mixed_tolerance(1e-3)
    assert us[n1024 + n512] < most * us[n1024], us
