"""The FP64 slow part, spectral unit and F-statistic where their forms change:
arm phases on both sides of the sinc series' limits (low and high frequency,
above f*), carrier arguments beyond the sine table's range, batches whose last
unit holds idle groups at every template size, and F-statistic cells at every
filter size in counts that leave groups of a warp idle.

Tolerances: 1e-10 of max(1, |term|) against the oracle (every rounding of the
~1e6 rad carrier phase is worth ~1e-10 rad, and both follow the reference's
order there); F-statistic 1e-9 (its filters are exact quarter turns, the
oracle's differ from them by that phase rounding).
"""
import math

import numpy as np
import pytest

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


def _bank(rng, port, f0s, NFFT, amp=1e-22, fdot=1e-17):
    qmin, rA, rE, iC, src = [], [], [], [], []
    for f0 in f0s:
        p = wl.draw_source(rng, f0, amp, fdot)
        q = int(p[0]) - NFFT // 2
        C = wl.aenoise_ff((q + np.arange(NFFT)) / T)
        qmin.append(q), src.append(p), iC.append(1.0 / C)
        for r in (rA, rE):
            r.append((rng.standard_normal(NFFT) + 1j * rng.standard_normal(NFFT)) * np.sqrt(C / 2))
    bank = wl.SegmentBank(T=T, NFFT=NFFT, qmin=np.array(qmin, np.int32), dA=np.array(rA), dE=np.array(rE),
                          invCA=np.array(iC), invCE=np.array(iC) * 1.3)
    return bank, np.array(src)


def _check(engine, port, bank, seg, params):
    rA, rE = bank.interleaved()
    ref = np.array([port.dlogl_term(p, T, bank.NFFT, int(bank.qmin[s]), rA[s], rE[s], bank.invCA[s], bank.invCE[s])[:2]
                    for s, p in zip(seg, params)])
    dl, ty, hh, st = engine.dlogl_host(seg, params, precision=gg.PREC_FP64)
    assert (st == 0).all()
    assert (np.abs(ty - ref[:, 0]) / np.maximum(1.0, np.abs(ref[:, 0]))).max() < 1e-10
    np.testing.assert_allclose(hh, ref[:, 1], rtol=1e-9)


@pytest.mark.parametrize("f0", [2e-4, 3.7e-3, 3.9e-3, 1.9e-2, 6e-2])
def test_arm_phase_ranges(engine, port, f0):
    rng = np.random.default_rng(int(f0 * 1e6))
    bank, src = _bank(rng, port, [f0] * 3, 2048)
    engine.upload(bank)
    _check(engine, port, bank, np.arange(3, dtype=np.int32), src)


@pytest.mark.parametrize("fdT2", [1e5, 4e6])
def test_carrier_beyond_the_sine_table(engine, port, fdT2):
    # pi fdot t^2 reaches 3e5 rad, and 1.3e7, where the library's sincos takes over inside a template
    rng = np.random.default_rng(3)
    bank, src = _bank(rng, port, [5e-3] * 2, 1024, fdot=fdT2 / T**2)
    engine.upload(bank)
    _check(engine, port, bank, np.arange(2, dtype=np.int32), src)


@pytest.mark.parametrize("N,n", [(32, 1), (32, 5), (64, 3), (128, 1), (128, 9), (256, 1), (256, 5), (512, 3), (1024, 1),
                                 (2048, 2), (4096, 1)])
def test_idle_groups_per_size(engine, port, N, n):
    rng = np.random.default_rng(N + n)
    NFFT = max(N, 256)
    bank, src = _bank(rng, port, [3e-3, 8e-3], NFFT)
    engine.upload(bank)
    seg = (np.arange(n) % 2).astype(np.int32)
    params = src[seg] + rng.standard_normal((n, 8)) * 1e-3
    params[:, [1, 4]] = np.clip(params[:, [1, 4]], -0.99, 0.99)
    engine.set_template_size(N)
    try:
        _, ty, hh, st = engine.dlogl_host(seg, params, precision=gg.PREC_FP64)
    finally:
        engine.set_template_size(0)
    assert (st == 0).all()
    for i, (s, p) in enumerate(zip(seg, params)):
        h = port.waveform(p, N, T)
        j0 = int(p[0]) - N // 2 - int(bank.qmin[s])
        k = np.arange(max(0, -j0), min(N, NFFT - j0))
        term = h2 = 0.0
        for d, w, c in ((bank.dA, bank.invCA, 3), (bank.dE, bank.invCE, 4)):
            z = (h[c][0::2] + 1j * h[c][1::2])[k]
            r, w = d[s][k + j0], w[s][k + j0]
            term += ((2 * (r.conj() * z).real - np.abs(z) ** 2) * w).sum()
            h2 += 2 * (np.abs(z) ** 2 * w).sum()
        assert abs(ty[i] - term) < 1e-10 * max(1.0, h2)
        assert abs(hh[i] - h2) < 1e-9 * h2


@pytest.mark.parametrize("fdot,n", [(0.0, 1), (0.0, 70), (1e-14, 3), (3e-13, 5), (3e-12, 2), (2e-11, 1)])
def test_fstat_sizes_and_idle_groups(engine, port, fdot, n):
    rng = np.random.default_rng(n)
    NFFT = 4096
    bank, src = _bank(rng, port, [2e-3, 9e-3], NFFT)
    engine.upload(bank)
    seg = (np.arange(n) % 2).astype(np.int32)
    f0 = (bank.qmin[seg] + rng.uniform(0, NFFT, n)) / T
    cells = np.stack([f0, np.full(n, fdot), np.arccos(rng.uniform(-0.95, 0.95, n)), rng.uniform(0, 2 * math.pi, n)], 1)
    rA, rE = bank.interleaved()
    ref = port.fstat_batch(T, NFFT, bank.qmin, rA, rE, bank.invCA, seg, cells)
    ll, fp, st = engine.fstat_host(seg, cells)
    assert (st == 0).all()
    np.testing.assert_allclose(ll, ref[:, 0], rtol=1e-9)
    np.testing.assert_allclose(fp[:, 0], ref[:, 1], rtol=1e-8)
    d = np.abs(fp[:, 1:] - ref[:, 2:])
    assert np.minimum(d, np.abs(d - 2 * math.pi)).max() < 1e-7


@pytest.mark.parametrize("N", [32, 64, 128, 256, 512, 1024, 2048, 4096])
def test_small_batches(engine, port, N):
    """Batches around the counts up to which a proposal has a cluster or a CTA, and 32
    samples a CTA, to themselves, against the packed form of a larger batch: 1e-12 of max(1, |h|^2)
    (sums of 2N products in another order: 1e-16 sqrt(2N) |w| |h|)."""
    import torch

    rng = np.random.default_rng(N)
    bank, src = _bank(rng, port, [1e-3, 4e-3, 2e-2], max(1024, N))
    bank.qmin[1] += max(1024, N) // 2 - 12  # clipped by the segment's edge
    engine.upload(bank)
    engine.set_template_size(N)
    try:
        seg = np.arange(400, dtype=np.int32) % 3
        _, ref, hh, st = engine.dlogl_host(seg, src[seg], precision=gg.PREC_FP64)
        assert (st[seg != 1] == 0).all()
        tol = 1e-12 * np.maximum(1.0, hh)
        for n in (1, 2, 5, 9, 10, 19, 30, 31, 38, 76, 152, 153, 303, 304, 305):
            _, ty, h, s2 = engine.dlogl_host(seg[:n], src[seg[:n]], precision=gg.PREC_FP64)
            assert (s2 == st[:n]).all()
            assert (np.abs(ty - ref[:n]) <= tol[:n]).all() and (np.abs(h - hh[:n]) <= tol[:n]).all()
        dev = lambda x: torch.tensor(x, device="cuda")
        dl, ch, ty = dev(np.zeros(7)), dev(np.zeros((7, 2))), dev(np.zeros(7))
        engine.dlogl_channels_device(dev(seg[:7]), dev(src[seg[:7]]), dl, ch, ty, precision=gg.PREC_FP64)
        torch.cuda.synchronize()
        assert (np.abs(ty.cpu().numpy() - ref[:7]) <= tol[:7]).all()
        ok = st[:7] == 0
        assert (np.abs(ch.cpu().numpy().sum(1) - ref[:7])[ok] <= tol[:7][ok]).all()
    finally:
        engine.set_template_size(0)
