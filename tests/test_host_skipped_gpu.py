"""Host calls with proposals that are not evaluated, with term_x: the plan writes their
outputs from the pinned block (up to 256 proposals) or the staged arrays (above).  A
template outside its segment leaves logL alone, so dlogl is exactly -term_x, of this
call's term_x also where a recorded graph is replayed; bad input gives NaN.
"""
import numpy as np
import pytest

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
T, NFFT, NSEG = wl.T_YEAR, 512, 3


@pytest.fixture(scope="module")
def engine():
    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    yield eng
    eng.close()


@pytest.mark.parametrize("n", [1, 4, 33, 256, 257])
@pytest.mark.parametrize("precision", [gg.PREC_FP64, gg.PREC_MIXED])
def test_term_x_of_skipped_proposals(engine, precision, n):
    import torch

    rng = np.random.default_rng(n)
    f0s = np.array([1e-3, 4e-3, 1.1e-2])
    qmin = (f0s * T).astype(np.int32) - NFFT // 2
    C = np.array([wl.aenoise_ff((q + np.arange(NFFT)) / T) for q in qmin])
    d = [(rng.standard_normal(C.shape) + 1j * rng.standard_normal(C.shape)) * np.sqrt(C / 2) for _ in range(2)]
    engine.upload(wl.SegmentBank(T=T, NFFT=NFFT, qmin=qmin, dA=d[0], dE=d[1], invCA=1 / C, invCE=1 / C))
    dev = lambda x: torch.tensor(x, device="cuda")
    for call in range(4):  # the first records a graph of the shape
        seg = (np.arange(n) % NSEG).astype(np.int32)
        p = np.array([wl.draw_source(rng, f0s[s], 2e-22, 1e-17) for s in seg])
        tx = rng.normal(0, 5, n)
        bad, seg_bad, out = np.arange(n) % 5 == 1, np.arange(n) % 5 == 2, (np.arange(n) + call) % 5 == 0
        out &= ~bad & ~seg_bad
        p[bad, 1] = 1.5
        p[out, 0] += 1e6
        seg[seg_bad] = NSEG
        dl, ty, hh, st = engine.dlogl_host(seg, p, term_x=tx, precision=precision)
        np.testing.assert_array_equal(st[bad], 1)
        np.testing.assert_array_equal(st[seg_bad], 2)
        np.testing.assert_array_equal(st[out], 4)
        assert (st[~(bad | seg_bad | out)] == 0).all()
        for a in (dl, ty, hh):
            assert np.isnan(a[bad | seg_bad]).all()
        np.testing.assert_array_equal(dl[out], -tx[out])
        assert (ty[out] == 0).all() and (hh[out] == 0).all()
        got = [dev(np.zeros(n)) for _ in range(3)] + [dev(np.zeros(n, np.int32))]
        engine.dlogl_device(dev(seg), dev(p), *got, dev(tx), precision)
        torch.cuda.synchronize()
        for a, b in zip((dl, ty, hh, st), got):
            np.testing.assert_array_equal(a, b.cpu().numpy())
