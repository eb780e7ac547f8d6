"""The plan kernel where its forms change: the bandwidth rule's FP32 estimate at
the poles, near zeros of its sine, at the ends of its range of frequencies and
amplitudes and at power-of-two boundaries; angles beyond the sine table; batches
that leave part of a CTA idle, fill one, and go beyond one wave.

Tolerances: FP64 1e-10 of max(1, |term|) against the oracle (a template of another
size, or another placement, is off by far more); mixed 1e-3, its default
tolerance; positions in a batch 1e-12 relative, the summation order's.
"""
import numpy as np
import pytest

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
T = wl.T_YEAR
NFFT = 4096
FSTAR = 299792458.0 / (2 * np.pi * 2.5e9)


@pytest.fixture(scope="module")
def engine():
    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    yield eng
    eng.close()


def _bank(rng, f0s):
    qmin, rA, rE, iC = [], [], [], []
    for f0 in f0s:
        q = int(f0 * T) - NFFT // 2
        C = wl.aenoise_ff((max(q, 1) + np.arange(NFFT)) / T)
        qmin.append(q), iC.append(1.0 / C)
        for r in (rA, rE):
            r.append((rng.standard_normal(NFFT) + 1j * rng.standard_normal(NFFT)) * np.sqrt(C / 2))
    return wl.SegmentBank(T=T, NFFT=NFFT, qmin=np.array(qmin, np.int32), dA=np.array(rA), dE=np.array(rE),
                          invCA=np.array(iC), invCE=np.array(iC) * 1.3)


def _source(rng, f0, lnA=np.log(1e-22), costh=0.3, psi=0.4, phi=1.0, fdT2=0.01):
    return np.array([f0 * T, costh, phi, lnA, 0.2, psi, rng.uniform(0, 6.28), fdT2])


def _cases():
    rng = np.random.default_rng(7)
    out = []
    for costh in (1.0, -1.0, 1 - 1e-9, 1 - 1e-7, -1 + 1e-5, 0.0):
        for f0 in (1e-3, 2.3e-2):
            out.append(_source(rng, f0, costh=costh))
    for f0 in (np.pi * FSTAR * (1 - 1e-3), np.pi * FSTAR * (1 + 1e-5), 1e-4, 3e-2):
        out.append(_source(rng, f0))
    for lnA in (-100.0, -81.0, -79.0, -52.0, -49.0, -47.5):
        out.append(_source(rng, 5e-3, lnA=lnA))
    for k in range(40):  # amplitudes across the size boundaries
        out.append(_source(rng, 6e-3, lnA=-50.5 + 0.05 * k))
    for ang in (-40.0, 1e4, 3e5):
        out.append(_source(rng, 4e-3, psi=ang, phi=-ang))
    out.append(_source(rng, 4e-3, fdT2=40.0))
    out.append(_source(rng, 4e-3, fdT2=-700.0))
    return np.array(out)


def test_sizes_and_constants(engine, port):
    rng = np.random.default_rng(3)
    params = _cases()
    seg = np.arange(len(params), dtype=np.int32)
    bank = _bank(rng, params[:, 0] / T)
    engine.upload(bank)
    rA, rE = bank.interleaved()
    ref = np.array([port.dlogl_term(p, T, NFFT, int(bank.qmin[s]), rA[s], rE[s], bank.invCA[s], bank.invCE[s])[:2]
                    for s, p in zip(seg, params)])
    scale = np.maximum(1.0, np.abs(ref[:, 0]))
    _, ty, hh, st = engine.dlogl_host(seg, params, precision=gg.PREC_FP64)
    assert (st == 0).all()
    assert (np.abs(ty - ref[:, 0]) / scale).max() < 1e-10
    np.testing.assert_allclose(hh, ref[:, 1], rtol=1e-9)
    _, tm, hm, st = engine.dlogl_host(seg, params, precision=gg.PREC_MIXED)
    assert (st == 0).all()
    assert (np.abs(tm - ref[:, 0]) / scale).max() < 1e-3
    np.testing.assert_allclose(hm, ref[:, 1], rtol=1e-4, atol=1e-30)  # FP32 sums: (h|h) of 1e-41 underflows


@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 2431, 2433, 4865])
def test_any_batch_gives_the_same(engine, n):
    rng = np.random.default_rng(5)
    f0s = np.array([1e-3, 4e-3, 1.1e-2])
    engine.upload(_bank(rng, f0s))
    base = np.array([_source(rng, f0s[k % 3], lnA=-52 + 0.4 * (k % 7), costh=0.9 - 0.2 * (k % 9)) for k in range(63)])
    one = [engine.dlogl_host(np.array([k % 3], np.int32), base[k : k + 1], precision=gg.PREC_FP64)[1][0] for k in range(63)]
    idx = np.arange(n) % 63
    for prec, tol in ((gg.PREC_FP64, 1e-12), (gg.PREC_MIXED, 1e-4)):
        _, ty, _, st = engine.dlogl_host((idx % 3).astype(np.int32), base[idx], precision=prec)
        assert (st == 0).all()
        np.testing.assert_allclose(ty, np.array(one)[idx], rtol=tol, atol=tol)


@pytest.mark.parametrize("n", [1, 5, 255, 256, 257])
def test_host_calls_of_small_batches(engine, n):
    """Up to 256 proposals the kernels read and write pinned memory in place: the
    same bits as the device entry, whose kernels they are, for new arrays in every
    call of one shape (the first records a graph), with and without term_x, and
    for proposals that are skipped."""
    import torch

    rng = np.random.default_rng(n)
    f0s = np.array([1e-3, 4e-3, 1.1e-2])
    engine.upload(_bank(rng, f0s))
    dev = lambda x: torch.tensor(x, device="cuda")
    for prec in (gg.PREC_FP64, gg.PREC_MIXED):
        for k in range(4):
            seg = (np.arange(n) % 3).astype(np.int32)
            p = np.array([_source(rng, f0s[s], lnA=rng.uniform(-52, -49), costh=rng.uniform(-1, 1)) for s in seg])
            if k == 2:
                p[0, 1] = 1.5  # not a cosine: status 1
                p[-1, 0] += 1e6  # outside its segment: status 4
            tx = rng.normal(0, 5, n) if k % 2 else None
            got = engine.dlogl_host(seg, p, term_x=tx, precision=prec)
            out = [dev(np.zeros(n)) for _ in range(3)] + [dev(np.zeros(n, np.int32))]
            engine.dlogl_device(dev(seg), dev(p), *out, None if tx is None else dev(tx), prec)
            torch.cuda.synchronize()
            for a, b in zip(got, out):
                np.testing.assert_array_equal(a, b.cpu().numpy())


@pytest.mark.parametrize("NFFT", [1024, 4096])
def test_chains_in_a_captured_graph(engine, NFFT):
    """The chained launches under stream capture, with the size kernels' side branches
    (banks beyond 1024 bins) and with and without the re-evaluation's conditional
    node: a replay gives the direct call's bits, for new inputs in the same arrays."""
    import torch

    rng = np.random.default_rng(NFFT)
    f0s = np.array([1e-3, 4e-3, 1.1e-2])
    bank = _bank(rng, f0s)
    if NFFT < 4096:
        off = (4096 - NFFT) // 2
        bank = wl.SegmentBank(T=T, NFFT=NFFT, qmin=(bank.qmin + off).astype(np.int32),
                              **{k: np.ascontiguousarray(getattr(bank, k)[:, off:off + NFFT])
                                 for k in ("dA", "dE", "invCA", "invCE")})
    engine.upload(bank)
    dev = lambda x: torch.tensor(x, device="cuda")
    s = torch.cuda.Stream()
    try:
        for prec in (gg.PREC_FP64, gg.PREC_MIXED):
            for n in (20, 700):
                seg = (np.arange(n) % 3).astype(np.int32)
                ps = [np.array([_source(rng, f0s[k], lnA=rng.uniform(-51, -48), costh=rng.uniform(-1, 1)) for k in seg])
                      for _ in range(3)]
                p, sg = dev(ps[0]), dev(seg)
                out = [dev(np.zeros(n)) for _ in range(3)] + [dev(np.zeros(n, np.int32))]
                ref = []
                for q in ps:
                    p.copy_(dev(q))
                    engine.dlogl_device(sg, p, *out, None, prec)
                    torch.cuda.synchronize()
                    ref.append([o.clone() for o in out])
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s):
                    engine.set_stream(torch.cuda.current_stream().cuda_stream)
                    engine.dlogl_device(sg, p, *out, None, prec)
                engine.set_stream(None)
                for q, r in zip(ps, ref):
                    p.copy_(dev(q))
                    for o in out:
                        o.zero_()
                    torch.cuda.synchronize()
                    g.replay()
                    torch.cuda.synchronize()
                    for a, b in zip(out, r):
                        assert torch.equal(a, b)
    finally:
        engine.set_stream(None)
