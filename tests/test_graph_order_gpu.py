"""A captured graph of a large raw mixed batch (re-evaluation off) on wide segments: the
2048-point templates, on a side branch, end it, and the launch for all smaller sizes
must not start ahead of them.  A replay takes 0.96 of the same call in the stream, 1.01
with the two the other way round; both are timed in turn here.
"""
import numpy as np
import pytest

import glass_gb300 as gg
from glass_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
T, NFFT, N = wl.T_YEAR, 2048, 10000


def test_size_kernels_first():
    import torch

    from glass_gb300 import build

    build.build()
    eng = gg.Engine(0)
    rng = np.random.default_rng(1)
    f0s = np.array([1.2e-3, 4e-3, 1.1e-2])
    qmin = (f0s * T).astype(np.int32) - NFFT // 2
    C = np.array([wl.aenoise_ff((q + np.arange(NFFT)) / T) for q in qmin])
    d = [(rng.standard_normal(C.shape) + 1j * rng.standard_normal(C.shape)) * np.sqrt(C / 2) for _ in range(2)]
    eng.upload(wl.SegmentBank(T=T, NFFT=NFFT, qmin=qmin, dA=d[0], dE=d[1], invCA=1 / C, invCE=1 / C))
    seg = (np.arange(N) % 3).astype(np.int32)
    p = np.array([wl.draw_source(rng, f0s[s], 1e-20 * 10 ** rng.uniform(-0.5, 0.5), 1e-17) for s in seg])
    dev = lambda x: torch.tensor(x, device="cuda")
    seg, p = dev(seg), dev(p)
    out = [dev(np.zeros(N)) for _ in range(3)] + [dev(np.zeros(N, np.int32))]
    call = lambda: eng.dlogl_device(seg, p, *out, None, gg.PREC_MIXED)
    try:
        eng.set_mixed_tolerance(0.0)
        for _ in range(3):
            call()
        torch.cuda.synchronize()
        ref = [o.clone() for o in out]
        s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        eng.set_stream(s.cuda_stream)
        with torch.cuda.graph(g, stream=s):
            call()

        def ms(f):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with torch.cuda.stream(s):
                f()
                a.record()
                for _ in range(10):
                    f()
                b.record()
            torch.cuda.synchronize()
            return a.elapsed_time(b) / 10

        t = np.array([[ms(call), ms(g.replay)] for _ in range(9)])
        for a, b in zip(out, ref):
            assert torch.equal(a, b)
    finally:
        eng.set_stream(None)
        eng.close()
    stream, graph = np.median(t, 0)
    assert graph < 0.99 * stream, (graph, stream)
