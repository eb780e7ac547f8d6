"""The noise likelihoods' split of a batch over CTAs: about four per SM of the device
that runs it where the batch allows, and never more partial sums than the buffer
kept for that many models holds.  The rules are host functions of the library (C++
names), called without a GPU.
"""
import ctypes

import pytest

import glass_gb300 as gg


@pytest.fixture(scope="module")
def rules():
    from glass_gb300 import build

    build.build()
    lib = gg.load_library()

    def get(name, nargs, res):
        f = getattr(lib, f"_ZN5glass{len(name)}{name}E" + "i" * nargs)
        f.argtypes, f.restype = [ctypes.c_int] * nargs, res
        return f

    return (get("noise_bins_per_thread", 3, ctypes.c_int), get("noise_partials", 3, ctypes.c_size_t),
            get("noise_wv_layers_per_cta", 4, ctypes.c_int), get("noise_wv_partials", 4, ctypes.c_size_t))


@pytest.mark.parametrize("sms", [19, 148, 152])
def test_split_follows_the_device(rules, sms):
    bins, room, layers, wv_room = rules
    up = lambda a, b: (a + b - 1) // b
    for cap in (1, 64, 128, 2048):
        for n in sorted({k for k in (1, 2, 3, 7, cap // 2, cap - 1, cap) if 1 <= k <= cap}):
            for N in (1, 127, 128, 129, 2048, 2049, 15360, 100001):
                R = bins(N, n, sms)
                ctas = n * up(N, 128 * R)
                assert 1 <= R <= 16 and ctas <= room(N, cap, sms)
                assert R == 16 or n * up(N, 256 * R) < 4 * sms  # a split by half was not enough
                assert R == 1 or ctas >= 4 * sms
            for Nl, Nc in ((1, 1), (5, 3), (460, 128), (512, 4096), (1000, 9000), (333, 61)):
                L = layers(Nl, Nc, n, sms)
                ctas = n * up(Nl, L)
                assert 1 <= L <= 64 and ctas <= wv_room(Nl, Nc, cap, sms)
                assert L == 1 or ctas >= 4 * sms or L == min(64, max(1, 4096 // Nc))
