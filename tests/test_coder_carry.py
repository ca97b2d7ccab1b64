"""Carries out of the encoder's accumulator into words that are already stored.  A sequence that keeps the
interval around its middle leaves a run of ones behind those words, which the next symbol turns into a
carry or settles: every symbol of the run is the one that holds the middle.  Streams against the oracle."""
import ctypes

import numpy as np
import pytest


def P(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def straddling(cdf, lead, run):
    """`lead`, then `run` symbols that each keep the middle of the range inside the interval."""
    low, high, out = 0, (1 << 32) - 1, []
    for i in range(len(lead) + run):
        span = high - low + 1
        bound = lambda s: low + ((span * int(cdf[s]) if s < len(cdf) - 1 else span << 16) >> 16)
        s = lead[i] if i < len(lead) else max(k for k in range(len(cdf) - 1) if bound(k) < 1 << 31)
        low, high = bound(s), bound(s + 1) - 1
        out.append(s)
        while (low ^ high) < 1 << 31 or (low >> 30 == 1 and high >> 30 == 2):
            sub = low & (1 << 31) if (low ^ high) < 1 << 31 else 1 << 30
            low, high = (low - sub) * 2, (high - sub) * 2 + 1
    return out


@pytest.mark.parametrize("lp", [4, 9, 33])
@pytest.mark.parametrize("run", [1, 5, 11, 16, 22, 40, 90, 200])
def test_runs_around_the_middle(oracle, host_model, run, lp):
    rng = np.random.default_rng(run)
    for _ in range(20):
        cdf = np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), size=lp - 2, replace=False)), [65535]))
        cdf = cdf.astype(np.uint16)
        lead = [int(v) for v in rng.integers(0, lp - 1, size=int(rng.integers(0, 4)))]
        head = straddling(cdf, lead, run)
        for tail in ([0], [lp - 2], [0] * 5, [lp - 2] * 5, []):
            sym = np.array((head + tail)[:256], dtype=np.int8)
            want = oracle.encode_stream(cdf, sym)
            cap = 2 * len(sym) + 8
            out = np.zeros(cap + 8, dtype=np.uint8)
            n = host_model.hm_encode_stream(P(cdf), lp, P(sym), len(sym), P(out), cap, 3)
            assert n == len(want) and (out[:n] == want).all()
