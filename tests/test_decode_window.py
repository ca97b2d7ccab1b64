"""The decode loop's window and shift rule where they can go wrong, on the CPU against the oracle: a range of 2^31 at a multiple
of it (the one case that the shift by the interval's size leaves to the exact step), full ranges again and again, and streams
that end inside the window."""
import ctypes

import numpy as np
import pytest


def P(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def pair(oracle, host_model, cdfs, syms, cut=(None, None)):
    lp, n = len(cdfs[0]), len(syms[0])
    full = max(2, (lp - 2).bit_length())
    streams = [oracle.encode_stream(c, s)[:k] for c, s, k in zip(cdfs, syms, cut)]
    want = [oracle.decode_stream(c, s, n) for c, s in zip(cdfs, streams)]
    for off in (0, 1, 2, 3):
        big = np.full(off + sum(map(len, streams)) + 8, 0xA5, np.uint8)
        big[off:off + len(streams[0])] = streams[0]
        big[off + len(streams[0]):off + len(streams[0]) + len(streams[1])] = streams[1]
        at = big.ctypes.data + off
        for fl in range(2, full + 1):
            out = np.zeros(2 * n, np.uint8)
            assert host_model.hm_decode_pair(P(cdfs[0]), P(cdfs[1]), lp, ctypes.c_void_p(at), len(streams[0]),
                                             ctypes.c_void_p(at + len(streams[0])), len(streams[1]), n, P(out), 5 + off, fl) == 0
            assert (out[0::2] == want[0]).all() and (out[1::2] == want[1]).all(), (off, fl)
        for i in range(2):
            out = np.zeros(n, np.uint8)
            host_model.hm_decode_stream(P(cdfs[i]), lp, ctypes.c_void_p(at + (len(streams[0]) if i else 0)), len(streams[i]), n, P(out), 9)
            assert (out == want[i]).all(), (off, i)
    return want


@pytest.mark.parametrize("before", [2208, 2209, 2210, 4419])
def test_a_range_of_half_of_all_values_at_a_multiple_of_it(oracle, host_model, before):
    # symbol 0 has 45,136 of 2^16 shares: by symbols 0 alone the 2,210th, 4,420th, ... leave a size of exactly 2^31 at 0
    rng = np.random.default_rng(before)
    cdf = np.array([0, 45136, 50000, 60000, 65000, 65535], np.uint16)
    first = np.concatenate((np.zeros(before, np.int8), rng.integers(0, 5, 40).astype(np.int8), np.zeros(200, np.int8)))
    first[before] = 0
    other = rng.integers(0, 5, len(first)).astype(np.int8)
    want = pair(oracle, host_model, [cdf, cdf], [first, other])
    assert (want[0] == first).all() and (want[1] == other).all()


@pytest.mark.parametrize("share,second,zeros", [(35107, 10873, 16), (33903, 15341, 63), (34067, 13388, 130)])
def test_the_same_within_a_sub_chunk(oracle, host_model, share, second, zeros):
    # symbol 2 leaves a range at 0, `zeros` symbols 0 after it one of 2^31 there
    rng = np.random.default_rng(share)
    cdf = np.array([0, share, 0xC000, 0xC000 + second, 65535], np.uint16)
    first = rng.integers(0, 4, 256).astype(np.int8)
    first[0], first[1:zeros + 1] = 2, 0
    other = rng.integers(0, 4, 256).astype(np.int8)
    want = pair(oracle, host_model, [cdf, cdf], [first, other])
    assert (want[0] == first).all() and (want[1] == other).all()


@pytest.mark.parametrize("lp", [2, 3, 5, 9, 17, 33])
@pytest.mark.parametrize("seed", [0, 1])
def test_equal_shares_come_back_to_the_full_range(oracle, host_model, lp, seed):
    rng = np.random.default_rng(lp + seed)
    n = int(rng.integers(1, 200))
    even = (np.arange(lp, dtype=np.int64) * (65536 // (lp - 1))).clip(max=65535).astype(np.uint16)
    skew = np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), lp - 1, replace=False)))).astype(np.uint16)
    syms = [rng.integers(0, lp - 1, n).astype(np.int8) for _ in range(2)]
    for cdfs in ([even, even], [even, skew], [skew, even]):
        want = pair(oracle, host_model, cdfs, syms)
        assert (want[0] == syms[0]).all() and (want[1] == syms[1]).all()


@pytest.mark.parametrize("cut", [(0, 0), (1, None), (4, 7), (8, 9), (11, 12), (13, 0)])
def test_streams_that_end_inside_the_window(oracle, host_model, cut):
    rng = np.random.default_rng(sum(k or 0 for k in cut))
    w = np.sort(rng.choice(np.arange(1, 65535), 32, replace=False))
    cdf = np.concatenate(([0], w)).astype(np.uint16)
    syms = [rng.integers(0, 31, 120).astype(np.int8) for _ in range(2)]
    pair(oracle, host_model, [cdf, cdf], syms, cut)
