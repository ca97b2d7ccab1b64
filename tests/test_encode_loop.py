"""The encoder's loop (two streams a lane, one vote for one or two symbols, rare cases left to a second pass) against the
oracle: runs of ones through whole words, ranges that are powers of two, tables whose symbols take the most bits."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_coder_carry import straddling

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def loop(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("encode_loop") / "libencode_loop.so")
    src = os.path.join(HERE, "host_model", "encode_loop_host.cpp")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so, src])
    lib = ctypes.CDLL(so)
    lib.el_encode.restype = ctypes.c_int64
    lib.el_encode.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p,
                              ctypes.c_int64, ctypes.c_int] + [ctypes.c_void_p] * 2

    def encode(cdf, sym, counted=0):
        sym = np.ascontiguousarray(sym, dtype=np.uint8)
        cap = 2 * len(sym) + 8
        out, again, most = np.zeros(cap, dtype=np.uint8), ctypes.c_int(0), ctypes.c_int(0)
        n = lib.el_encode(cdf.ctypes.data, len(cdf), sym.ctypes.data, len(sym), out.ctypes.data, cap, counted,
                          ctypes.byref(again), ctypes.byref(most))
        assert 0 <= n <= cap and most.value < 64
        return out[:n], again.value

    encode.lib = lib
    return encode


def same(loop, oracle, cdf, sym, counted=0):
    got, again = loop(cdf, sym, counted)
    want = oracle.encode_stream(cdf, np.asarray(sym, dtype=np.int8))
    assert len(got) == len(want) and (got == want).all()
    return again


def test_carries_through_whole_words(loop, oracle):
    rng = np.random.default_rng(0)
    again = 0
    for run in (1, 11, 22, 33, 40, 64, 90, 200):
        for _ in range(10):
            for lp in (4, 9, 33):
                cdf = np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), size=lp - 2, replace=False)),
                                      [65535])).astype(np.uint16)
                head = straddling(cdf, [int(v) for v in rng.integers(0, lp - 1, size=int(rng.integers(0, 4)))], run)
                for tail in ([0], [lp - 2], [0] * 5, [lp - 2] * 5, []):
                    again += same(loop, oracle, cdf, (head + tail)[:256])
    assert again  # the second pass was taken


@pytest.mark.parametrize("step", [1 << 10, 1 << 12, 1 << 13, 1 << 14, 1 << 15])
def test_ranges_that_are_powers_of_two(loop, oracle, step):
    rng = np.random.default_rng(step)
    edges = np.arange(0, 65536, step)
    for k in range(300):
        inner = edges[1:] if len(edges) < 4 else np.sort(rng.choice(edges[1:], size=int(rng.integers(1, min(62, len(edges)))), replace=False))
        cdf = np.concatenate(([0], inner, [65535])).astype(np.uint16)
        n = int(rng.integers(1, 257))
        sym = rng.integers(0, len(cdf) - 1, size=n) if k % 2 else np.full(n, rng.integers(0, len(cdf) - 1))
        same(loop, oracle, cdf, sym)


@pytest.mark.parametrize("tokens", [1, 2, 3, 60, 61, 255, 256, 257, 1999, 2047, 2048, 8191, 21823, 21824])
def test_two_symbols_a_vote_with_counted_tables(loop, oracle, tokens):
    rng = np.random.default_rng(tokens)
    for kind in range(4):
        sym = rng.integers(0, 61, size=tokens) if kind == 0 else np.where(rng.random(tokens) < 0.97, 30, rng.integers(0, 61, size=tokens))
        if kind == 2:  # symbols that occur once, one after the other: the most bits a symbol can take
            sym[:] = 30
            k = min(tokens, 61)
            sym[:k] = rng.permutation(61)[:k]
        if kind == 3:
            sym[:] = rng.integers(0, 61)
        cdf = oracle.calculate_cdf(sym.astype(np.int8).reshape(1, -1, 1), 62)[0, 0].view(np.uint16).copy()
        for s in range(0, tokens, 256)[:4]:
            same(loop, oracle, cdf, sym[s:s + 256], counted=tokens)


def test_high_water_leaves_room_for_two_symbols(loop):
    for tokens in (1, 256, 257, 2048, 8192, 16384, 21824):
        w = (0xFFFF - 63) // tokens + 1
        most = 18 - (w.bit_length() - 1)
        high = loop.lib.el_pair_high_water(tokens)
        assert high and max(high - 1, 31) + 2 * most <= 63
    assert loop.lib.el_pair_high_water(32737) == 0 and loop.lib.el_pair_high_water(65535) == 0
