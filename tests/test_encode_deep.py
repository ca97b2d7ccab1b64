"""The encoder's loop with the accumulator's upper word kept from before the last shift, as the kernels run it: streams of one
warp, which store words together, against the oracle.  Nothing may be lost when a last shift moves pending bits out of the accumulator."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_coder_carry import straddling

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def encode(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("encode_deep") / "libencode_deep.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so, os.path.join(HERE, "host_model", "encode_deep_host.cpp")])
    lib = ctypes.CDLL(so)

    def run(oracle, cdf, sym, counted):
        """cdf [lanes, lp], sym [n, lanes]; returns (most bits pending in front of a last shift, behind it, streams coded again)."""
        n, lanes = sym.shape
        cdf, sym = np.ascontiguousarray(cdf, np.uint16), np.ascontiguousarray(sym, np.uint8)
        cap = 2 * n + 8
        out, length, again = np.zeros((lanes, cap), np.uint8), np.zeros(lanes, np.int32), np.zeros(lanes, np.uint8)
        most, deepest = ctypes.c_int(), ctypes.c_int()
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
        assert lib.ed_encode(p(cdf), cdf.shape[1], p(sym), n, lanes, p(out), ctypes.c_int64(cap), counted, p(length), p(again),
                             ctypes.byref(most), ctypes.byref(deepest)) == 0
        for i in range(lanes):
            want = oracle.encode_stream(cdf[i], sym[:, i].astype(np.int8))
            assert length[i] == len(want) and (out[i, :len(want)] == want).all(), i
        assert most.value <= 63  # what a store can put together
        return most.value, deepest.value, int(again.sum())

    return run


@pytest.mark.parametrize("tokens", [1, 2, 3, 61, 255, 256, 257, 1999, 8191, 21824])
def test_counted_tables_two_symbols_a_vote(encode, oracle, tokens):
    rng = np.random.default_rng(tokens)
    deepest = 0
    for kind in range(4):
        lanes = 24
        sym = np.where(rng.random((tokens, lanes)) < 0.9 ** np.arange(lanes), 30, rng.integers(0, 61, (tokens, lanes)))
        if kind == 1:  # symbols that occur once, next to each other: the most bits a symbol can take
            sym[:, ::2] = 30
            k = min(tokens, 61)
            for i in range(0, lanes, 2):
                sym[:k, i] = rng.permutation(61)[:k]
        elif kind == 2:
            sym = rng.integers(0, 61, (tokens, lanes))
        elif kind == 3:
            sym[:, :] = 30
            sym[rng.integers(0, tokens, 3), :] = rng.integers(0, 61, (3, lanes))
        cdf = oracle.calculate_cdf(sym.astype(np.int8)[None], 62)[0].view(np.uint16)
        for s in range(0, tokens, 256)[:3]:
            deepest = max(deepest, encode(oracle, cdf, sym[s:s + 256], tokens)[1])
    assert tokens < 61 or deepest >= 64  # pending bits did leave the accumulator


@pytest.mark.parametrize("lp", [3, 9, 33, 64])
@pytest.mark.parametrize("seed", range(4))
def test_any_tables_one_symbol_a_vote(encode, oracle, lp, seed):
    rng = np.random.default_rng(lp * 10 + seed)
    lanes, n = 16, int(rng.integers(60, 257))
    cdf = np.stack([np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), lp - 2, replace=False)), [65535])) for _ in range(lanes)])
    if seed == 1:  # shares of one: 16 bits a symbol
        cdf[:, 1:-1] = np.arange(1, lp - 1)
    sym = rng.integers(0, lp - 1, (n, lanes))
    if seed == 2:
        sym = np.stack([(straddling(cdf[i], [0], n - 1))[:n] for i in range(lanes)], axis=1)
        sym[-1] = rng.integers(0, lp - 1, lanes)
    deepest = encode(oracle, cdf, sym, 0)[1]
    assert seed != 1 or lp < 9 or deepest >= 64


def test_carries_through_whole_words_next_to_other_streams(encode, oracle):
    rng = np.random.default_rng(5)
    again = 0
    for run in (22, 40, 64, 90, 200):
        for lp in (4, 9, 33):
            lanes, n = 12, run + 6
            cdf = np.stack([np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), lp - 2, replace=False)), [65535])) for _ in range(lanes)])
            sym = rng.integers(0, lp - 1, (n, lanes))
            for i in range(0, lanes, 2):
                sym[:run + 1, i] = straddling(cdf[i], [int(rng.integers(0, lp - 1))], run)
            again += encode(oracle, cdf, sym, 0)[2]
    assert again  # the second pass was taken
