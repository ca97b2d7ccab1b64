"""The encoder's step in the form and at the marks that the kernels run, two streams a lane that store together, against the oracle."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_coder_carry import straddling

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def loop(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("encode_kernel_loop") / "libencode_kernel_loop.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so, os.path.join(HERE, "host_model", "encode_kernel_loop_host.cpp")])
    lib = ctypes.CDLL(so)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)

    def encode(oracle, cdf, sym, counted=0):
        """cdf [2, lp], sym [n, 2]; returns (the most bits pending behind a step, streams coded again)."""
        cdf, sym = np.ascontiguousarray(cdf, np.uint16), np.ascontiguousarray(sym, np.uint8)
        cap = 2 * len(sym) + 8
        out, length, again, deepest = np.zeros((2, cap), np.uint8), np.zeros(2, np.int32), np.zeros(2, np.uint8), ctypes.c_int()
        assert lib.ek_encode(p(cdf), cdf.shape[1], p(sym), len(sym), p(out), ctypes.c_int64(cap), counted, p(length), p(again), ctypes.byref(deepest)) == 0
        for i in range(2):
            want = oracle.encode_stream(cdf[i], sym[:, i].astype(np.int8))
            assert length[i] == len(want) and (out[i, :len(want)] == want).all(), i
        return deepest.value, int(again.sum())

    encode.lib = lib
    return encode


@pytest.mark.parametrize("tokens", [1, 2, 3, 61, 255, 256, 257, 1999, 21824])
def test_pairs_of_symbols_of_counted_tables(loop, oracle, tokens):
    rng = np.random.default_rng(tokens)
    deepest = 0
    for kind in range(4):
        sym = rng.integers(0, 61, (tokens, 2))
        if kind == 1:
            sym[rng.random(tokens) < 0.97, 1] = 30
        elif kind == 2:  # symbols that occur once, one after the other, beside a stream that stays short
            sym[:] = 30
            k = min(tokens, 61)
            sym[:k, 0] = rng.permutation(61)[:k]
        elif kind == 3:
            sym[:] = rng.integers(0, 61, 2)
        cdf = oracle.calculate_cdf(sym.astype(np.int8)[None], 62)[0].view(np.uint16)
        for s in range(0, tokens, 256)[:4]:
            deepest = max(deepest, loop(oracle, cdf, sym[s:s + 256], tokens)[0])
    assert tokens < 61 or deepest >= 64  # pending bits did leave the accumulator


@pytest.mark.parametrize("lp", [3, 9, 33, 64])
def test_carries_and_last_symbols_of_any_tables(loop, oracle, lp):
    rng = np.random.default_rng(lp)
    again = 0
    for run in (1, 22, 40, 64, 200):
        for tail in ([0], [lp - 2] * 5, []):
            cdf = np.stack([np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), lp - 2, replace=False)), [65535])) for _ in range(2)]).astype(np.uint16)
            first = (straddling(cdf[0], [int(rng.integers(0, lp - 1))], run) + tail)[:256]
            sym = np.stack((first, rng.integers(0, lp - 1, len(first))), 1)
            again += loop(oracle, cdf, sym)[1]
    assert again or lp == 3


def test_marks_leave_room_in_front_of_the_second_symbol(loop):
    for tokens in (1, 256, 257, 2048, 8192, 16384, 21824):
        most = 18 - (((0xFFFF - 63) // tokens + 1).bit_length() - 1)
        mark = loop.lib.ek_deep_pair_high_water(tokens)
        # at most 63 bits, in a stream below the mark and in one that has just stored a word
        assert mark and mark - 1 + most <= 63 and mark - 1 + 2 * most - 32 + most <= 63
    assert loop.lib.ek_deep_pair_high_water(32737) == 0
