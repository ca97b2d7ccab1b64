"""Decode of symbols where the upper half of a table holds next to nothing: blocks that search the lower half only, among them
streams with symbols of the upper half, next to blocks that search all of it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lp", [9, 10, 17, 18, 33, 34, 64])
@pytest.mark.parametrize("C,T", [(128, 256), (300, 37), (640, 5)])
def test_tables_with_an_empty_upper_half(oracle, lp, C, T):
    from cachegen_b200.serde import CacheGenGPUBytestream, cachegen_decoder
    rng = np.random.default_rng(lp * C + T)
    n, half = lp - 1, 1
    while 2 * half < n:
        half *= 2
    cdf, sym = np.zeros((2, C, lp), np.uint16), np.zeros((2, T, C), np.int8)
    for r in range(2):
        for c in range(C):
            deep = c // 128 % 3 == 2 and rng.random() < 0.02  # one channel is enough for its block
            used = n if deep else half - rng.integers(0, 2)
            w = np.ones(n, dtype=np.int64)
            w[:used] += rng.multinomial(65535 - n, rng.dirichlet(np.full(used, 0.7)))
            cdf[r, c, :n] = np.concatenate(([0], np.cumsum(w)[:-1]))
            cdf[r, c, n] = 65535
            sym[r, :, c] = rng.choice(n, size=T, p=w / w.sum())
            if c % 5 == 0:
                sym[r, rng.integers(0, T), c] = rng.integers(half - 1, n)
    data, lengths = oracle.encode_chunk(cdf.view(np.int16), sym)
    out = torch.zeros((2, T, C), dtype=torch.uint8, device="cuda")
    streams = CacheGenGPUBytestream(torch.from_numpy(data.copy()).cuda(), torch.from_numpy(lengths.astype(np.int32)).cuda(), T)
    cachegen_decoder.decode_chunk(torch.from_numpy(cdf.view(np.int16)).cuda(), streams, out)
    assert (out.cpu().numpy() == sym.view(np.uint8)).all()
