"""The encode kernels at sequences that their loop leaves to a second pass, and at the symbols that take the most bits,
against the oracle: separate calls with given tables, and whole encodes of KV whose symbols are given (one channel
holds the scale)."""
import numpy as np
import pytest
import torch

from test_coder_carry import straddling

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run", [22, 64, 200])
def test_carries_through_whole_words(oracle, run):
    from cachegen_b200.serde import cachegen_encoder as E
    rng = np.random.default_rng(run)
    lp, C = 33, 200
    cdf, sym = np.zeros((2, C, lp), np.uint16), np.zeros((2, 256, C), np.int8)
    for r in range(2):
        for c in range(C):
            cdf[r, c] = np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), size=lp - 2, replace=False)), [65535]))
            head = straddling(cdf[r, c], [int(v) for v in rng.integers(0, lp - 1, size=c % 4)], run)
            tail = [int(v) for v in rng.integers(0, lp - 1, size=256)]
            sym[r, :, c] = (head + tail)[:256]
    payload, lengths, _ = E.encode_streams(torch.from_numpy(cdf.view(np.int16)).cuda(), torch.from_numpy(sym).cuda())
    want, want_len = oracle.encode_chunk(cdf.view(np.int16), sym)
    assert (lengths[0].cpu().numpy() == want_len).all()
    assert payload.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize("tokens", [1, 2, 61, 256, 257, 2048, 21824, 32737])
def test_symbols_that_take_the_most_bits(oracle, tokens):
    from cachegen_b200.serde import cachegen_encoder as E
    rng = np.random.default_rng(tokens)
    C, mid = 136, 30
    sym = np.full((2, tokens, C), mid, np.int8)
    for r in range(2):
        for c in range(1, C):
            k = min(tokens, int(rng.integers(0, 62)))
            at = int(rng.integers(0, tokens - k + 1))
            sym[r, at:at + k, c] = rng.permutation(61)[:k]
    sym[:, :, 0] = 60
    kv = torch.from_numpy((sym - mid).astype(np.float16)).reshape(1, 2, tokens, 17, 8).cuda()
    bins = torch.full((1,), 62.0).cuda()
    out = E.encode_function(kv, None, bins, bins, tokens)
    cdf = oracle.calculate_cdf(sym, 62)
    assert (out.cdf.cpu().numpy() == cdf).all()
    for j, piece in enumerate(out.data_chunks):
        want, want_len = oracle.encode_chunk(cdf, sym[:, 256 * j:256 * (j + 1)])
        assert (piece.bytestream_lengths.cpu().numpy() == want_len).all()
        assert piece.bytestream.cpu().numpy().tobytes() == want.tobytes()
