"""calculate_cdf around the sizes of its batches of loads (eight warps of 32, of 8 and of single tokens), at groups of channels that are
not full, on adjacent bytes and on strides, with symbols outside the table and up to the most tokens."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 7, 8, 63, 64, 65, 200, 255, 256, 257, 321, 512])
@pytest.mark.parametrize("channels, max_bins", [(4, 32), (128, 16), (132, 62), (300, 32), (130, 31), (31, 5)])
def test_tables_of_symbols(oracle, tokens, channels, max_bins):
    from cachegen_b200 import torchac_cuda
    sym = np.random.default_rng(tokens * channels).integers(0, max_bins, (3, tokens, channels)).astype(np.int8)
    sym[1] = np.minimum(sym[1], 2)
    want = oracle.calculate_cdf(sym, max_bins)
    dev = torch.from_numpy(sym).cuda()
    for x in (dev, torch.stack((dev, dev), 3)[..., 0]):
        assert (torchac_cuda.calculate_cdf(x, max_bins).cpu().numpy() == want).all()


def tables(sym, max_bins):
    """The reference's, from counts that leave out what is outside the table (a channel with nothing inside counts as empty)."""
    counts = np.stack([(sym.view(np.uint8) == v).sum(1) for v in range(max_bins)], -1).astype(np.uint64)
    below = np.concatenate((np.zeros_like(counts[..., :1]), np.cumsum(counts, -1, dtype=np.uint64)), -1)
    total = np.maximum(below[..., -1:], 1)
    return ((np.uint64(0xFFFF - max_bins) * below // total + np.arange(max_bins + 1, dtype=np.uint64)) & np.uint64(0xFFFF)).astype(np.uint16).view(np.int16)


@pytest.mark.parametrize("tokens, channels, max_bins", [(1, 128, 32), (3, 132, 9), (255, 128, 32), (256, 132, 32), (300, 300, 62), (519, 31, 5), (65535, 132, 32)])
@pytest.mark.parametrize("share", [0.02, 0.5, 1.0])
def test_symbols_outside_the_table_are_not_counted(oracle, tokens, channels, max_bins, share):
    """From max_bins to 127 and below zero, in the batches and behind them: a few in every channel, most, and in some channels all."""
    from cachegen_b200 import torchac_cuda
    rng = np.random.default_rng(tokens + channels)
    rows = 2 if tokens < 1000 else 1
    sym = rng.integers(0, max_bins, (rows, tokens, channels)).astype(np.int8)
    outside = np.concatenate((np.arange(max_bins, 128), np.arange(-128, 0))).astype(np.int8)
    sym = np.where(rng.random(sym.shape) < share, rng.choice(outside, sym.shape), sym)
    sym[:, :, ::3] = np.minimum(sym[:, :, ::3] % max_bins, max_bins - 1)  # channels with none
    sym[:, -1, 1] = -1
    sym[:, 0, 2], sym[:, -1, 2] = max_bins, 127
    want = tables(sym, max_bins)
    inside = ((sym >= 0) & (sym < max_bins)).any(1)  # the others have no table in the oracle either
    for r in range(rows):
        few = np.flatnonzero(inside[r])[:8]
        assert (oracle.calculate_cdf(np.ascontiguousarray(sym[r:r + 1, :, few]), max_bins) == want[r:r + 1, few]).all()
    dev = torch.from_numpy(sym).cuda()
    for x in (dev, torch.stack((dev, dev), 3)[..., 0]):
        assert (torchac_cuda.calculate_cdf(x, max_bins).cpu().numpy() == want).all()
