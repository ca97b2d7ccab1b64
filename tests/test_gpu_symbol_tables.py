"""calculate_cdf around the sizes of its batches of loads (eight warps of 32, of 8 and of single tokens), at groups of channels that are
not full, on adjacent bytes and on strides, with symbols outside the table and histograms that wrap at 65,536."""
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
