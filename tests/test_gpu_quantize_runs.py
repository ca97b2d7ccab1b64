"""The quantiser of the fused encode at the channel counts where a thread goes from one run of channels to two, where the second
runs end, and at the largest block: scales and tables equal those of the separate calls, alone and for several settings."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads, head", [(1, 8), (127, 8), (1, 1016), (128, 8), (8, 128), (129, 8), (193, 8), (12, 128), (255, 8), (16, 128), (32, 128),
                                         (513, 8), (40, 128), (1023, 8), (64, 128)])
@pytest.mark.parametrize("tokens, dtype", [(3, torch.float16), (260, torch.bfloat16)])
def test_scales_and_tables(heads, head, tokens, dtype):
    from cachegen_b200.serde import cachegen_encoder as E
    kv = torch.randn((2, 2, tokens, heads, head), generator=torch.Generator().manual_seed(heads)).to(dtype).cuda()
    kv[:, :, 1] = 0
    kv[0, 0, 2, heads - 1, head - 1] = 50.0  # the last channel alone decides the scale
    b, c = torch.tensor([32.0, 16.0]).cuda(), torch.tensor([8.0, 32.0]).cuda()
    _, scales, cdf = E.quantize_and_tables(kv, b, c, 32)
    for out in [E.encode_function(kv, None, b, c, tokens)] + E.encode_levels(kv, [(b, c), (b, c)]):
        assert torch.equal(torch.cat((out.max_tensors_key, out.max_tensors_value))[..., 0].view(torch.int16), scales.view(torch.int16))
        assert torch.equal(out.cdf, cdf)
