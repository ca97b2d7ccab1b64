"""encode_levels (up to four bin settings in one launch for each step) against an encode of its own for each setting: one
launch's worth of settings and more, one and several sub-chunks, shapes of the fused passes and of the separate calls."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 5, 256, 257, 600])
@pytest.mark.parametrize("H,D,dtype", [(1, 8, torch.float16), (3, 80, torch.bfloat16), (17, 8, torch.float16), (3, 7, torch.bfloat16)])
@pytest.mark.parametrize("settings", [[32], [62, 4, 17], [16, 32, 32, 8], [8, 62, 32, 16, 5, 32, 9]])
def test_settings_together_equal_settings_alone(T, H, D, dtype, settings):
    from cachegen_b200.serde import cachegen_encoder as E
    L = 2
    kv = torch.randn((L, 2, T, H, D), generator=torch.Generator().manual_seed(T + H)).to(dtype).cuda()
    kv[:, :, T // 2] = 0
    bins = [(torch.tensor([float(b), max(4.0, b // 2)]).cuda(), torch.tensor([max(4.0, b // 3), float(b)]).cuda()) for b in settings]
    together = E.encode_levels(kv, bins)
    assert len(together) == len(bins)
    for out, (kb, vb) in zip(together, bins):
        want = E.encode_function(kv, None, kb, vb, T)
        assert torch.equal(out.cdf, want.cdf)
        assert torch.equal(out.max_tensors_key, want.max_tensors_key) and torch.equal(out.max_tensors_value, want.max_tensors_value)
        assert len(out.data_chunks) == len(want.data_chunks)
        for a, b in zip(out.data_chunks, want.data_chunks):
            assert a.ntokens == b.ntokens and torch.equal(a.bytestream, b.bytestream)
            assert torch.equal(a.bytestream_lengths, b.bytestream_lengths)


def test_no_settings():
    from cachegen_b200.serde import cachegen_encoder as E
    assert E.encode_levels(torch.zeros((1, 2, 4, 1, 8), dtype=torch.float16, device="cuda"), []) == []
