"""Tables made from sparse byte counts at every number of counts and at every byte that they may start at, up to all 32 symbols of a row:
a container decodes to what the same chunk's int16 tables decode to, on both decoders (two channels a thread and one)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 2, 3, 37, 64, 200, 255, 256])
@pytest.mark.parametrize("bins, max_bins", [(34, 34), (33, 62), (32, 32), (16, 32), (4, 32), (5, 5)])
@pytest.mark.parametrize("heads, head", [(2, 64), (3, 43)])
def test_columns_from_sparse_counts(tokens, bins, max_bins, heads, head):
    from cachegen_b200.serde import cachegen_decoder as M
    from cachegen_b200.serde import cachegen_encoder as E
    from cachegen_b200.serde import flat_format as ff
    g = torch.Generator().manual_seed(tokens * bins)
    # from a few symbols a channel to all of them
    kv = ((torch.rand((2, 2, tokens, heads, head), generator=g) * 2 - 1) * torch.rand((2, 2, 1, heads, head), generator=g) ** 2).half().cuda()
    b = torch.full((2,), float(bins)).cuda()
    eo = E.encode_function(kv, None, b, b, tokens, max_bins=max_bins)
    chunk = E.encode_flat(kv, b, b, True, max_bins=max_bins)
    assert chunk.header.table_kind in (ff.TABLES_SPARSE, ff.TABLES_CDF)  # (a symbol may come up 256 times)
    both = torch.cat((b, b))
    want = M.decode_many([eo], both, "vllm", torch.float16, workspace={})
    host_bins = M._HostBins(both)
    for k in (1, 30):  # the quick form and the other
        got = M.decode_many([chunk] * k, both, "vllm", torch.float16, workspace={}, host_bins=host_bins)
        assert torch.equal(got.view(torch.int16), want.repeat(1, 1, k, 1, 1).view(torch.int16))
