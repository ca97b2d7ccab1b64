"""The coder of one sub-chunk starts while its quantiser still runs: a workspace that is used again at once, for other symbols,
gives every chunk its own tables, sizes and streams."""
import numpy as np
import pytest
import torch

from gpu_util import bits_np, kv_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,H,T", [(1, 1, 3), (10, 8, 61), (32, 2, 255), (20, 30, 256)])
def test_workspace_used_again_at_once(oracle, L, H, T):
    from cachegen_b200.serde import cachegen_encoder as E
    bins = torch.tensor([32.0] * (L - L // 2) + [16.0] * (L // 2))
    info = E._BinsInfo(bins, bins)
    g = torch.Generator(device="cuda").manual_seed(L)
    # caches whose symbols differ from one to the next: near the ends of the range, then near its middle
    kvs = [torch.randn((L, 2, T, H, 128), generator=g, device="cuda").sign() * torch.rand((L, 2, T, H, 128), generator=g, device="cuda") ** p
           for p in (0.1, 8.0, 0.3, 3.0)]
    kvs = [kv.half() for kv in kvs]
    torch.cuda.synchronize()
    workspace, pending = None, []
    for kv in kvs:
        pending.append(E._PendingChunk(kv, info, 32, workspace=workspace))
        workspace = pending[0].workspace
    try:
        last = pending[-1].finish()
        ends = [p.tail[:2].tolist()[1] if p.tail is not None else last.data_chunks[0].bytestream.numel() for p in pending]
    finally:
        for p in pending:
            p.abandon()
    both = torch.cat((bins, bins)).numpy()
    for kv, p, end in zip(kvs, pending, ends):
        sym, mx = oracle.quantize(bits_np(kv_rows(kv)), both)
        cdf = oracle.calculate_cdf(sym, 32)
        assert (p.cdf.cpu().numpy() == cdf).all()
        assert (np.concatenate((bits_np(p.scales_k), bits_np(p.scales_v))).reshape(2 * L, T) == mx.reshape(2 * L, T)).all()
        want, want_len = oracle.encode_chunk(cdf, sym)
        assert end == want.size
    assert (last.data_chunks[0].bytestream_lengths.cpu().numpy() == want_len).all()
    assert last.data_chunks[0].bytestream.cpu().numpy().tobytes() == want.tobytes()
