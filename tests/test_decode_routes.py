"""Which decodes try the native call."""
import types

import torch


def test_chunks_in_host_memory_go_straight_to_the_general_path(monkeypatch):
    """Nothing is prepared for a call that cannot take them."""
    from cachegen_b200 import _lib
    from cachegen_b200.serde import cachegen_decoder as M
    from cachegen_b200.serde import flat_format as ff
    from cachegen_b200.serde.cachegen_basics import CacheGenGPUEncoderOutput

    def refuse():
        raise AssertionError("the native call was tried")

    monkeypatch.setattr(_lib, "calls", refuse)
    L, H, D, T = 2, 1, 8, 3
    header = ff.layout(L, H, D, T, 33, torch.float16, ff.TABLES_CDF, 2 * 2 * L * H * D * 33, ff.LENGTHS_U16, [0, 16])
    flat = ff.FlatChunk(torch.zeros(header.total, dtype=torch.uint8), header)
    pickled = CacheGenGPUEncoderOutput([], torch.zeros((2 * L, H * D, 33), dtype=torch.int16), torch.zeros((L, T, 1)), torch.zeros((L, T, 1)), H, D)
    bins = types.SimpleNamespace(is_cuda=True, device=torch.device("cpu"))
    host_bins = M._HostBins(torch.full((2 * L,), 32.0))
    for chunk in (flat, pickled):
        workspace = {}
        assert M._decode_usual([chunk], bins, "vllm", torch.float16, None, workspace, host_bins) is None
        assert not workspace
