"""Tables of chunks of several sub-chunks: groups of channels that are not full, tokens around the kernel's batches (eight warps of four
words of four tokens) and words that are not, against the oracle; int16 tables and byte counts."""
import numpy as np
import pytest
import torch

from gpu_util import bits_np, kv_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,D", [(1, 8), (3, 24), (1, 136), (5, 80)])
@pytest.mark.parametrize("T", [257, 260, 511, 512, 513, 515, 543, 1027])
def test_tables_of_several_sub_chunks(oracle, H, D, T):
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.serde.cachegen_basics import CacheGenConfig
    cfg = CacheGenConfig(1, 1, 2, 32, 12, 12, 1, 32, 16)
    config, meta = LMCacheEngineConfig.from_defaults(chunk_size=2048), LMCacheEngineMetadata("m", 1, 0, "vllm")
    ser, de = CacheGenSerializer(config, meta, cfg), CacheGenDeserializer(config, meta, cfg, out_dtype=torch.float16)
    torch.manual_seed(T + H * D)
    kv = (torch.randn(2, 2, T, H, D) * torch.exp(torch.randn(2, 2, 1, H, D))).half()
    sym, _ = oracle.quantize(bits_np(kv_rows(kv)), np.array([32, 12, 32, 16], np.float32), oracle.F16)
    eo = ser.encode(kv.cuda())
    assert (eo.cdf.cpu().numpy() == oracle.calculate_cdf(sym, 32)).all()
    want = bits_np(de.decode(eo))
    for compact in (True, "counts", False):  # (counts above 255 go back to whole tables)
        assert (bits_np(de.decode(ser.encode_flat(kv.cuda(), compact_tables=compact))) == want).all()
