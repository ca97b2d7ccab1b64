"""Decode kernels at the edges of their rules: groups of channels that are not full (lanes that repeat the last channels), tables of
every length that is staged by words, half-words and columns, tokens too far apart for 32-bit steps."""
import numpy as np
import pytest
import torch

from gpu_util import bits_np, kv_rows

pytestmark = pytest.mark.gpu


def coded(oracle, rng, lp, C, T, rows=2):
    n = lp - 1
    cdf, sym = np.zeros((rows, C, lp), np.uint16), np.zeros((rows, T, C), np.int8)
    for r in range(rows):
        for c in range(C):
            w = 1 + rng.multinomial(65535 - n, rng.dirichlet(np.full(n, 0.5)))
            cdf[r, c] = np.concatenate(([0], np.cumsum(w)))
            sym[r, :, c] = rng.choice(n, size=T, p=w / w.sum())
    return cdf, sym


@pytest.mark.parametrize("lp", [2, 3, 9, 16, 17, 18, 32, 33, 34])
@pytest.mark.parametrize("C,T", [(128, 65), (136, 30), (202, 30), (130, 1)])
def test_symbols(oracle, lp, C, T):
    from cachegen_b200.serde import CacheGenGPUBytestream, cachegen_decoder
    cdf, sym = coded(oracle, np.random.default_rng(lp * C + T), lp, C, T)
    data, lengths = oracle.encode_chunk(cdf.view(np.int16), sym)
    out = torch.zeros((2, T, C), dtype=torch.uint8, device="cuda")
    streams = CacheGenGPUBytestream(torch.from_numpy(data.copy()).cuda(), torch.from_numpy(lengths.astype(np.int32)).cuda(), T)
    cachegen_decoder.decode_chunk(torch.from_numpy(cdf.view(np.int16)).cuda(), streams, out)
    assert (out.cpu().numpy() == sym.view(np.uint8)).all()


@pytest.mark.parametrize("share,second,zeros", [(35107, 10873, 16), (33903, 15341, 63), (34067, 13388, 130)])
def test_a_range_of_half_of_all_values_at_a_multiple_of_it(oracle, share, second, zeros):
    # see tests/test_decode_window.py
    from cachegen_b200 import torchac_cuda
    rng = np.random.default_rng(share)
    cdf = np.tile(np.array([0, share, 0xC000, 0xC000 + second, 65535], np.uint16), (1, 64, 1))
    sym = rng.integers(0, 4, (1, 256, 64)).astype(np.int8)
    sym[0, 0, ::3], sym[0, 1:zeros + 1, ::3] = 2, 0
    streams = [oracle.encode_stream(cdf[0, c], sym[0, :, c]) for c in range(64)]
    ends = np.cumsum([len(s) for s in streams]).astype(np.int64).reshape(1, 64)
    out = torch.zeros((1, 256, 64), dtype=torch.uint8, device="cuda")
    torchac_cuda.decode_fast_prefsum(torch.from_numpy(cdf.view(np.int16)).cuda(), torch.from_numpy(np.concatenate(streams)).cuda(),
                                     torch.from_numpy(ends).cuda(), out)
    assert (out.cpu().numpy() == sym.view(np.uint8)).all()


@pytest.mark.parametrize("bins,H,D", [(12, 3, 40), (16, 5, 24), (24, 1, 8), (32, 2, 136)])
@pytest.mark.parametrize("T", [1, 37, 257])
def test_values_of_groups_that_are_not_full(bins, H, D, T):
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.serde.cachegen_basics import CacheGenConfig
    cfg = CacheGenConfig(1, 1, 2, bins, bins, bins, 1, bins, bins)
    config, meta = LMCacheEngineConfig.from_defaults(chunk_size=512), LMCacheEngineMetadata("m", 1, 0, "vllm")
    ser, de = CacheGenSerializer(config, meta, cfg), CacheGenDeserializer(config, meta, cfg, out_dtype=torch.float16)
    torch.manual_seed(bins * T)
    kv = (torch.randn(2, 2, T, H, D) * torch.exp(torch.randn(2, 2, 1, H, D))).half().cuda()
    eo = ser.encode(kv)
    want = de.decode(eo)
    # the general kernel, one channel a thread, takes an output whose rows are an odd number of values apart
    odd = torch.zeros((2, 2, T, H, D + 1), dtype=torch.float16, device="cuda")[..., :D]
    assert (bits_np(de.decode(eo, out=odd)) == bits_np(want)).all()
    for compact in (True, "counts", False):
        assert (bits_np(de.decode(ser.encode_flat(kv, compact_tables=compact))) == bits_np(want)).all()


@pytest.mark.parametrize("step", [8388608 - 128, 8388608, 8388608 + 128])
def test_tokens_too_far_apart_for_32_bit_steps(step):
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.serde.cachegen_basics import CacheGenConfig
    cfg = CacheGenConfig(1, 1, 1, 16, 16, 16, 1, 16, 16)
    config, meta = LMCacheEngineConfig.from_defaults(chunk_size=512), LMCacheEngineMetadata("m", 1, 0, "vllm")
    ser, de = CacheGenSerializer(config, meta, cfg), CacheGenDeserializer(config, meta, cfg, out_dtype=torch.float16)
    torch.manual_seed(step % 1000)
    kv = torch.randn(1, 2, 256, 2, 64).half().cuda()
    eo = ser.encode(kv)
    room = torch.empty(256 * step, dtype=torch.float16, device="cuda")
    far = room.as_strided((1, 2, 256, 2, 64), (256, 128, step, 64, 1))
    assert (bits_np(de.decode(eo, out=far)) == bits_np(de.decode(eo))).all()
