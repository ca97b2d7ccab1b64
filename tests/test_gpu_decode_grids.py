"""One chunk's decode at every size of grid that gets a form of its own: a few blocks an SM (the quick form), one wave, a second wave
of one to four blocks an SM, and more; and the symbol decoder at the second of those."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def chunk():
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenConfig, CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.synth import generate_kv
    config = CacheGenConfig.from_model_name("Yukang/LongAlpaca-70B-16k").layer_slice(0, 10)
    engine, meta = LMCacheEngineConfig.from_defaults(chunk_size=256), LMCacheEngineMetadata("m", 1, 0, "vllm")
    ser = CacheGenSerializer(engine, meta, config, table_max_bins=32)
    de = CacheGenDeserializer(engine, meta, config, out_dtype=torch.float16)
    kv = generate_kv(10, 4, 128, 90, seed=3, device="cuda", dtype=torch.float16)
    return ser, de, kv, ser.encode(kv)


def test_the_same_values_from_every_size_of_grid(chunk, oracle):
    ser, de, kv, eo = chunk
    import numpy as np
    rows = kv.cpu().transpose(0, 1).reshape(20, 90, 512).contiguous()
    bins = torch.cat((ser.key_bins, ser.value_bins)).cpu().numpy()
    sym, mx = oracle.quantize(rows.view(torch.int16).numpy().view(np.uint16), bins)
    cq = np.floor(bins / 2).astype(np.float32)[:, None, None] - 1
    want = ((sym.astype(np.float32) - cq) / cq) * torch.from_numpy(mx.view(np.int16).copy()).view(torch.float16).float().numpy().reshape(20, 90, 1)
    want = torch.from_numpy(want).half().reshape(2, 10, 90, 4, 128).transpose(0, 1)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for per_sm in (0.3, 4, 5, 12, 13, 14, 15, 16, 17):  # 80 blocks a copy
        n = max(1, int(per_sm * sms / 80))
        got = de.decode_many([eo] * n)
        for i in range(n):
            assert torch.equal(got[:, :, 90 * i:90 * (i + 1)].cpu().view(torch.int16), want.view(torch.int16)), (per_sm, i)
    de.check_status()


@pytest.mark.parametrize("bins", [4, 8, 12, 16, 17, 30, 32, 62])
def test_the_quick_form_at_every_depth(bins):
    """Few and many blocks of the same streams, at two to six levels of the search."""
    from cachegen_b200.serde import cachegen_decoder as M
    from cachegen_b200.serde import cachegen_encoder as E
    kv = torch.randn((2, 2, 200, 3, 64), generator=torch.Generator().manual_seed(bins)).half().cuda()
    b = torch.full((2,), float(bins)).cuda()
    eo = E.encode_function(kv, None, b, b, 200)
    one = M.decode_many([eo], torch.cat((b, b)), "vllm", torch.float16, workspace={})
    many = M.decode_many([eo] * 120, torch.cat((b, b)), "vllm", torch.float16, workspace={})
    assert torch.equal(many.view(torch.int16), one.repeat(1, 1, 120, 1, 1).view(torch.int16))
    x = kv.float()
    assert ((one.float() - x).abs() <= x.abs().amax((3, 4), keepdim=True) * (0.51 / (bins // 2 - 1))).all()


@pytest.mark.parametrize("rows, channels", [(20, 512), (60, 4096), (64, 4096)])
def test_symbols_come_back_at_either_side_of_a_wave(rows, channels):
    from cachegen_b200 import torchac_cuda
    sym = torch.randint(0, 31, (rows, 70, channels), generator=torch.Generator().manual_seed(rows)).to(torch.int8).cuda()
    sym[: rows // 2] %= 9
    from cachegen_b200.serde import cachegen_encoder as E
    cdf = torchac_cuda.calculate_cdf(sym, 32)
    buf = torch.empty((rows, channels, 520), dtype=torch.uint8, device="cuda")
    lengths = torch.empty((rows, channels), dtype=torch.int32, device="cuda")
    streams = E.encode_ntokens(cdf, sym, buf, lengths)
    out = torch.empty((rows, 70, channels), dtype=torch.uint8, device="cuda")
    torchac_cuda.decode_by_lengths(cdf, streams, lengths, out)
    assert torch.equal(out.view(torch.int8), sym)


@pytest.mark.parametrize("heads, bins, tokens, delta", [(31, 32, 64, None), (32, 32, 70, None), (34, 32, 64, None), (37, 32, 65, None),
                                                        (32, 16, 64, None), (32, 8, 64, None), (32, 62, 64, None), (32, 32, 63, None), (34, 32, 64, 16)])
def test_grids_with_blocks_held_back(heads, bins, tokens, delta):
    """One chunk of 14 to 16 blocks an SM, some of them held back, and the same streams twice in a grid that holds none back; long
    tables, fewer tokens and delta coding, where none are."""
    from cachegen_b200.serde import cachegen_decoder as M
    from cachegen_b200.serde import cachegen_encoder as E
    from cachegen_b200.serde.cachegen_basics import DeltaCoding
    kv = torch.randn((32, 2, tokens, heads, 128), generator=torch.Generator("cuda").manual_seed(bins), device="cuda").half()
    b, delta = torch.full((32,), float(bins)).cuda(), delta and DeltaCoding(delta)
    eo = E.encode_function(kv, None, b, b, tokens, delta=delta)
    one = M.decode_many([eo], torch.cat((b, b)), "vllm", torch.float16, workspace={}, delta=delta)
    two = M.decode_many([eo] * 2, torch.cat((b, b)), "vllm", torch.float16, workspace={}, delta=delta)
    assert torch.equal(two.view(torch.int16), one.repeat(1, 1, 2, 1, 1).view(torch.int16))
    if delta is None:
        x = kv.float()
        assert ((one.float() - x).abs() <= x.abs().amax((3, 4), keepdim=True) * (0.51 / (bins // 2 - 1))).all()
