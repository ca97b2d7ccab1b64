"""The decode in native code gives what the general path gives wherever it takes a call, and leaves to it what that refuses or
has to stage first."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu

L, H, D = 10, 2, 64


@pytest.fixture(scope="module")
def parts():
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenConfig, CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.synth import generate_kv
    config = CacheGenConfig.from_model_name("Yukang/LongAlpaca-70B-16k").layer_slice(0, L)
    engine = LMCacheEngineConfig.from_defaults(chunk_size=1024)

    def make(fmt, out_dtype=torch.float16, dtype=torch.float16, tokens=(1, 300, 37)):
        meta = LMCacheEngineMetadata("m", 1, 0, fmt)
        kv = [generate_kv(L, H, D, t, seed=t, device="cuda", dtype=dtype) for t in tokens]
        if fmt == "huggingface":
            kv = [x.permute(0, 1, 3, 2, 4) for x in kv]
        return CacheGenSerializer(engine, meta, config, table_max_bins=32), CacheGenDeserializer(engine, meta, config, out_dtype), kv
    return make


def both(de, chunks, out=None):
    """(native result or None, the general path's)"""
    from cachegen_b200.serde import cachegen_decoder as M
    plan = M.DecodePlan(chunks, de._bins, de.fmt, de.out_dtype, workspace=de._workspace, host_bins=de._host_bins,
                        out=None if out is None else torch.full_like(out, 3.0))
    want = plan.run()
    return M._decode_usual(chunks, de._bins, de.fmt, de.out_dtype, out, de._workspace, de._host_bins), want


def same(a, b):
    return a.shape == b.shape and a.stride() == b.stride() and torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("wire", ["pickle", "sparse", "counts", "cdf"])
@pytest.mark.parametrize("fmt", ["vllm", "huggingface"])
@pytest.mark.parametrize("out_dtype, dtype", [(torch.float16, torch.float16), (torch.bfloat16, torch.float16), (torch.float16, torch.bfloat16)])
def test_native_decode_equals_the_general_path(parts, wire, fmt, out_dtype, dtype):
    ser, de, kv = parts(fmt, out_dtype, dtype)
    encode = ser.encode if wire == "pickle" else lambda x: ser.encode_flat(x, {"sparse": True, "counts": "counts", "cdf": False}[wire])
    chunks = [encode(x) for x in kv]
    for some in (chunks[:1], chunks[1:2], chunks):
        got, want = both(de, some)
        assert got is not None and same(got, want)
        got = de.decode_many(some)
        assert same(got, want)
    # a caller's tensor: a part of a larger one along the tokens, so that no stride is the result's own
    T = sum(x.shape[2 if fmt == "vllm" else 3] for x in kv)
    room = torch.zeros((L, 2, T + 5, H, D) if fmt == "vllm" else (L, 2, H, T + 5, D), dtype=out_dtype, device="cuda")
    part = room[:, :, 2:2 + T] if fmt == "vllm" else room[:, :, :, 2:2 + T]
    got, want = both(de, chunks, part)
    assert got.data_ptr() == part.data_ptr() and torch.equal(got.view(torch.int16), want.view(torch.int16))
    untouched = torch.ones_like(room, dtype=torch.bool)
    (untouched[:, :, 2:2 + T] if fmt == "vllm" else untouched[:, :, :, 2:2 + T]).zero_()
    assert not room[untouched].any()
    de.check_status()


def pieces(eo, **kw):
    return [dataclasses.replace(p, **{k: f(p) for k, f in kw.items()}) for p in eo.data_chunks]


# what the general path stages, copies or accepts as it is
OTHER = {
    "host": lambda eo: dataclasses.replace(eo, cdf=eo.cdf.cpu().pin_memory()),
    "host lengths": lambda eo: dataclasses.replace(eo, data_chunks=pieces(eo, bytestream_lengths=lambda p: p.bytestream_lengths.cpu())),
    "strided tables": lambda eo: dataclasses.replace(eo, cdf=torch.cat((eo.cdf, eo.cdf), 2)[:, :, :eo.cdf.shape[2]]),
    "strided scales": lambda eo: dataclasses.replace(eo, max_tensors_key=torch.stack((eo.max_tensors_key,) * 2, 2)[:, :, 0]),
    "strided bytes": lambda eo: dataclasses.replace(eo, data_chunks=pieces(eo, bytestream=lambda p: torch.stack((p.bytestream,) * 2, 1)[:, 0])),
    "parameter": lambda eo: dataclasses.replace(eo, max_tensors_key=torch.nn.Parameter(eo.max_tensors_key)),
    "flat scales": lambda eo: dataclasses.replace(eo, max_tensors_key=eo.max_tensors_key[..., 0]),
    "tuple of pieces": lambda eo: dataclasses.replace(eo, data_chunks=tuple(eo.data_chunks)),
}
# what it refuses
BAD = {
    "tables' type": lambda eo: dataclasses.replace(eo, cdf=eo.cdf.int()),
    "tables' shape": lambda eo: dataclasses.replace(eo, cdf=eo.cdf[:, :-1].contiguous()),
    "heads": lambda eo: dataclasses.replace(eo, num_heads=H + 1),
    "scales' type": lambda eo: dataclasses.replace(eo, max_tensors_value=eo.max_tensors_value.bfloat16()),
    "32-bit scales": lambda eo: dataclasses.replace(eo, max_tensors_key=eo.max_tensors_key.float(), max_tensors_value=eo.max_tensors_value.float()),
    "scales' shape": lambda eo: dataclasses.replace(eo, max_tensors_value=eo.max_tensors_value[:, :-1].contiguous()),
    "scales' layers": lambda eo: dataclasses.replace(eo, max_tensors_key=eo.max_tensors_key[:-1]),
    "tokens": lambda eo: dataclasses.replace(eo, data_chunks=pieces(eo, ntokens=lambda p: p.ntokens - 1)),
    "a piece less": lambda eo: dataclasses.replace(eo, data_chunks=eo.data_chunks[:-1]),
    "lengths' type": lambda eo: dataclasses.replace(eo, data_chunks=pieces(eo, bytestream_lengths=lambda p: p.bytestream_lengths.long())),
    "lengths": lambda eo: dataclasses.replace(eo, data_chunks=pieces(eo, bytestream_lengths=lambda p: p.bytestream_lengths[:-1])),
    "bytes' type": lambda eo: dataclasses.replace(eo, data_chunks=pieces(eo, bytestream=lambda p: p.bytestream.char())),
}


@pytest.mark.parametrize("kind", sorted(OTHER))
def test_other_chunks_are_left_to_the_general_path(parts, kind):
    ser, de, kv = parts("vllm")
    eo = ser.encode(kv[1])
    want = de.decode(eo).clone()
    other = OTHER[kind](eo)
    got, general = both(de, [other])
    assert same(general, want)
    assert got is None or (kind in ("flat scales", "parameter") and same(got, want))  # both are plain tensors with one scale a token
    assert same(de.decode(other), want)


@pytest.mark.parametrize("kind", sorted(BAD))
def test_malformed_chunks_are_refused_as_before(parts, kind):
    from cachegen_b200.serde import cachegen_decoder as M
    ser, de, kv = parts("vllm")
    eo = ser.encode(kv[1])
    de.decode(eo)  # the workspace has its buffers: the native path is tried
    bad = BAD[kind](eo)
    assert M._decode_usual([bad], de._bins, de.fmt, de.out_dtype, None, de._workspace, de._host_bins) is None
    with pytest.raises((RuntimeError, TypeError)):
        de.decode(bad)
    with pytest.raises((RuntimeError, TypeError)):
        de.decode_many([eo, bad])


@pytest.mark.parametrize("change", [dict(lp=20), dict(T=299), dict(H=4), dict(bins_checksum=12345), dict(off_lengths=1 << 30), dict(nsub=1),
                                    dict(scale_code=1)])
def test_containers_that_do_not_fit_are_left_to_the_general_path(parts, change):
    """With a good one in front; what the general path makes of them alone is its own affair."""
    from cachegen_b200.serde import cachegen_decoder as M
    from cachegen_b200.serde import flat_format
    ser, de, kv = parts("vllm")
    good = ser.encode_flat(kv[1], False if "lp" in change else True)
    de.decode(good)
    bad = flat_format.FlatChunk(good.blob, dataclasses.replace(good.header, **change))
    call = lambda chunks: M._decode_usual(chunks, de._bins, de.fmt, de.out_dtype, None, de._workspace, de._host_bins)
    assert call([good]) is not None
    if change != dict(T=299):  # (one token less in the header reads like a smaller container)
        assert call([good, bad]) is None
    assert call([good, ser.encode(kv[0])]) is None  # of two kinds


def test_outputs_that_do_not_fit_are_refused(parts):
    ser, de, kv = parts("vllm")
    eo = ser.encode(kv[2])
    de.decode(eo)
    T = kv[2].shape[2]
    for out in (torch.empty((L, 2, T, H, D), dtype=torch.bfloat16, device="cuda"), torch.empty((L, 2, T + 1, H, D), dtype=torch.float16, device="cuda"),
                torch.empty((L, 2, T, H, D), dtype=torch.float16), torch.empty((L, 2, T, H, 2 * D), dtype=torch.float16, device="cuda")[..., ::2]):
        with pytest.raises(RuntimeError):
            de.decode(eo, out=out)


def test_the_stream_of_a_native_decode_is_noted_and_used(parts):
    """On a side stream, behind other work, with the chunk's memory given back before it has run."""
    ser, de, kv = parts("vllm")
    want = de.decode(ser.encode(kv[1])).clone()
    side = torch.cuda.Stream()
    eo = ser.encode(kv[1])
    torch.cuda.synchronize()
    sizes = [p.bytestream.numel() for p in eo.data_chunks] + [eo.cdf.numel() * 2]
    with torch.cuda.stream(side):
        torch.cuda._sleep(50_000_000)
        got = de.decode(eo)
    del eo
    junk = [torch.full((n,), 255, dtype=torch.uint8, device="cuda") for n in sizes for _ in range(4)]
    side.synchronize()
    assert same(got, want)
    del junk
