"""Without the host module: the classes work all the same, through Python, and give the same."""
import sys

import pytest
import torch


@pytest.fixture
def unbuilt(monkeypatch):
    import cachegen_b200
    from cachegen_b200 import _lib, build
    build.build()
    monkeypatch.setattr(_lib, "_calls", None)
    monkeypatch.delattr(cachegen_b200, "_calls", raising=False)
    monkeypatch.setitem(sys.modules, "cachegen_b200._calls", None)  # importing it raises ImportError
    return _lib


def test_the_entries_are_there(unbuilt):
    with pytest.raises(unbuilt.CacheGenLibraryMissing):
        unbuilt.native_calls()
    with pytest.warns(RuntimeWarning, match="time on the host"):
        plain = unbuilt.calls()
    assert plain.decode([], None) is None and callable(plain.encode_start) and callable(plain.encode_finish)
    assert unbuilt.calls() is plain


def test_a_module_of_another_torch_is_not_used(monkeypatch):
    from cachegen_b200 import _lib, build
    build.build()
    _lib.native_calls()
    monkeypatch.setattr(torch, "__version__", "9.9")
    with pytest.raises(_lib.CacheGenLibraryMissing, match="this is torch 9.9"):
        _lib.native_calls()


def test_a_missing_library_is_still_an_error(unbuilt, monkeypatch):
    monkeypatch.setattr(unbuilt, "_lib", None)
    monkeypatch.setattr(unbuilt, "LIB_PATH", "/nowhere/libcachegen_b200.so")
    with pytest.raises(unbuilt.CacheGenLibraryMissing, match="nowhere"):
        unbuilt.calls()


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["vllm", "huggingface"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("delta", [None, 16])
@pytest.mark.filterwarnings("ignore:calls spend more time")
def test_encode_and_decode_are_the_same(unbuilt, monkeypatch, fmt, dtype, delta):
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenConfig, CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.serde.cachegen_basics import DeltaCoding
    from cachegen_b200.synth import generate_kv
    config = CacheGenConfig.from_model_name("Yukang/LongAlpaca-70B-16k").layer_slice(0, 10)
    engine, meta = LMCacheEngineConfig.from_defaults(chunk_size=1024), LMCacheEngineMetadata("m", 1, 0, fmt)
    delta = delta and DeltaCoding(delta)
    ser = CacheGenSerializer(engine, meta, config, table_max_bins=32, delta=delta)
    de = CacheGenDeserializer(engine, meta, config, out_dtype=dtype, delta=delta)
    kv = generate_kv(10, 2, 64, 300, seed=1, device="cuda", dtype=dtype)
    if fmt == "huggingface":
        kv = kv.permute(0, 1, 3, 2, 4)

    def run():
        chunks = [ser.encode(kv)] + ser.encode_many(kv, 128) + ([] if delta else ser.encode_levels(kv, [config, config.with_bins_divided(2)]))
        flat = ser.encode_flat(kv)
        return ([t for c in chunks for t in [c.cdf, c.max_tensors_key, c.max_tensors_value] + [x for p in c.data_chunks for x in (p.bytestream, p.bytestream_lengths)]]
                + [flat.blob, de.decode(chunks[0]), de.decode_many(chunks[1:4]), de.decode(flat), de.from_bytes(ser.to_bytes(kv))])

    from cachegen_b200 import _plain_calls
    plain = run()
    assert unbuilt.calls() is _plain_calls
    monkeypatch.undo()
    assert unbuilt.calls() is not _plain_calls
    native = run()
    assert len(plain) == len(native) and all(a.dtype == b.dtype and torch.equal(a, b) for a, b in zip(plain, native))
    de.check_status()
