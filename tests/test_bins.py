"""The bins an encode runs with are those that the tensors hold at the call, however they were made or written to."""
import pytest
import torch


def configs():
    from cachegen_b200.serde.cachegen_basics import CacheGenConfig
    base = CacheGenConfig(1, 2, 4, 32, 16, 16, 2, 32, 16)
    return base, base.with_bins_divided(2)


def serializer(config):
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenSerializer
    return CacheGenSerializer(LMCacheEngineConfig.from_defaults(chunk_size=256),
                              LMCacheEngineMetadata("bins", 1, 0, "vllm"), config)


def deserializer(config, delta=None):
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenDeserializer
    return CacheGenDeserializer(LMCacheEngineConfig.from_defaults(chunk_size=256),
                                LMCacheEngineMetadata("bins", 1, 0, "vllm"), config, torch.float16, delta)


def make_kv():
    return torch.randn((4, 2, 70, 2, 64), generator=torch.Generator().manual_seed(4)).half().cuda()


def parts(eo):
    return [eo.cdf, eo.max_tensors_key.view(torch.int16), eo.max_tensors_value.view(torch.int16),
            eo.data_chunks[0].bytestream, eo.data_chunks[0].bytestream_lengths]


def same(a, b):
    return all(torch.equal(x, y) for x, y in zip(parts(a), parts(b)))


def test_bins_made_in_inference_mode():
    from cachegen_b200.serde import cachegen_basics as B, cachegen_encoder as E
    base, _ = configs()
    with torch.inference_mode():
        info = E._BinsInfo(B.make_key_bins(base, "cpu"), B.make_value_bins(base, "cpu"))
    assert info.cpu.tolist() == [32, 16, 16, 16, 32, 32, 16, 16] and info.table_bins() == 32


class _Blob:
    """Looks like a KV blob on a GPU up to the checks."""
    dtype, is_cuda, shape, device = torch.float16, True, (4, 2, 70, 2, 64), "no device"

    def dim(self):
        return 5

    def stride(self, *at):
        return (2 * 70 * 128, 70 * 128, 128, 64, 1)[at[0]] if at else (2 * 70 * 128, 70 * 128, 128, 64, 1)


@pytest.mark.parametrize("keys,values", [(4, 3), (4, 5), (3, 4), (5, 4), (2, 2)])
def test_bins_of_other_counts_than_the_blob_has_rows_are_refused(keys, values):
    from cachegen_b200.serde import cachegen_encoder as E
    pair = torch.full((keys,), 16.0), torch.full((values,), 16.0)
    for encode in (lambda: E.encode_function(_Blob(), None, *pair, 70, max_bins=16), lambda: E.encode_levels(_Blob(), [pair]),
                   lambda: E.encode_flat(_Blob(), *pair, max_bins=16)):
        with pytest.raises(RuntimeError, match="bins describe"):
            encode()


def test_residual_bins_are_those_of_the_values():
    from cachegen_b200.serde.cachegen_basics import DeltaCoding
    delta = DeltaCoding(4, 2, "all")
    kb, vb = torch.tensor([32.0, 16.0]), torch.tensor([16.0, 16.0])
    assert delta.residual_bins(kb, vb, "cpu").tolist() == [16, 8, 8, 8]
    assert delta.residual_bins(vb, kb, "cpu").tolist() == [8, 8, 16, 8]
    kb.data[0] = 12
    assert delta.residual_bins(kb, vb, "cpu").tolist() == [6, 8, 8, 8]


@pytest.mark.gpu
def test_a_serializer_made_in_inference_mode_encodes():
    base, half = configs()
    kv = make_kv()
    want, want_half = serializer(base).encode(kv), serializer(half).encode(kv)
    flat, many = serializer(base).encode_flat(kv), serializer(base).encode_many(kv, 30)
    with torch.inference_mode():
        ser = serializer(base)
        assert same(ser.encode(kv), want)
        assert all(same(a, b) for a, b in zip(ser.encode_levels(kv, [base, half]), (want, want_half)))
        assert all(same(a, b) for a, b in zip(ser.encode_many(kv, 30), many))
        assert torch.equal(ser.encode_flat(kv).blob, flat.blob)
        assert len(ser.key_bins) == 4 and same(ser.encode(kv), want)
    assert same(ser.encode(kv), want)


@pytest.mark.gpu
@pytest.mark.parametrize("inference", [False, True])
def test_bins_that_were_written_to(inference):
    from cachegen_b200.serde import cachegen_basics as B, cachegen_encoder as E
    base, half = configs()
    kv = make_kv()
    want, want_half = serializer(base).encode(kv), serializer(half).encode(kv)
    with torch.inference_mode(inference):
        kb, vb = B.make_key_bins(base), B.make_value_bins(base)
        assert same(E.encode_function(kv, None, kb, vb, 70), want)
        kb.data.copy_(B.make_key_bins(half))  # no version counter sees this
        vb.data.copy_(B.make_value_bins(half))
        assert same(E.encode_function(kv, None, kb, vb, 70), want_half)

        ser = serializer(base)
        assert same(ser.encode(kv), want)
        ser.key_bins.data.copy_(kb)
        ser.value_bins.copy_(vb)
        assert same(ser.encode(kv), want_half)
        ser.key_bins, ser.value_bins = B.make_key_bins(base), B.make_value_bins(base)
        assert same(ser.encode(kv), want)
        assert torch.equal(ser.encode_flat(kv).blob, serializer(base).encode_flat(kv).blob)


@pytest.mark.gpu
def test_bins_of_a_subclass():
    from cachegen_b200.serde import CacheGenSerializer
    base, half = configs()

    class Halved(CacheGenSerializer):
        def make_key_bins(self, config):
            return super().make_key_bins(half)

        def make_value_bins(self, config):
            return super().make_value_bins(half)

    plain = serializer(half)
    ser = Halved(type("C", (), {"chunk_size": 256}), type("M", (), {"fmt": "vllm"}), base)
    kv = make_kv()
    assert same(ser.encode(kv), plain.encode(kv))


@pytest.mark.gpu
def test_bins_of_replaced_methods(monkeypatch):
    from cachegen_b200.serde import CacheGenDeserializer, CacheGenSerializer, cachegen_basics as B
    base, half = configs()
    kv = make_kv()
    flat = serializer(half).encode_flat(kv)
    want = deserializer(half).decode(flat)
    for cls in (CacheGenSerializer, CacheGenDeserializer):
        monkeypatch.setattr(cls, "make_key_bins", lambda self, config: B.make_key_bins(half))
        monkeypatch.setattr(cls, "make_value_bins", lambda self, config: B.make_value_bins(half))
    assert torch.equal(serializer(base).encode_flat(kv).blob, flat.blob)
    assert torch.equal(deserializer(base).decode(flat), want)


@pytest.mark.gpu
@pytest.mark.parametrize("compact", [True, "counts", False])
def test_one_workspace_for_decodes_with_different_bins(compact):
    from cachegen_b200.serde import cachegen_basics as B, cachegen_decoder as D, cachegen_encoder as E
    kv, ws = make_kv(), {}
    for config in (*configs(), configs()[0]):
        kb, vb = B.make_key_bins(config), B.make_value_bins(config)
        chunk, bins = E.encode_flat(kv, kb, vb, compact_tables=compact), torch.cat((kb, vb))
        got = D.decode_to_kv(chunk, bins, "vllm", torch.float16, workspace=ws)
        assert torch.equal(got, D.decode_to_kv(E.encode_function(kv, None, kb, vb, 70), bins, "vllm", torch.float16))
        assert int(ws["status"].item()) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("wire", ["pickle", "flat"])
@pytest.mark.parametrize("host,groups", [(False, 1), (False, 2), (True, 1), (True, 2), (True, None)])
def test_delta_coded_chunks_through_the_pipelined_decode(wire, host, groups):
    import dataclasses
    from cachegen_b200.serde import cachegen_basics as B, cachegen_decoder as D
    base, _ = configs()
    delta = B.DeltaCoding(4)
    ser, de = serializer(base), deserializer(base, delta)
    ser.delta = delta
    kvs = [make_kv(), make_kv().flip(2), make_kv().flip(0)]
    chunks = [ser.encode_flat(kv) if wire == "flat" else ser.encode(kv) for kv in kvs]
    want = torch.cat([de.decode(c) for c in chunks], dim=2)

    def pinned(c):
        if wire == "flat":
            return c.pin_memory()
        pin = lambda t: t.cpu().pin_memory()
        data = [dataclasses.replace(d, bytestream=pin(d.bytestream), bytestream_lengths=pin(d.bytestream_lengths)) for d in c.data_chunks]
        return dataclasses.replace(c, data_chunks=data, cdf=pin(c.cdf), max_tensors_key=pin(c.max_tensors_key),
                                   max_tensors_value=pin(c.max_tensors_value))
    given = [pinned(c) for c in chunks] if host else chunks
    for some in (given, given[:1]):
        got = de.decode_many_host(some, groups=groups)
        assert torch.equal(got, want[:, :, :70 * len(some)])
    bins = torch.cat((B.make_key_bins(base), B.make_value_bins(base)))
    got = D.decode_many_pipelined(given, bins, "vllm", torch.float16, groups=groups or 4, delta=delta)
    assert torch.equal(got, want)


@pytest.mark.gpu
def test_what_is_kept_from_a_call_in_inference_mode_serves_calls_outside_it(monkeypatch):
    import cachegen_b200.torchac_cuda as tc
    base, _ = configs()
    de, kv = deserializer(base), make_kv()
    chunks = [serializer(base).encode_flat(kv).pin_memory() for _ in range(2)]
    monkeypatch.setattr(tc, "_status", {})
    with torch.inference_mode():
        want = de.decode_many_host(chunks, groups=2)
        tc.check_status()
    assert torch.equal(de.decode_many_host(chunks, groups=2), want)
    for word, check in ((de.group_status_words()[0], de.check_status), (tc._status_word(kv.device), tc.check_status)):
        word.fill_(2)
        with pytest.raises(RuntimeError, match="stream lengths"):
            check()
        check()  # set back
