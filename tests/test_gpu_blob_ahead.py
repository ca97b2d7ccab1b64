"""Blobs whose bytes go to the GPU while they are parsed (from 2 MB on): every tensor at whatever byte it lies, on other streams
and in several threads, after blobs that fail, several blobs at once."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec():
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.synth import generate_kv
    config = LMCacheEngineConfig.from_defaults(chunk_size=1024)
    meta = LMCacheEngineMetadata("lmsys/longchat-7b-16k", 1, 0, "vllm")
    make = lambda: CacheGenDeserializer(config, meta, out_dtype=torch.float16)
    ser = CacheGenSerializer(config, meta)
    kv = lambda tokens, seed: generate_kv(32, 5, 128, tokens, seed, device="cuda", dtype=torch.float16)
    return ser, make, kv


@pytest.mark.parametrize("tokens", [33, 100, 255, 256, 257, 300, 611])
def test_blob_equals_decode_of_the_chunk(codec, tokens):
    ser, make, kv = codec
    for seed in range(3):
        x = kv(tokens, seed)
        blob = ser.to_bytes(x)
        assert len(blob) > 2 << 20
        want = make().decode(ser.encode(x))
        assert torch.equal(make().from_bytes(blob), want)
        assert torch.equal(make().from_bytes(bytearray(blob)), want)


def test_other_streams(codec):
    ser, make, kv = codec
    x = kv(256, 7)
    blob, want = ser.to_bytes(x), make().decode(ser.encode(x))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(5):
            out = make().from_bytes(blob)
    side.synchronize()
    assert torch.equal(out, want)


def test_blobs_that_fail(codec):
    ser, make, kv = codec
    x = kv(256, 9)
    blob, want = ser.to_bytes(x), make().decode(ser.encode(x))
    for bad in (blob[:len(blob) // 2], blob[:-3], b"\x80\x04" + blob[2:1 << 20] + bytes(2 << 20)):
        with pytest.raises(Exception):
            make().from_bytes(bad)
        assert torch.equal(make().from_bytes(blob), want)
    assert torch.equal(make().from_bytes_many([blob, blob]), torch.cat((want, want), dim=2))
    with pytest.raises(Exception):
        make().from_bytes_many([blob, blob[:len(blob) // 2], blob])
    assert torch.equal(make().from_bytes(blob), want)


def test_several_blobs_and_threads(codec):
    ser, make, kv = codec
    xs = [kv(t, t) for t in (256, 256, 100, 37)]
    blobs = [ser.to_bytes(x) for x in xs]
    want = torch.cat([make().decode(ser.encode(x)) for x in xs], dim=2)
    failed = []

    def work():
        try:
            de = make()
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(4):
                    assert torch.equal(de.from_bytes_many(blobs), want)
                    for blob, part in zip(blobs, want.split([256, 256, 100, 37], dim=2)):
                        assert torch.equal(de.from_bytes(blob), part)
        except BaseException as e:
            failed.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_calls_that_follow_each_other_without_a_wait(codec):
    # everything that a blob passes through (pinned memory, its copy on the GPU, tensors) is used again by the next ones
    ser, make, kv = codec
    xs = [kv(256, 20 + k) * (0.01 * 3 ** k) for k in range(6)]
    blobs = [ser.to_bytes(x) for x in xs]
    want = [make().decode(ser.encode(x)) for x in xs]
    de = make()
    torch.cuda.synchronize()
    for _ in range(4):
        single = [de.from_bytes(blob) for blob in blobs]
        many = [de.from_bytes_many(blobs[k:] + blobs[:k]) for k in range(6)]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(single, want))
        for k, out in enumerate(many):
            assert torch.equal(out, torch.cat(want[k:] + want[:k], dim=2)), k
