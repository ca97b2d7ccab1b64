"""A decode captured into a graph, its offsets' launch behind a copy, behind a kernel and first of all: a replay decodes what the chunk's
tensors hold by then."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("front", ["copy", "kernel", "nothing"])
@pytest.mark.parametrize("chunks", [1, 45])
def test_captured_decode(front, chunks):
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenConfig, CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.synth import generate_kv
    config = CacheGenConfig.from_model_name("Yukang/LongAlpaca-70B-16k").layer_slice(0, 10)
    engine, meta = LMCacheEngineConfig.from_defaults(chunk_size=256), LMCacheEngineMetadata("m", 1, 0, "vllm")
    ser, de = (CacheGenSerializer(engine, meta, config, table_max_bins=32), CacheGenDeserializer(engine, meta, config, out_dtype=torch.float16))
    eo = ser.encode(generate_kv(10, 4, 128, 50, seed=2, device="cuda", dtype=torch.float16))
    lengths = eo.data_chunks[0].bytestream_lengths
    kept, out = lengths.clone(), torch.empty((10, 2, 50 * chunks, 4, 128), dtype=torch.float16, device="cuda")
    want = de.decode_many([eo] * chunks).clone()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        de.decode_many([eo] * chunks, out=out)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        if front == "copy":
            lengths.copy_(kept)
        elif front == "kernel":
            torch.add(kept, 0, out=lengths)
        de.decode_many([eo] * chunks, out=out)
    for _ in range(3):
        out.zero_()
        if front != "nothing":
            lengths.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    de.check_status()


@pytest.mark.parametrize("wire", ["pickle", "flat", "general"])
def test_other_decodes_between_capture_and_replay(wire):
    """A larger decode and one of other channels replace what the deserializer keeps, and the memory that they give back goes to others:
    a replay neither writes to it nor reads from it."""
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenConfig, CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.synth import generate_kv
    config = CacheGenConfig.from_model_name("Yukang/LongAlpaca-70B-16k").layer_slice(0, 10)
    engine, meta = LMCacheEngineConfig.from_defaults(chunk_size=256), LMCacheEngineMetadata("m", 1, 0, "vllm")
    ser, de = (CacheGenSerializer(engine, meta, config, table_max_bins=32), CacheGenDeserializer(engine, meta, config, out_dtype=torch.float16))
    encode = ser.encode_flat if wire == "flat" else ser.encode
    first, other = (encode(generate_kv(10, heads, 128, 50, seed=heads, device="cuda", dtype=torch.float16)) for heads in (4, 2))
    if wire == "general":  # a chunk that the native call leaves to DecodePlan
        first.data_chunks = tuple(first.data_chunks)
    out = torch.empty((10, 2, 50, 4, 128), dtype=torch.float16, device="cuda")
    want = de.decode(first).clone()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        de.decode(first, out=out)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        de.decode(first, out=out)
    kept = {k: v for k, v in de._workspace.items() if isinstance(v, torch.Tensor)}
    sizes = [t.numel() * t.element_size() for t in kept.values()]
    place = kept["group_off"].data_ptr()
    del kept
    de.decode_many([first] * 45)
    want_other = de.decode(other).clone()
    assert de._workspace["group_off"].data_ptr() != place
    junk, got = [], [t for t in de._workspace.values() if isinstance(t, torch.Tensor)]
    # until what was given back is somebody else's
    while not any(t.data_ptr() <= place < t.data_ptr() + t.numel() * t.element_size() for t in got + junk[-len(sizes):]):
        junk += [torch.full((n,), 0xA5, dtype=torch.uint8, device="cuda") for n in sizes]
        assert len(junk) < 20000
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert all((t == 0xA5).all() for t in junk)
    assert torch.equal(de.decode(other).view(torch.int16), want_other.view(torch.int16))
    assert torch.equal(de.decode(first).view(torch.int16), want.view(torch.int16))
    de.check_status()
