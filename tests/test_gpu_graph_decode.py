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
