"""The offsets of 128-channel groups against a cumulative sum: fewer groups than a cluster has blocks, both sizes of clusters and
the line between them, groups that four lengths a load do not divide."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows, channels", [(1, 1), (1, 128), (7, 128), (3, 130), (2, 4096), (64, 2048), (64, 2049), (41, 3200), (64, 4096),
                                            (160, 1024), (5, 100003), (31, 4224)])
def test_group_offsets(rows, channels):
    from cachegen_b200 import _lib
    lib = _lib.lib()
    slabs = (channels + 127) // 128
    lengths = np.random.default_rng(rows * channels).integers(0, 521, (rows, channels)).astype(np.int32)
    sums = np.add.reduceat(lengths, np.arange(0, channels, 128), axis=1).astype(np.int64).reshape(-1)
    want = np.concatenate(([0], np.cumsum(sums)))
    dev = torch.from_numpy(lengths).cuda()
    tail = torch.zeros(4, dtype=torch.int64, pin_memory=True)
    for _ in range(3):  # behind each other: each is launched under the one in front
        off = torch.full((rows * slabs,), -1, dtype=torch.int64, device="cuda")
        assert lib.cg_stream_sizes(dev.data_ptr(), rows, channels, 520, None, off.data_ptr(), tail.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert tail.tolist() == [want[-1], 0, 0, 1]
        assert (off.cpu().numpy() == want[:-1]).all()


@pytest.mark.parametrize("heads, layers", [(8, 10), (20, 32), (32, 32)])
def test_offsets_follow_what_wrote_the_lengths(heads, layers):
    """A decode whose lengths a kernel right in front of it still writes: nothing is read before that has ended."""
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenConfig, CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.synth import generate_kv
    config = CacheGenConfig.from_model_name("Yukang/LongAlpaca-70B-16k").layer_slice(0, layers)
    engine, meta = LMCacheEngineConfig.from_defaults(chunk_size=256), LMCacheEngineMetadata("m", 1, 0, "vllm")
    ser, de = (CacheGenSerializer(engine, meta, config, table_max_bins=32), CacheGenDeserializer(engine, meta, config, out_dtype=torch.float16))
    eo = ser.encode(generate_kv(layers, heads, 128, 40, seed=2, device="cuda", dtype=torch.float16))
    want = de.decode(eo).clone()
    lengths, piece = eo.data_chunks[0].bytestream_lengths.clone(), eo.data_chunks[0]
    for _ in range(20):
        piece.bytestream_lengths.zero_()
        torch.add(lengths, 0, out=piece.bytestream_lengths)
        got = de.decode(eo)
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    de.check_status()


def test_offsets_of_several_batches_beside_each_other():
    """130 jobs are four batches, whose offsets are made at the same time: right behind a kernel that still writes the lengths, and again
    and again into the same buffer, which the decode in front may still read."""
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenConfig, CacheGenDeserializer, CacheGenSerializer
    from cachegen_b200.synth import generate_kv
    config = CacheGenConfig.from_model_name("Yukang/LongAlpaca-70B-16k").layer_slice(0, 10)
    engine, meta = LMCacheEngineConfig.from_defaults(chunk_size=256), LMCacheEngineMetadata("m", 1, 0, "vllm")
    ser, de = (CacheGenSerializer(engine, meta, config, table_max_bins=32), CacheGenDeserializer(engine, meta, config, out_dtype=torch.float16))
    chunks = [ser.encode(generate_kv(10, 4, 128, 20 + i, seed=i, device="cuda", dtype=torch.float16)) for i in range(3)]
    want = [de.decode(c).clone() for c in chunks]
    lengths = [c.data_chunks[0].bytestream_lengths.clone() for c in chunks]
    order = [i % 3 for i in range(130)]
    for turn in range(6):
        torch.cuda._sleep(200_000)
        for c, n in zip(chunks, lengths):
            c.data_chunks[0].bytestream_lengths.zero_()
        for c, n in zip(chunks, lengths):
            torch.add(n, 0, out=c.data_chunks[0].bytestream_lengths)
        order = order[turn:] + order[:turn]
        got = de.decode_many([chunks[i] for i in order])
        assert torch.equal(got.view(torch.int16), torch.cat([want[i] for i in order], 2).view(torch.int16)), turn
    de.check_status()
