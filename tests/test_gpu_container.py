"""A container is filled by one launch: every byte of it is written, whatever its memory held before, at channel counts that
fill no group, leave gaps between rows of masks, and in chunks of several sub-chunks."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compact", [True, "counts", False])
@pytest.mark.parametrize("heads, head, tokens", [(8, 128, 61), (1, 1, 7), (1, 13, 40), (3, 5, 33), (3, 24, 300), (5, 8, 700), (2, 64, 256)])
def test_every_byte_of_a_container(heads, head, tokens, compact):
    from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
    from cachegen_b200.serde import CacheGenConfig, CacheGenSerializer
    from cachegen_b200.serde import flat_format as ff
    from cachegen_b200.synth import generate_kv
    L = 10
    config = CacheGenConfig.from_model_name("Yukang/LongAlpaca-70B-16k").layer_slice(0, L)
    ser = CacheGenSerializer(LMCacheEngineConfig.from_defaults(chunk_size=1024), LMCacheEngineMetadata("m", 1, 0, "vllm"), config,
                             table_max_bins=32)
    kv = generate_kv(L, heads, head, tokens, seed=5, device="cuda", dtype=torch.float16)
    blobs = []
    for before in (255, 0):
        junk = [torch.full((n,), before, dtype=torch.uint8, device="cuda") for n in (1 << 12, 1 << 16, 1 << 20, 1 << 24) for _ in range(4)]
        del junk  # what the allocator gives out next held this
        chunk = ser.encode_flat(kv, compact)
        blobs.append(chunk.tobytes())
    assert blobs[0] == blobs[1]
    # the sections, from the chunk as separate tensors
    raw, h, eo, C = np.frombuffer(blobs[0], np.uint8), chunk.header, ser.encode(kv), heads * head
    want, known = np.zeros(h.total, np.uint8), np.zeros(h.total, bool)

    def put(at, data):
        data = np.frombuffer(data if isinstance(data, bytes) else np.ascontiguousarray(data).tobytes(), np.uint8)
        assert not known[at:at + data.size].any()
        want[at:at + data.size], known[at:at + data.size] = data, True
    put(0, h.pack())
    put(h.off_scales, torch.stack((eo.max_tensors_key, eo.max_tensors_value)).view(torch.int16).cpu().numpy())
    for j, piece in enumerate(eo.data_chunks):
        put(h.off_lengths + j * 4 * L * C, piece.bytestream_lengths.cpu().numpy().astype(np.uint16))
        put(h.off_payload + h.sub_off[j], piece.bytestream.cpu().numpy())
    if h.table_kind == ff.TABLES_CDF:
        put(h.off_tables, eo.cdf.cpu().numpy())
    else:
        bins = ser._info.cpu
        counts = ser.encode_flat(kv, "counts")
        dense = counts.blob[counts.header.off_tables:counts.header.off_lengths].cpu().numpy()
        rows, masks = ff.table_row_offsets(bins, C), ff.mask_row_offsets(bins, C)
        if h.table_kind == ff.TABLES_COUNTS:
            put(h.off_tables, dense[:rows[-1]])
        else:
            off_masks, off_counts = ff.sparse_parts(2 * L, C, masks[-1])
            groups, at = [0], h.off_tables + off_counts
            for r in range(2 * L):
                n = 2 * (int(bins[r]) // 2 - 1)
                of = dense[rows[r]:rows[r + 1]].reshape(n, C)
                mask = ((of > 0).astype(np.uint32) << np.arange(n, dtype=np.uint32)[:, None]).sum(0)
                put(h.off_tables + off_masks + masks[r], mask.astype(np.uint16 if n <= 16 else np.uint32))
                for g in range(0, C, 128):
                    some = of[:, g:g + 128].T
                    put(at, some[some > 0])
                    at += int((some > 0).sum())
                    groups.append(at - h.off_tables - off_counts)
            put(h.off_tables, np.array(groups, np.uint32))
    assert (raw == want).all()
