"""Which blobs leave for the GPU before they are parsed: those whose tensors belong to the current one."""
import pickle

import pytest
import torch

from cachegen_b200.serde import cachegen_basics as B


def chunk(device, nbytes):
    lengths = torch.full((4, 8), 3, dtype=torch.int32, device=device)
    scales = torch.ones((2, 16, 1), dtype=torch.float16, device=device)
    return B.CacheGenGPUEncoderOutput([B.CacheGenGPUBytestream(torch.arange(nbytes, device=device).to(torch.uint8), lengths, 16)],
                                      torch.zeros((4, 8, 33), dtype=torch.int16, device=device), scales, scales * 2, 1, 8)


@pytest.mark.parametrize("nbytes", [10, 1000, 70000, 3 << 20])
def test_location_of_a_blobs_first_storage(nbytes):
    for blob in (B.dump_blob(chunk("cpu", nbytes)), pickle.dumps(chunk("cpu", nbytes))):
        assert B._blob_location(blob) == "cpu"
        for short in (0, 1, 30, 400):
            assert B._blob_location(blob[:short]) is None
    for location in ("cpu", "cuda:0", "cuda:1", "cuda:15"):
        head = B._legacy_stream_head(torch.int16, "94", location, nbytes)
        assert B._blob_location(b"\x80\x04names B\0\0\0\0" + head + bytes(nbytes)) == location
    assert B._blob_location(bytes(nbytes)) is None
    assert B._blob_location(b"x" * B._FIRST_STREAM_WITHIN + B.dump_blob(chunk("cpu", nbytes))) is None


@pytest.mark.gpu
def test_only_blobs_of_the_current_gpu_are_sent_ahead():
    st = B.staging()
    size = 3 << 20
    for location, early, ahead in (("cpu", False, False), ("cuda:0", True, True), ("cuda:1", True, False), (None, True, False)):
        head = B._legacy_stream_head(torch.int16, "94", location, size) if location else b""
        blob = b"\x80\x04names B\0\0\0\0" + head + bytes(size)  # kept until its copies are done
        with torch.cuda.device(0):
            st.start(blob, ahead=True)
        try:
            assert (st.early is not None) == early, location
            assert early is False or (st.early[3] is not None) == ahead, location
        finally:
            st.finish()


@pytest.mark.gpu
def test_a_blob_of_host_tensors_takes_no_memory_of_the_gpu():
    eo = chunk("cpu", 24 << 20)
    blob = B.dump_blob(eo)
    B.load_blob(B.dump_blob(chunk("cuda", 3 << 20)))  # what is made once
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = B.load_blob(blob)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() == before
    assert got.cdf.device.type == "cpu" and torch.equal(got.data_chunks[0].bytestream, eo.data_chunks[0].bytestream)


@pytest.mark.gpu
@pytest.mark.parametrize("host_first", [True, False])
def test_blobs_with_tensors_on_both_sides(host_first):
    eo, size = chunk("cuda", 5 << 20), 5 << 20
    if host_first:
        eo.data_chunks[0].bytestream = eo.data_chunks[0].bytestream.cpu()
    else:
        eo.cdf, eo.data_chunks[0].bytestream_lengths = eo.cdf.cpu(), eo.data_chunks[0].bytestream_lengths.cpu()
    for blob in (B.dump_blob(eo), pickle.dumps(eo)):
        assert len(blob) > size
        got = B.load_blob(blob)
        torch.cuda.synchronize()
        for a, b in zip([got.cdf, got.max_tensors_key, got.max_tensors_value, *vars(got.data_chunks[0]).values()],
                        [eo.cdf, eo.max_tensors_key, eo.max_tensors_value, *vars(eo.data_chunks[0]).values()]):
            assert (a.device == b.device and torch.equal(a, b)) if isinstance(a, torch.Tensor) else a == b
