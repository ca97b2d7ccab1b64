"""Lifetimes in the decode that copies one group of chunks while another is decoded."""
import pytest
import torch

from test_gpu_serde import make_serde

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wire", ["flat", "pickle"])
def test_pipelined_decode_notes_the_stream_that_reads_its_temporaries(monkeypatch, wire):
    """What is made on the copy stream and read by the decode on the caller's stream must not go back to the copy
    stream's pool before the decode has run."""
    from cachegen_b200.serde import cachegen_decoder as D
    from cachegen_b200.synth import generate_kv
    ser, de = make_serde(1024, "vllm", out_dtype=torch.float16)
    kv = generate_kv(32, 2, 64, 100, seed=3, device="cpu", dtype=torch.float16).cuda()
    chunks = [ser.encode_flat(kv).pin_memory() for _ in range(3)] if wire == "flat" else [ser.encode(kv) for _ in range(3)]
    if wire == "pickle":
        for c in chunks:
            c.cdf = c.cdf.cpu().pin_memory()
    noted, plans, record, init = [], [], torch.Tensor.record_stream, D.DecodePlan.__init__
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: (noted.append((t.data_ptr(), s.cuda_stream)), record(t, s))[1])
    monkeypatch.setattr(D.DecodePlan, "__init__", lambda p, *a, **kw: (plans.append(p), init(p, *a, **kw))[1])
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        D.decode_many_pipelined(chunks, de._bins_on(kv.device), de.fmt, torch.float16, groups=3)
    side.synchronize()
    assert len(plans) == 3
    for p in plans:
        for t in (p.goff, p.status, *p.keep):
            assert (t.data_ptr(), side.cuda_stream) in noted
