"""from_bytes_many decodes on the GPU that the first chunk comes back on, whichever device is current.  Without a second
GPU: streams, loads and plans are stand-ins that note which device each step was given."""
import types

import pytest
import torch


class Stream:
    def __init__(self, device):
        self.device, self.waits = torch.device(device), []

    def wait_stream(self, other):
        self.waits.append(other)

    def wait_event(self, event):
        pass


@pytest.mark.parametrize("devices,want", [(["cuda:1", "cuda:1"], 1), (["cuda:0", "cuda:0"], 0), (["cpu", "cpu"], 0),
                                          (["cuda:1", "cpu", "flat"], 1), (["flat", "flat"], 0), (["cuda:1", "cuda:0"], 1)])
def test_from_bytes_many_decodes_where_the_first_chunk_is(monkeypatch, devices, want):
    from cachegen_b200.serde import cachegen_basics as B, cachegen_decoder as D
    dev = torch.device("cuda", want)
    cur, copies, plans, synced = {}, {}, [], []
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: cur.setdefault(torch.device(d), Stream(d)))
    monkeypatch.setattr(D, "_copy_stream", lambda d: copies.setdefault(d, Stream(d)))
    monkeypatch.setattr(torch.cuda, "synchronize", lambda d=None: synced.append(torch.device(d)))
    monkeypatch.setattr(torch.cuda, "Event", lambda: types.SimpleNamespace(record=lambda stream: None))
    monkeypatch.setattr(torch.cuda, "device", lambda d: B._NOTHING)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: B._NOTHING)

    class Load:
        pairs = ()

        def __enter__(self):
            return self

        def __exit__(self, *exc):
            pass

        def unpickle(self, blob):
            d = torch.device(blob.decode())
            self.pairs = [(0, 1, types.SimpleNamespace(device=d), None)] if d.type == "cuda" else []
            return types.SimpleNamespace(cdf=types.SimpleNamespace(device=d, is_cuda=d.type == "cuda"), num_heads=1, head_size=8,
                                         max_tensors_key=torch.zeros(1, 5, 1))

        def flat(self, blob, device):
            self.pairs = [(0, 1, types.SimpleNamespace(device=device), None)]
            return types.SimpleNamespace(cdf=types.SimpleNamespace(device=device, is_cuda=True), num_heads=1, head_size=8,
                                         max_tensors_key=torch.zeros(1, 5, 1))

        def send(self, stream):
            assert stream is copies[dev]

    class Plan:
        def __init__(self, chunks, bins, fmt, dtype, out=None, device=None, **kw):
            plans.append((torch.device(device), bins, out.shape[2]))

        def run(self):
            pass

    monkeypatch.setattr(B, "BlobLoad", Load)
    monkeypatch.setattr(D, "DecodePlan", Plan)
    monkeypatch.setattr(D.flat_format, "is_flat", lambda blob: blob == b"flat")
    de = object.__new__(D.CacheGenDeserializer)
    de.__dict__.update(fmt="vllm", chunk_size=256, out_dtype=torch.float16, delta=None, _workspace={}, _bins=torch.zeros(2),
                       _host_bins=None, _bins_on=lambda d: d)
    out = torch.zeros((1, 2, 5 * len(devices), 1, 8), dtype=torch.float16)
    assert de.from_bytes_many([d.encode() for d in devices], out=out) is out
    assert plans == [(dev, dev, 5)] * len(devices)
    assert list(copies) == [dev] and copies[dev].waits == [cur[dev]] and cur[dev].waits == [copies[dev]]
    assert set(synced) == {torch.device(d) for d in devices if d.startswith("cuda")} - {dev}  # tensors of another GPU
