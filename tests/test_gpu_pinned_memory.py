"""Pinned memory that the GPU still writes to, or reads from, stays what it is until the GPU is done: after errors, and when
the thread that it belongs to has ended."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BUSY = 100_000_000  # cycles, some 50 ms: what is enqueued behind them has not run when the call returns


class Stop(Exception):
    pass


def written_after(buffer):
    """Whether the GPU writes to the buffer from here on."""
    buffer.zero_()
    torch.cuda.synchronize()
    return bool(buffer.any())


@pytest.mark.parametrize("call", ["encode_function", "encode_levels", "encode_many"])
def test_sizes_of_an_encode_that_fails_after_its_launch(monkeypatch, call):
    from cachegen_b200.serde import cachegen_encoder as E
    kv = torch.randn((2, 2, 40, 2, 64), generator=torch.Generator().manual_seed(1)).half().cuda()
    b = torch.full((2,), 16.0).cuda()
    run = {"encode_function": lambda: E.encode_function(kv, None, b, b, 40), "encode_levels": lambda: E.encode_levels(kv, [(b, b)]),
           "encode_many": lambda: E.encode_many(kv, b, b, 40)}[call]
    run()
    tail, empty = torch.zeros(64, dtype=torch.int64, pin_memory=True), torch.empty

    def no_memory(*size, **kw):
        if kw.get("dtype") == torch.int32:  # the lengths' tensors, made when the kernels have been launched
            raise Stop
        return empty(*size, **kw)
    monkeypatch.setattr(E, "_take_tail", lambda n: tail)
    monkeypatch.setattr(torch, "empty", no_memory)
    torch.cuda._sleep(BUSY)
    with pytest.raises(Stop):
        run()
    assert not written_after(tail)


@pytest.mark.parametrize("step", ["pickling", "collecting"])
def test_transfers_of_a_dump_that_fails(monkeypatch, step):
    from cachegen_b200.serde import cachegen_basics as B
    one = torch.arange(1 << 20, dtype=torch.int32).cuda()
    eo = B.CacheGenGPUEncoderOutput([B.CacheGenGPUBytestream(one.to(torch.uint8), one, 1)], one.short(), one.half(), one.half(), 1, 1)
    for _ in range(2):
        B.dump_blob(eo)  # both buffers are large enough from here on
    st, download = B.staging(), B._Staging._download

    def fail(*a):
        raise Stop

    def fail_second(self, phase):
        if phase == 2:
            raise Stop
        download(self, phase)
    if step == "pickling":
        monkeypatch.setattr(B._BlobPickler, "dump", fail)
    else:
        monkeypatch.setattr(B._Staging, "_download", fail_second)
    torch.cuda._sleep(BUSY)
    with pytest.raises(Stop):
        B.dump_blob(eo)
    assert not written_after(st.bufs[st.turn])
    monkeypatch.undo()
    assert B.load_blob(B.dump_blob(eo)).cdf.equal(eo.cdf)


def test_uploads_of_a_thread_that_has_ended():
    import threading
    from cachegen_b200.serde import cachegen_basics as B
    host = torch.arange(3 << 20, dtype=torch.int32).to(torch.uint8)
    device, got = torch.device("cuda", torch.cuda.current_device()), []

    def upload():
        B.staging().begin(host.numel())  # pins the memory; the copies below take the other buffer
        B.staging().end()
        torch.cuda._sleep(BUSY)
        got.append((B.staging().whole_to_device(host, device), B.staging().bufs[B.staging().turn].numel()))
    t = threading.Thread(target=upload)
    t.start()
    t.join()
    del t
    others = [torch.empty(got[0][1], dtype=torch.uint8, pin_memory=True).fill_(255) for _ in range(4)]
    assert torch.equal(got[0][0].cpu(), host) and len(others) == 4


def test_threads_that_come_and_go():
    import threading
    from cachegen_b200.serde import cachegen_basics as B
    data, same = torch.arange(1 << 18, dtype=torch.int32).cuda(), []

    def there_and_back():
        same.append(B.staging().whole_from_device(data) == data.cpu().numpy().tobytes())
    for _ in range(20):
        t = threading.Thread(target=there_and_back)
        t.start()
        t.join()
    assert same == [True] * 20
