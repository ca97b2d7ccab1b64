"""The status word that all callers of the extension module's functions share."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_the_status_word_is_zero_for_callers_on_other_streams(monkeypatch):
    import cachegen_b200.torchac_cuda as tc
    monkeypatch.setattr(tc, "_status", {})
    slow, failed = torch.cuda.Stream(), []
    with torch.cuda.stream(slow):
        used = [torch.full((1,), -1, dtype=torch.int32, device="cuda") for _ in range(64)]  # what the word's memory held before
        slow.synchronize()
        del used
        torch.cuda._sleep(100_000_000)
        tc._status_word(torch.device("cuda", torch.cuda.current_device()))

    def other():
        with torch.cuda.stream(torch.cuda.Stream()):
            try:
                tc.check_status()
            except RuntimeError as e:
                failed.append(e)
    t = threading.Thread(target=other)
    t.start()
    t.join()
    slow.synchronize()
    assert not failed
