"""Launches that ask for more shared memory than a kernel gets by itself: several threads with different shapes."""
import ctypes
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def pending(L, T, H, D, bins, max_bins=None):
    from cachegen_b200.serde import cachegen_encoder as E
    kv = torch.randn((L, 2, T, H, D), generator=torch.Generator().manual_seed(L)).half().cuda()
    b = torch.full((L,), float(bins)).cuda()
    return E._PendingChunk(kv, E._BinsInfo(b, b), max_bins or bins)


@pytest.mark.parametrize("tokens", [256, 300])  # one sub-chunk (tables in the coder's launch), two
def test_threads_with_different_shapes_do_not_lower_each_others_limit(tokens):
    from cachegen_b200 import _lib
    lib, codes = _lib.lib(), []
    jobs = [pending(L, tokens, 8, 128, 32) for L in (32, 10, 5)]  # 512, 160 and 80 blocks: other paddings of the last wave
    torch.cuda.synchronize()

    def launch(p):
        stream = torch.cuda.Stream()
        codes.append({lib.cg_encode_kv(ctypes.byref(p.job), ctypes.c_void_p(stream.cuda_stream)) for _ in range(1500)})
        stream.synchronize()

    threads = [threading.Thread(target=launch, args=(p,)) for p in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for p in jobs:
        p.abandon()
    assert codes == [{0}] * len(jobs)
