"""Launches that ask for more shared memory than a kernel gets by itself: several threads with different shapes, and the
longest tables, whose columns take all that is given without asking."""
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


@pytest.mark.parametrize("T", [40, 256, 300])
@pytest.mark.parametrize("bins", [62, 63])
def test_longest_tables(T, bins):
    from cachegen_b200.serde import cachegen_decoder as D, cachegen_encoder as E
    L, H, dim = 2, 2, 64
    kv = torch.randn((L, 2, T, H, dim), generator=torch.Generator().manual_seed(T)).half().cuda()
    b = torch.full((L,), float(bins)).cuda()
    sym, _, cdf = E.quantize_and_tables(kv, b, b, 63)
    payload, _, offs = E.encode_streams(cdf, sym)
    out = E.encode_function(kv, None, b, b, T, max_bins=63)
    assert torch.equal(out.cdf, cdf)
    assert torch.equal(torch.cat([p.bytestream for p in out.data_chunks]), payload)
    got = D.decode_to_kv(out, torch.cat((b, b)), "vllm", torch.float16)
    flat = E.encode_flat(kv, b, b, max_bins=63)
    assert torch.equal(D.decode_to_kv(flat, torch.cat((b, b)), "vllm", torch.float16), got)


def test_longest_tables_with_delta_coding():
    from cachegen_b200.serde import cachegen_basics as B, cachegen_decoder as D, cachegen_encoder as E
    kv = torch.randn((2, 2, 70, 2, 64), generator=torch.Generator().manual_seed(2)).half().cuda()
    b, delta = torch.full((2,), 62.0).cuda(), B.DeltaCoding(4)
    # the same symbols whatever the tables' length, so the same values
    got, want = (D.decode_to_kv(E.encode_function(kv, None, b, b, 70, max_bins=m, delta=delta), torch.cat((b, b)), "vllm",
                                torch.float16, delta=delta) for m in (63, 62))
    assert torch.equal(got, want)
