"""The encode of a chunk in fused launches (cg_encode_kv and its gathers) against the separate calls, which the other
tests hold against the oracle, at the edges of its tiles: tokens around words of four, groups of sixteen and
sub-chunks of 256, channels around groups of 128, and shapes that the fused passes leave to the separate calls."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def bins_of(L, level):
    first = torch.full((L,), float(level))
    first[L // 2:] = max(4, level // 2)
    return first.cuda(), first.flip(0).contiguous().cuda()


def make_kv(L, T, H, D, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    kv = torch.randn((L, 2, T, H, D), generator=g) * torch.exp(torch.randn((L, 2, 1, H, D), generator=g))
    kv[:, :, T // 2] = 0  # an all-zero token
    return kv.to(dtype).cuda()


@pytest.mark.parametrize("T", [1, 3, 4, 5, 15, 17, 255, 256, 257, 260, 515])
@pytest.mark.parametrize("H,D,dtype", [(1, 8, torch.float16), (2, 64, torch.bfloat16), (3, 80, torch.float16),
                                       (17, 8, torch.bfloat16), (1, 130, torch.float16), (3, 7, torch.bfloat16)])
def test_fused_encode_equals_the_separate_calls(T, H, D, dtype):
    from cachegen_b200.serde import cachegen_encoder as E
    L = 2
    kb, vb = bins_of(L, 32)
    kv = make_kv(L, T, H, D, dtype, 1000 * T + H)
    sym, scales, cdf, counts, _ = E.quantize_and_tables(kv, kb, vb, 32, with_counts=True)
    payload, lengths, offs = E.encode_streams(cdf, sym)
    out = E.encode_function(kv, None, kb, vb, T)
    assert torch.equal(out.cdf, cdf)
    assert torch.equal(out.max_tensors_key[..., 0].view(torch.int16), scales[:L].view(torch.int16))
    assert torch.equal(out.max_tensors_value[..., 0].view(torch.int16), scales[L:].view(torch.int16))
    assert len(out.data_chunks) == len(offs) - 1
    for j, piece in enumerate(out.data_chunks):
        assert torch.equal(piece.bytestream_lengths, lengths[j])
        assert torch.equal(piece.bytestream, payload[offs[j]:offs[j + 1]])
    flat = E.encode_flat(kv, kb, vb, compact_tables="counts")
    if flat.header.table_kind == 1:
        assert torch.equal(flat.tables()[:counts.numel()], counts)
    assert torch.equal(flat.blob[flat.header.off_payload:], payload)


def test_streams_of_high_entropy_overflow_the_gather_stage():
    # uniform symbols: five bits each, more than the shared memory of a warp's run holds
    from cachegen_b200.serde import cachegen_encoder as E
    L, T, H, D = 1, 256, 2, 128
    kb = vb = torch.full((L,), 62.0).cuda()
    kv = torch.rand((L, 2, T, H, D), generator=torch.Generator().manual_seed(5)).mul(2).sub(1).half().cuda()
    sym, _, cdf = E.quantize_and_tables(kv, kb, vb, 62)
    payload, _, _ = E.encode_streams(cdf, sym)
    assert payload.numel() > 2 * L * H * D * 150
    assert torch.equal(E.encode_function(kv, None, kb, vb, T).data_chunks[0].bytestream, payload)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_kv_that_is_not_finite_is_reported(value):
    from cachegen_b200.serde import cachegen_encoder as E
    kb, vb = bins_of(2, 32)
    kv = make_kv(2, 40, 2, 64, torch.float16, 9)
    kv[1, 0, 7, 1, 3] = value
    with pytest.raises(RuntimeError, match="outside the table"):
        E.encode_function(kv, None, kb, vb, 40)
    E.encode_function(make_kv(2, 40, 2, 64, torch.float16, 9), None, kb, vb, 40)  # and nothing is left behind


@pytest.mark.parametrize("nbytes", [1, 255, 256, 4097, 128 << 10, (512 << 10) + 1, (9 << 20) + 13])
def test_byte_strings_to_the_gpu_and_back(nbytes):
    from cachegen_b200.serde.cachegen_basics import staging
    g = torch.Generator().manual_seed(nbytes)
    host = torch.randint(0, 256, (nbytes,), generator=g, dtype=torch.uint8)
    for _ in range(4):  # results in fresh memory and in memory used before
        dev = staging().whole_to_device(host, torch.device("cuda", torch.cuda.current_device()))
        assert staging().whole_from_device(dev) == host.numpy().tobytes()


def test_more_sub_chunks_than_one_launch_takes():
    from cachegen_b200 import _lib
    from cachegen_b200.serde import cachegen_decoder as D, cachegen_encoder as E
    L, H, dim, n = 1, 2, 64, 2 * _lib.CG_MAX_DECODE_JOBS + 3
    kb, vb = bins_of(L, 16)
    kv = make_kv(L, 5 * n, H, dim, torch.float16, 3)
    chunks = E.encode_many(kv, kb, vb, 5)
    bins = torch.cat((kb, vb))
    ws = {}
    got = D.decode_many(chunks, bins, "vllm", torch.float16, workspace=ws)
    want = torch.cat([D.decode_to_kv(c, bins, "vllm", torch.float16) for c in chunks], dim=2)
    assert int(ws["status"].item()) == 0 and torch.equal(got.view(torch.int16), want.view(torch.int16))


def test_encode_many_of_a_cache_with_another_innermost_stride(monkeypatch):
    """What has to be copied first is copied before the side streams start, not beside them."""
    from cachegen_b200.serde import cachegen_encoder as E
    kb, vb = bins_of(2, 16)
    kv = make_kv(2, 90, 2, 64, torch.float16, 6)
    want = E.encode_many(kv, kb, vb, 30)
    strided, contiguous = kv.transpose(3, 4).contiguous().transpose(3, 4), torch.Tensor.contiguous

    def late(t, *a, **kw):  # copies of the cache, or of a part of it, run some 20 ms after they were asked for
        if t.dim() == 5:
            torch.cuda._sleep(40_000_000)
        return contiguous(t, *a, **kw)
    monkeypatch.setattr(torch.Tensor, "contiguous", late)
    torch.cuda.synchronize()
    got = E.encode_many(strided, kb, vb, 30)
    assert strided.stride(4) != 1 and len(got) == 3
    for a, b in zip(got, want):
        assert torch.equal(a.cdf, b.cdf) and torch.equal(a.data_chunks[0].bytestream, b.data_chunks[0].bytestream)
