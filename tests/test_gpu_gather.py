"""The gather of streams takes `length` bytes of every row and none of what lies behind them."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rows_of(rng, NL, C, stride, most):
    buf = rng.integers(0, 256, (NL, C, stride), dtype=np.uint8)  # no row is zero behind its stream
    lens = rng.integers(0, most + 1, (NL, C)).astype(np.int32)
    lens[0, C - 1], lens[0, 0] = 0, most
    return buf, lens


def gathered(buf, lens):
    b, n = buf.reshape(-1, buf.shape[-1]), lens.reshape(-1)
    return np.concatenate([b[i, :n[i]] for i in range(len(n))])


@pytest.mark.parametrize("C", [1, 31, 32, 33, 127, 128, 129, 300])
# runs that a warp's shared memory takes at once (up to 5,105 bytes), in halves (from 32 rows of 160 on) and in quarters
@pytest.mark.parametrize("stride,most", [(4, 1), (4, 4), (8, 7), (12, 9), (64, 61), (188, 188), (192, 192), (196, 195), (520, 519)])
def test_collect_bytes_of_rows_with_data_behind_the_streams(C, stride, most):
    from cachegen_b200.serde import cachegen_encoder as E
    buf, lens = rows_of(np.random.default_rng(C * 1000 + stride), 3, C, stride, most)
    got = E.collect_bytes(torch.from_numpy(buf).cuda(), torch.from_numpy(lens).cuda())
    assert got.cpu().numpy().tobytes() == gathered(buf, lens).tobytes()


@pytest.mark.parametrize("short", [0, 1, 2, 3, 5, 16])
def test_runs_that_fill_a_warps_shared_memory(short):
    from cachegen_b200.serde import cachegen_encoder as E
    # 32 streams of 192 bytes go in halves; the first one starts its warp's run at every offset from 16 bytes
    buf, lens = rows_of(np.random.default_rng(short), 2, 128, 196, 192)
    lens[:] = 192
    lens[:, 32] -= short
    lens[0, 5] = 192 - short
    got = E.collect_bytes(torch.from_numpy(buf).cuda(), torch.from_numpy(lens).cuda())
    assert got.cpu().numpy().tobytes() == gathered(buf, lens).tobytes()


@pytest.mark.parametrize("C", [1, 31, 128, 161])
# what a warp's shared memory takes whatever byte its run starts at: 5,105 bytes, as one run, in halves and in quarters of the
# warp; what does not fit then goes byte by byte
@pytest.mark.parametrize("parts", [1, 2, 4])
@pytest.mark.parametrize("above", [-1, 0, 1, 40])
def test_runs_on_both_sides_of_what_fits(C, parts, above):
    from cachegen_b200.serde import cachegen_encoder as E
    n = 32 // parts
    each, rest = divmod(5105 + above, n)
    stride = (each + rest + 7) // 4 * 4
    buf, lens = rows_of(np.random.default_rng(C + 100 * parts + above), 3, C, stride, each)
    lens[:] = each
    lens[:, ::n] += rest
    lens[2] = np.random.default_rng(parts).integers(0, stride + 1, C)  # parts of every kind in a warp
    got = E.collect_bytes(torch.from_numpy(buf).cuda(), torch.from_numpy(lens).cuda())
    assert got.cpu().numpy().tobytes() == gathered(buf, lens).tobytes()


@pytest.mark.parametrize("offset", range(16))
def test_the_longest_run_at_once_from_every_byte(offset):
    from cachegen_b200.serde import cachegen_encoder as E
    buf, lens = rows_of(np.random.default_rng(offset), 2, 64, 176, 160)
    lens[:] = 0
    lens[0, 3] = offset  # the first warp's run; the second one's starts there, 32 streams of 5,105 and then of 5,106 bytes
    lens[0, 32:] = 159
    lens[0, 40] += 17
    lens[1, 32:] = 159
    lens[1, 32] += 1  # (and starts where the first row's ends)
    lens[1, 40] += 17
    got = E.collect_bytes(torch.from_numpy(buf).cuda(), torch.from_numpy(lens).cuda())
    assert got.cpu().numpy().tobytes() == gathered(buf, lens).tobytes()


def test_several_sub_chunks_through_the_c_abi():
    from cachegen_b200 import _lib
    NL, C, stride, nsub = 2, 200, 100, 3
    rng = np.random.default_rng(8)
    parts = [rows_of(rng, NL, C, stride, 99) for _ in range(nsub)]
    sizes = np.array([[p[1][r, c:c + 128].sum() for r in range(NL) for c in range(0, C, 128)] for p in parts], dtype=np.int64)
    group_off = np.cumsum(sizes, axis=1) - sizes
    sub_off = np.concatenate(([0], np.cumsum(sizes.sum(axis=1))))
    dev = [torch.from_numpy(a).cuda() for a in (np.stack([p[0] for p in parts]), np.stack([p[1] for p in parts]), group_off, sub_off)]
    out = torch.empty(int(sub_off[-1]), dtype=torch.uint8, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in (*dev, out)]
    rc = _lib.lib().cg_compact_streams(p[0], stride, p[1], p[2], p[3], nsub, NL, C, p[4],
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and out.cpu().numpy().tobytes() == np.concatenate([gathered(*q) for q in parts]).tobytes()


def test_recombined_rows_are_collected_again():
    from cachegen_b200.serde import cachegen_decoder as D, cachegen_encoder as E
    buf, lens = rows_of(np.random.default_rng(3), 4, 130, 256, 90)
    lens_t = torch.from_numpy(lens).cuda()
    b = torch.from_numpy(gathered(buf, lens)).cuda()
    assert torch.equal(E.collect_bytes(D.recombine_bytes(b, lens_t), lens_t), b)


def test_collect_bytes_keeps_no_tensor_filled_on_one_callers_stream(monkeypatch):
    """A tensor that is filled on the first caller's stream and kept would be read on another stream before it is."""
    from cachegen_b200.serde import cachegen_encoder as E
    buf, lens = rows_of(np.random.default_rng(4), 2, 60, 64, 50)
    buf_t, lens_t = torch.from_numpy(buf).cuda(), torch.from_numpy(lens).cuda()

    def refuse(*a, **kw):
        raise AssertionError("a filled tensor")
    for name in ("zeros", "full", "tensor", "zeros_like"):
        monkeypatch.setattr(torch, name, refuse)
    for value in vars(E).values():
        if hasattr(value, "cache_clear"):
            value.cache_clear()
    for _ in range(2):
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
            got = E.collect_bytes(buf_t, lens_t).cpu()
        assert got.numpy().tobytes() == gathered(buf, lens).tobytes()


def test_collect_bytes_refuses_lengths_in_host_memory():
    from cachegen_b200.serde import cachegen_encoder as E
    buf, lens = rows_of(np.random.default_rng(5), 2, 60, 64, 50)
    with pytest.raises(RuntimeError, match="on the buffer's GPU"):
        E.collect_bytes(torch.from_numpy(buf).cuda(), torch.from_numpy(lens))


def test_the_finest_bins_are_gathered_like_others():
    """Uniform values at the most bins an encode accepts give streams of 184 bytes: their runs pass through shared memory too
    (copied byte by byte they take 20 times as long as others)."""
    from cachegen_b200 import _lib
    from cachegen_b200.serde import cachegen_encoder as E
    kv = (torch.rand((8, 2, 256, 32, 128), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") * 2 - 1).half()
    times = {}
    for bins in (24, 63):
        b = torch.full((8,), float(bins))
        p = E._PendingChunk(kv, E._BinsInfo(b, b), bins)
        try:
            size = p.sizes()[0][1]
            out = torch.empty(size, dtype=torch.uint8, device="cuda")
            pointer = p.pointers(out.data_ptr())
            best = float("inf")
            for _ in range(12):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for _ in range(20):
                    _lib.check(p.lib.cg_encode_kv_gather(ctypes.byref(p.job), pointer, p.length_pointers, p.stream_ptr), "gather")
                b.record()
                b.synchronize()
                best = min(best, a.elapsed_time(b))
            times[bins] = best / (size / (16 * 4096))
        finally:
            p.abandon()
    assert times[63] < 4 * times[24], times  # a byte
